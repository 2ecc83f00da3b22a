"""Edges of the forms a call can take inside the library that are chosen by a rule on its sizes, against the CPU oracle (or, for
matrix products, float64), with the launch counters that show which kernel ran."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import convcases as cc
from oracle import oracle
from tracea_b200 import ffi, ops

pytestmark = pytest.mark.gpu

TORCH_DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def conv(case, dtype):
    """Runs one case (N, C, H, W, K, R, stride, pad, epilogue, channels-last) and returns (output, oracle's output)."""
    N, C, H, W, K, R, stride, pad, epi, last = case
    x, w = cc.normal((N, C, H, W), 57, "forms/x"), cc.kaiming((K, C, R, R), 57, "forms/w")
    ho, wo = oracle.out_shape(x.shape, w.shape, stride, pad, 1)[2:]
    b = cc.normal((K,), 57, "forms/b", 0.1) if "bias" in epi else None
    r = cc.normal((N, K, ho, wo), 57, "forms/r") if "residual" in epi else None
    dev = lambda a: torch.from_numpy(a).to(TORCH_DT[dtype]).cuda().contiguous(
        memory_format=torch.channels_last if last else torch.contiguous_format)
    got = ops.conv2d_nchw(dev(x), dev(w), torch.from_numpy(b).cuda() if b is not None else None,
                          dev(r) if r is not None else None, stride, pad, 1, 1, epi, channels_last_out=last)
    act = next((o for o in epi.split("+") if o in ("relu", "silu", "gelu")), "none")
    want = oracle.conv2d_gemm(cc.channels_last(cc.round_to(x, dtype)), cc.round_to(w, dtype), b,
                              cc.channels_last(cc.round_to(r, dtype)) if r is not None else None, stride, pad, 1, act)
    return got, cc.round_to(np.ascontiguousarray(want), dtype)


def check(case, dtype):
    got, want = conv(case, dtype)
    err = cc.rel_err(got.float().cpu().numpy(), want)
    assert err <= cc.tol_for(dtype), (case, dtype, err)
    return got


# Staging boxes per epilogue warp: two below 8 k-steps, with a residual and with SiLU or GELU, otherwise one, none for NCHW. The bias:
# one copy for the CTA up to 512 columns (whole tiles counted), above them a copy of its tile's columns per epilogue warp. Outputs moved
# by the TMA unit and, where rows are of odd length, by the warps. More tiles than SMs, so that every buffer comes round again.
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("steps", [7, 8, 9])
@pytest.mark.parametrize("K,epi,last", [(264, "bias+relu", True), (512, "bias+residual+relu", True), (520, "bias+silu", True),
                                        (1000, "bias+residual", True), (600, "bias", False), (72, "bias+gelu", True),
                                        (520, "bias", True), (1000, "bias+relu", True), (261, "bias+relu", True),
                                        (777, "bias", True)])
def test_staging_depth_and_bias_forms(dtype, steps, K, epi, last):
    C = steps * (32 if dtype == "f32" else 64)
    before = ffi.launch_count_of(ffi.KERNEL_GENERAL)
    check((4, C, 73, 67, K, 1, 1, 0, epi.replace("bias+gelu", "gelu"), last), dtype)
    assert ffi.launch_count_of(ffi.KERNEL_GENERAL) == before + 1


# Row-major B of 16-bit elements, read in place 64 columns at a time: columns and rows of K at the edges of those blocks, all
# tilings (rows up to one small tile, one wave, many). The sums are added in the order of a K-major B: the same bits.
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("M", [1, 65, 3000, 20000])
def test_row_major_b_is_read_in_place(dtype, M):
    for N, K in ((8, 64), (64, 40), (72, 72), (136, 200), (264, 520), (1000, 776), (640, 1024)):
        a = torch.from_numpy(cc.normal((M, K), 58, "mn/a")).to(TORCH_DT[dtype]).cuda()
        b = torch.from_numpy(cc.normal((K, N), 58, "mn/b", K ** -0.5)).to(TORCH_DT[dtype]).cuda()
        before = ffi.launch_count_of(ffi.KERNEL_LAYOUT)
        got = ops.gemm(a, b)
        assert ffi.launch_count_of(ffi.KERNEL_LAYOUT) == before, (M, N, K)
        want = a.double() @ b.double()
        assert float((got.double() - want).abs().max() / want.abs().max()) <= cc.TOL_16BIT, (M, N, K)
        assert torch.equal(got, ops.gemm(a, b.t().contiguous().t())), (M, N, K)
    wide = torch.from_numpy(cc.normal((96, 136), 58, "mn/w")).to(TORCH_DT[dtype]).cuda()
    a = torch.from_numpy(cc.normal((M, 96), 58, "mn/a2")).to(TORCH_DT[dtype]).cuda()
    part = wide[:, 8:128]            # columns of a wider matrix
    assert torch.equal(ops.gemm(a, part), ops.gemm(a, part.t().contiguous().t()))
    odd = wide[:, 1:100]             # no 16-byte rows: repacked as ever
    assert torch.equal(ops.gemm(a, odd), ops.gemm(a, odd.t().contiguous().t()))


# The same form where tiles are cut over K (an option, read once per process): a piece begins at a row of B that is not the first. All
# tilings, tiles cut in two and in many, and the general kernel's whole tiles beside them.
_SPLIT_ROW_MAJOR = """
import sys; sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
import torch, convcases as cc
from tracea_b200 import ffi, ops
for dt in (torch.bfloat16, torch.float16):
    for M, N, K in ((65, 1000, 776), (3000, 640, 1024), (20000, 264, 520), (5000, 512, 2048), (9000, 64, 1032), (300, 72, 136)):
        a = torch.from_numpy(cc.normal((M, K), 58, "mn/a")).to(dt).cuda()
        b = torch.from_numpy(cc.normal((K, N), 58, "mn/b", K ** -0.5)).to(dt).cuda()
        split, copies = ffi.launch_count_of(ffi.KERNEL_SPLIT_K), ffi.launch_count_of(ffi.KERNEL_LAYOUT)
        got = ops.gemm(a, b)
        assert ffi.launch_count_of(ffi.KERNEL_SPLIT_K) == split + 1 and ffi.launch_count_of(ffi.KERNEL_LAYOUT) == copies, (M, N, K)
        want = a.double() @ b.double()
        assert float((got.double() - want).abs().max() / want.abs().max()) <= cc.TOL_16BIT, (M, N, K)
        assert torch.equal(got, ops.gemm(a, b.t().contiguous().t())), (M, N, K)
assert ffi.load().tracea_b200_device_status(0) == 0
print("row-major ok")
"""


def test_row_major_b_in_tiles_cut_over_k():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", _SPLIT_ROW_MAJOR, root], capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, TRACEA_B200_SPLIT_K="2"))
    assert done.returncode == 0 and "row-major ok" in done.stdout, done.stdout[-1000:] + done.stderr[-2000:]


# One-tap filters whose output channels are contiguous are read in place like a row-major B: 1x1 layers, strided or on NCHW memory (whose
# copy is the call's only one), and the one-tap phases of a transposed convolution beside phases of more taps. The bits of K-major filters.
@pytest.mark.parametrize("dtype", ["bf16", "f16", "f32"])
def test_one_tap_filters_with_contiguous_output_channels(dtype):
    in_place = dtype != "f32"
    for N, C, H, W, K, stride, last in ((2, 128, 9, 11, 64, 1, True), (3, 72, 14, 13, 136, 2, True), (40, 256, 28, 28, 320, 1, True),
                                        (2, 100, 15, 9, 72, 1, False), (16, 576, 28, 28, 128, 1, False)):
        x = torch.from_numpy(cc.normal((N, C, H, W), 65, "tap/x")).to(TORCH_DT[dtype]).cuda()
        if last:
            x = x.contiguous(memory_format=torch.channels_last)
        w = torch.from_numpy(cc.normal((C, K), 65, "tap/w", C ** -0.5)).to(TORCH_DT[dtype]).cuda()
        before = ffi.launch_count_of(ffi.KERNEL_LAYOUT)
        got = ops.conv2d_nchw(x, w.t()[:, :, None, None], None, None, stride)
        assert ffi.launch_count_of(ffi.KERNEL_LAYOUT) - before == (0 if in_place and last else 1), (C, K)
        want = torch.nn.functional.conv2d(x.double(), w.double().t()[:, :, None, None], stride=stride)
        assert float((got.double() - want).abs().max() / want.abs().max()) <= cc.tol_for(dtype), (C, K)
        assert torch.equal(got, ops.conv2d_nchw(x, w.t().contiguous()[:, :, None, None], None, None, stride)), (C, K)
    for N, C, H, W, K, R, pad in ((2, 64, 9, 7, 72, 2, 0), (3, 128, 8, 10, 64, 3, 1), (1, 192, 5, 6, 136, 3, 0)):
        x = torch.from_numpy(cc.normal((N, H, W, C), 66, "tap/x")).to(TORCH_DT[dtype]).cuda()
        w = torch.from_numpy(cc.normal((R, R, C, K), 66, "tap/w", (C * R * R) ** -0.5)).to(TORCH_DT[dtype]).cuda().permute(3, 0, 1, 2)
        before = ffi.launch_count_of(ffi.KERNEL_LAYOUT)
        got = ops.conv_transpose2d(x, w, None, None, "relu", 2, pad)
        taps = [(R + 1 - a) // 2 for a in (0, 1)]   # of the filter's rows, those that even and odd output rows see
        assert ffi.launch_count_of(ffi.KERNEL_LAYOUT) - before == sum(not in_place or a * b > 1 for a in taps for b in taps), (C, R)
        want = torch.nn.functional.conv_transpose2d(x.double().permute(0, 3, 1, 2), w.double().permute(3, 0, 1, 2), stride=2,
                                                    padding=pad).permute(0, 2, 3, 1).relu()
        assert float((got.double() - want).abs().max() / want.abs().max()) <= cc.tol_for(dtype), (C, R)
        assert torch.equal(got, ops.conv_transpose2d(x, w.contiguous(), None, None, "relu", 2, pad)), (C, R)


# Filter rows as k-chunks: channel counts around the pixel pitches of 16 and 32 bytes and around whole chunks, both memory formats
# that are staged (NCHW, channels-last of odd channel counts), strides, no padding, narrow and one-pixel images, every filter width.
# The last column: element sizes that take this form; the others save no chunk, or their copy would double.
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_filter_rows_as_chunks(dtype):
    for *case, sizes in ((3, 20, 31, 23, 50, 5, 1, 2, "gelu", False, (2, 4)), (2, 33, 17, 40, 100, 3, 2, 1, "bias+relu", False, (2, 4)),
                 (1, 12, 40, 41, 64, 7, 2, 3, "bias+relu", False, (2, 4)), (2, 96, 14, 15, 72, 3, 1, 1, "bias+residual+relu", False, (2,)),
                 (2, 50, 9, 11, 33, 3, 1, 1, "residual+relu", True, (4,)), (1, 17, 1, 1, 20, 3, 1, 1, "bias", False, ()),
                 (2, 25, 8, 6, 40, 2, 1, 0, "relu", False, (2,)), (1, 200, 12, 12, 130, 3, 1, 0, "bias+silu", False, (2, 4)),
                 (40, 40, 28, 28, 64, 3, 1, 1, "bias+relu", False, (2, 4)), (1, 11, 30, 30, 9, 16, 1, 8, "bias", False, (2, 4)),
                 (2, 9, 5, 7, 70, 5, 3, 2, "bias", True, (2, 4)), (2, 104, 11, 13, 40, 7, 1, 3, "bias+relu", False, (2, 4)),
                 (1, 200, 9, 10, 33, 5, 2, 2, "bias", False, (2, 4)), (3, 100, 10, 9, 70, 7, 1, 3, "silu", False, (2, 4))):
        before = ffi.launch_count_of(ffi.FORM_FILTER_ROWS)
        check(case, dtype)
        taken = ffi.launch_count_of(ffi.FORM_FILTER_ROWS) - before
        assert taken == int((4 if dtype == "f32" else 2) in sizes), case


# One layer in both memory formats. Tap by tap the two agree bit for bit; filter rows as k-chunks, which only a copied input takes,
# add the same products in another order: apart by what two fp32 sums of R*S*C products can be -- 2^-23 of the sum of their
# magnitudes for each product, a generous bound for either -- and one step of the storage type.
@pytest.mark.parametrize("dtype", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("C,sizes", [(40, (2, 4)), (24, (2,)), (64, ()), (256, ())])   # sizes: of elements that take filter rows
def test_memory_formats_of_one_layer(dtype, C, sizes):
    rows = (4 if dtype == "f32" else 2) in sizes
    x = torch.from_numpy(cc.normal((3, C, 19, 21), 67, "fmt/x")).to(TORCH_DT[dtype]).cuda()
    w = torch.from_numpy(cc.kaiming((72, C, 3, 3), 67, "fmt/w")).to(TORCH_DT[dtype]).cuda()
    last = dict(memory_format=torch.channels_last)
    before = ffi.launch_count_of(ffi.FORM_FILTER_ROWS)
    planes = ops.conv2d_nchw(x, w, None, None, 1, 1)
    assert ffi.launch_count_of(ffi.FORM_FILTER_ROWS) - before == rows
    pixels = ops.conv2d_nchw(x.contiguous(**last), w.contiguous(**last), None, None, 1, 1)
    assert ffi.launch_count_of(ffi.FORM_FILTER_ROWS) - before == rows
    if not rows:
        assert torch.equal(planes, pixels)
        return
    sums = torch.nn.functional.conv2d(x.double().abs(), w.double().abs(), padding=1)
    step = {"bf16": 2.0 ** -7, "f16": 2.0 ** -10, "f32": 2.0 ** -23}[dtype]
    bound = 2 * 9 * C * 2.0 ** -23 * sums + step * torch.maximum(planes.double().abs(), pixels.double().abs())
    assert bool(((planes.double() - pixels.double()).abs() <= bound).all())


# An im2col map's corners go from -128 to 127: wider paddings are refused in every memory format, also where the padding would be copied.
@pytest.mark.parametrize("C", [20, 24, 64])
@pytest.mark.parametrize("last", [False, True])
def test_paddings_beyond_the_im2col_corners_are_refused(C, last):
    fmt = torch.channels_last if last else torch.contiguous_format
    x = torch.randn((2, C, 9, 300), device="cuda").bfloat16().contiguous(memory_format=fmt)
    w = torch.randn((8, C, 3, 3), device="cuda").bfloat16().contiguous(memory_format=fmt)
    got = ops.conv2d_nchw(x, w, None, None, 1, (1, 128))
    want = torch.nn.functional.conv2d(x.double(), w.double(), padding=(1, 128))
    assert float((got.double() - want).abs().max() / want.abs().max()) <= cc.TOL_16BIT
    for pad in (129, 200):
        with pytest.raises(ffi.TraceaError) as e:
            ops.conv2d_nchw(x, w, None, None, 1, (1, pad))
        assert e.value.status == ffi.CUDA_ERROR and "Im2col" in e.value.message


# The phases of a transposed convolution pad front and back differently.
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_filter_rows_in_the_phases_of_a_transposed_convolution(dtype):
    for N, C, H, W, K, R, stride, pad, opad in ((2, 20, 9, 13, 24, 4, 2, 1, 0), (1, 33, 7, 6, 40, 5, 2, 2, 1), (1, 50, 5, 8, 17, 5, 3, 1, 2)):
        x = torch.from_numpy(cc.normal((N, H, W, C), 59, "ct/x")).to(TORCH_DT[dtype]).cuda()
        w = torch.from_numpy(cc.normal((K, R, R, C), 59, "ct/w", (C * R * R) ** -0.5)).to(TORCH_DT[dtype]).cuda()
        got = ops.conv_transpose2d(x, w, None, None, None, stride, pad, opad)
        want = torch.nn.functional.conv_transpose2d(x.double().permute(0, 3, 1, 2), w.double().permute(3, 0, 1, 2), stride=stride,
                                                    padding=pad, output_padding=opad).permute(0, 2, 3, 1)
        assert float((got.double() - want).abs().max() / want.abs().max()) <= cc.tol_for(dtype)


# 32-wide small tiles whatever the number of k-steps: walks longer than the 31 steps up to which they used to be chosen, bit for bit against
# the general kernel; pixels that do not start on 32-byte sectors keep it beyond a few tiles.
LONG_WALKS = [(1, 256, 14, 14, 256, 3, 1, 1, "bias+relu", True), (2, 512, 7, 7, 520, 3, 1, 1, "bias+residual+relu", True),
              (1, 128, 20, 20, 96, 5, 1, 2, "gelu", False), (3, 320, 9, 7, 33, 3, 2, 1, "bias", True)]


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_small_tiles_for_long_walks(dtype, tmp_path):
    got = []
    for case in LONG_WALKS:
        before = ffi.launch_count_of(ffi.KERNEL_SMALL_TILE)
        got.append(check(case, dtype))
        assert ffi.launch_count_of(ffi.KERNEL_SMALL_TILE) == before + 1, case
    before = ffi.launch_count_of(ffi.KERNEL_GENERAL)
    check((93, 120 if dtype != "f32" else 124, 12, 12, 128, 3, 2, 1, "bias+silu", True), dtype)
    assert ffi.launch_count_of(ffi.KERNEL_GENERAL) == before + 1
    here = os.path.dirname(os.path.abspath(__file__))
    out = str(tmp_path / "general.npz")
    code = ("import sys; sys.path.insert(0, %r); sys.path.insert(0, %r)\n"
            "import numpy as np, test_forms_gpu as t\n"
            "np.savez(%r, *[t.conv(c, %r)[0].float().cpu().numpy() for c in t.LONG_WALKS])\n"
            "assert t.ffi.launch_count_of(t.ffi.KERNEL_SMALL_TILE) == 0\n" % (os.path.dirname(here), here, out, dtype))
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, TRACEA_B200_FORCE_BN="64"), timeout=300)
    general = np.load(out)
    for i, g in enumerate(got):
        assert np.array_equal(general["arr_%d" % i], g.float().cpu().numpy()), LONG_WALKS[i]


# The resident-filter kernel's tile height follows the number of tiles: heights for one to four blocks of pixels, with and without a
# shorter tile at the bottom, odd tile counts.
@pytest.mark.parametrize("case", [(32, 64, 56, 56, 64, 3, 1, 1, "bias+relu", True), (21, 64, 56, 56, 48, 3, 1, 1, "silu", True),
                                  (39, 64, 40, 40, 64, 3, 1, 1, "bias", True), (37, 64, 37, 46, 56, 3, 1, 1, "gelu", True),
                                  (13, 64, 112, 112, 64, 3, 1, 1, "relu", True), (80, 64, 56, 56, 8, 3, 1, 1, "bias", True)])
def test_resident_filter_tile_heights(case):
    before = ffi.launch_count_of(ffi.KERNEL_RESIDENT_FILTER)
    check(case, "bf16")
    assert ffi.launch_count_of(ffi.KERNEL_RESIDENT_FILTER) == before + 1


# The copy in front of the RGB stem: odd and even padding, rows that are no multiple of a block's eight, widths over and under a block's
# 128 pixel pairs, images of a wider batch, rows that start on odd elements (the general copy).
@pytest.mark.parametrize("case", [(2, 3, 33, 160, 64, 7, 2, 3, "bias+relu", True), (3, 3, 21, 166, 48, 5, 2, 2, "relu", True),
                                  (1, 3, 40, 600, 64, 3, 2, 1, "bias", True), (5, 3, 17, 170, 16, 7, 2, 0, "bias", True),
                                  (2, 3, 30, 165, 64, 7, 2, 3, "bias+relu", True)])
def test_rgb_stem_copies(case):
    before = ffi.launch_count_of(ffi.KERNEL_ROW_BAND)
    check(case, "bf16")
    check(case, "f16")
    assert ffi.launch_count_of(ffi.KERNEL_ROW_BAND) == before + 2


# Calls right behind one another hand the same scratch on: the copy and the packed filter bank of one are rewritten for the next
# while the launch that read them drains. Three banks and two inputs in turn; one image is the least work a launch can have, and with 300
# the copy is more than a wave, which the next launch does not start beside.
@pytest.mark.parametrize("images", [1, 300])
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
def test_rgb_stems_behind_one_another(dtype, images):
    xs = [torch.from_numpy(cc.normal((images, 40, 66, 3), 61 + i, "stems/x")).to(TORCH_DT[dtype]).cuda() for i in range(2)]
    ws = [torch.from_numpy(cc.normal((64, 7, 7, 3), 63 + i, "stems/w", 0.1)).to(TORCH_DT[dtype]).cuda() for i in range(3)]
    want = {}
    for i, x in enumerate(xs):
        for k, w in enumerate(ws):
            want[i, k] = ops.conv2d(x, w, None, None, "relu", 2, 3)
            torch.cuda.synchronize()
    got = [(n % 2, n % 3, ops.conv2d(xs[n % 2], ws[n % 3], None, None, "relu", 2, 3)) for n in range(240 if images == 1 else 24)]
    assert all(torch.equal(out, want[i, k]) for i, k, out in got)
