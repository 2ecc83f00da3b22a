"""Problems of up to one wave take 64-row tiles of their own kernel. Against the CPU oracle, and bit for bit against the general
kernel (a child process that forces its tiling): both add the products of an output in the same order, so that a batch of any
size gives an image the same result. The launch counter shows on both sides which kernel ran."""
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

# N, C, H, W, K, R, stride, pad, epilogue, channels-last: tile and k-step edges -- one to three and many k-steps (two share a
# stage, four stages are in flight), 1 / 63 / 64 / 65 pixels, 1 / 31 / 33 / 64 / 65 / 130 output channels, ragged channel
# counts, a plain matrix and an im2col A operand, both memory formats. With im2col copies 32-wide tiles are chosen whatever the number
# of k-steps, 64-wide ones up to 34 of 128 bytes.
CASES = [
    (1, 64, 1, 1, 64, 1, 1, 0, "bias", True), (1, 128, 7, 9, 33, 1, 1, 0, "relu", True),
    (1, 192, 8, 8, 65, 1, 1, 0, "bias+residual+relu", True), (5, 64, 13, 1, 31, 1, 1, 0, "gelu", True),
    (1, 1024, 14, 14, 256, 1, 1, 0, "bias+relu", True), (1, 64, 16, 16, 130, 3, 1, 1, "bias+silu", True),
    (2, 96, 7, 7, 64, 3, 1, 1, "bias+residual+relu", True), (3, 96, 9, 9, 66, 3, 2, 1, "residual", True),
    (1, 256, 14, 14, 96, 1, 2, 0, "bias", True), (1, 40, 10, 10, 64, 3, 1, 1, "bias+relu", True),
    (2, 72, 6, 7, 1, 3, 1, 1, "bias", True), (1, 100, 1, 37, 129, 1, 1, 0, "bias+residual", True),
    (1, 64, 56, 56, 64, 3, 1, 1, "bias+relu", False), (1, 72, 11, 13, 50, 3, 1, 0, "bias+residual+relu", False),
    (2, 64, 8, 8, 64, 1, 1, 0, "silu", False),
    # more 32-wide tiles than SMs, but no more 64-wide ones: those take 64 columns (a ring of three stages, two blocks of columns
    # in the epilogue). Rows of 16 bytes, of single elements and NCHW; 8 pixels in the last tile; an odd last k-step; im2col
    (2, 256, 14, 14, 1000, 1, 1, 0, "bias+residual+relu", True), (2, 256, 14, 14, 1001, 1, 1, 0, "bias+residual+relu", True),
    (2, 192, 14, 14, 1000, 1, 1, 0, "bias+residual+relu", False), (2, 96, 14, 14, 1000, 1, 1, 0, "gelu", True),
    (1, 128, 24, 24, 600, 2, 1, 0, "bias+residual", True),
]
# 64-wide tiles with an im2col operand, the ring filled twice and more: 16 and 9 k-steps of 128 bytes
CASES_OF = {
    2: [(1, 256, 24, 24, 600, 2, 1, 0, "bias+silu", True), (1, 64, 24, 24, 601, 3, 1, 1, "bias+residual+relu", False)],
    4: [(1, 128, 24, 24, 600, 2, 1, 0, "bias+silu", True), (1, 32, 24, 24, 601, 3, 1, 1, "bias+residual+relu", False)],
}


def cases(dtype):
    return CASES + CASES_OF[4 if dtype == "f32" else 2]


def inputs(case):
    N, C, H, W, K, R, stride, pad, epi, last = case
    x, w = cc.normal((N, C, H, W), 31, "small/x"), cc.kaiming((K, C, R, R), 31, "small/w")
    ho, wo = oracle.out_shape(x.shape, w.shape, stride, pad, 1)[2:]
    return x, w, cc.normal((K,), 31, "small/b", 0.1), cc.normal((N, K, ho, wo), 31, "small/r")


def run(case, dtype):
    N, C, H, W, K, R, stride, pad, epi, last = case
    x, w, b, r = inputs(case)
    fmt = torch.channels_last if last else torch.contiguous_format
    dev = lambda a: torch.from_numpy(a).to(TORCH_DT[dtype]).cuda().contiguous(memory_format=fmt)
    return ops.conv2d_nchw(dev(x), dev(w), torch.from_numpy(b).cuda() if "bias" in epi else None,
                           dev(r) if "residual" in epi else None, stride, pad, 1, 1, epi, channels_last_out=last)


@pytest.mark.parametrize("dtype", ["bf16", "f16", "f32"])
def test_small_tiles_match_the_oracle_and_the_general_kernel_bit_for_bit(dtype, tmp_path):
    got = []
    for case in cases(dtype):
        before = ffi.launch_count_of(ffi.KERNEL_SMALL_TILE)
        got.append(run(case, dtype))
        assert ffi.launch_count_of(ffi.KERNEL_SMALL_TILE) == before + 1, case
    torch.cuda.synchronize()
    assert ffi.load().tracea_b200_device_status(0) == 0
    for case, g in zip(cases(dtype), got):
        x, w, b, r = inputs(case)
        act = next((o for o in case[8].split("+") if o in ("relu", "silu", "gelu")), "none")
        want = oracle.conv2d_gemm(cc.channels_last(cc.round_to(x, dtype)), cc.round_to(w, dtype),
                                  b if "bias" in case[8] else None,
                                  cc.channels_last(cc.round_to(r, dtype)) if "residual" in case[8] else None,
                                  case[6], case[7], 1, act)
        err = cc.rel_err(g.float().cpu().numpy(), cc.round_to(np.ascontiguousarray(want), dtype))
        assert err <= cc.tol_for(dtype), (case, err)
    here = os.path.dirname(os.path.abspath(__file__))
    out = str(tmp_path / "general.npz")
    code = ("import sys; sys.path.insert(0, %r); sys.path.insert(0, %r)\n"
            "import numpy as np, test_small_tiles_gpu as t\n"
            "np.savez(%r, *[t.run(c, %r).float().cpu().numpy() for c in t.cases(%r)])\n"
            "assert t.ffi.launch_count_of(t.ffi.KERNEL_SMALL_TILE) == 0\n"
            "assert t.ffi.launch_count_of(t.ffi.KERNEL_GENERAL) == len(t.cases(%r))\n"
            % (os.path.dirname(here), here, out, dtype, dtype, dtype))
    env = dict(os.environ, TRACEA_B200_FORCE_BN="64")
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)
    general = np.load(out)
    for i, (case, g) in enumerate(zip(cases(dtype), got)):
        assert np.array_equal(general["arr_%d" % i], g.float().cpu().numpy()), case
