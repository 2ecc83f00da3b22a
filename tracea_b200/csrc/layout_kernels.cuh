// Layout adapters for callers that hand over NCHW-contiguous activations or OIHW-contiguous
// weights (the layouts include/tracea.hpp:101-105 documents). The conv kernel itself reads
// channels-last memory, which is what the reference's kernel reads too (NHWC input, conv.rs:202-247).
// The adapters read through arbitrary element strides and write dense, channel-padded buffers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tb200 {

// One copy src[n][c][p] (element strides) -> dst[n][p][Cp], channels C .. Cp-1 zero-filled: an activation tensor (p: its
// pixels), a filter bank (n: output channels, p: taps) or a matrix. Cp * sizeof(T) is a multiple of 16 bytes and dst is
// 16-byte aligned, except in kCopyElements. With pad_lo / pad_hi > 0 (never in kCopyTaps) every row of W pixels is written
// with that many zero pixels in front of and behind it.
enum : int {
  kCopyPlanes = 0,     // pixels contiguous (NCHW): 128-byte x 64-pixel tiles transposed through shared memory
  kCopyTaps = 1,       // pixels contiguous, few of them, and channels right behind one another (OIHW filters): a group of
                       // channels is one contiguous run
  kCopyRows = 2,       // channels contiguous but rows unaligned or short: rows copied with their padding
  kCopyElements = 3,   // anything else: 32 x 32 tiles, element by element
};
struct CopyJob {
  const void* src;
  void* dst;
  int mode;
  int vec;             // elements per source access (kCopyPlanes: along pixels, kCopyRows: along channels)
  int C, Cp, P, W, H;  // W: pixels per row of the source (pixel p is at (p / W) * sh + (p % W) * sw), H: rows
  int pad_lo, pad_hi;
  long long N;
  long long sn, sc, sh, sw;
  long long blocks;
};
struct CopyJobs {
  CopyJob job[2];
};
constexpr int kCopyThreads = 256;
constexpr int kCopyMaxTaps = 32;                       // kCopyTaps: pixels per image
template <typename T> constexpr int kCopyTileC = 128 / sizeof(T);   // channels per tile: 128 bytes
constexpr int kCopyTileP = 64;
template <typename T> constexpr int kCopyPitch = kCopyTileC<T> + 4 / static_cast<int>(sizeof(T));   // 33 words: an odd number

template <typename T, int kVec> struct CopyVec;
template <> struct CopyVec<uint16_t, 8> { using type = uint4; };
template <> struct CopyVec<uint16_t, 4> { using type = uint2; };
template <> struct CopyVec<uint16_t, 2> { using type = uint32_t; };
template <> struct CopyVec<uint16_t, 1> { using type = uint16_t; };
template <> struct CopyVec<uint32_t, 4> { using type = uint4; };
template <> struct CopyVec<uint32_t, 2> { using type = uint2; };
template <> struct CopyVec<uint32_t, 1> { using type = uint32_t; };

// Planes: every thread's source accesses are issued before the first is used, consecutive lanes read consecutive pixels.
template <typename T, int kVec>
__device__ __forceinline__ void copy_tile_in(const CopyJob& j, T* tile, const T* src, int c0, int p0) {
  using V = typename CopyVec<T, kVec>::type;
  constexpr int kPerRow = kCopyTileP / kVec;
  constexpr int kIters = kCopyTileC<T> * kPerRow / kCopyThreads;
  V v[kIters];
#pragma unroll
  for (int i = 0; i < kIters; ++i) {
    const int t = i * kCopyThreads + static_cast<int>(threadIdx.x);
    const int c = c0 + t / kPerRow, p = p0 + t % kPerRow * kVec;
    v[i] = V{};
    if (c < j.C && p < j.P) v[i] = *reinterpret_cast<const V*>(src + c * j.sc + p);   // P is a multiple of kVec
  }
#pragma unroll
  for (int i = 0; i < kIters; ++i) {
    const int t = i * kCopyThreads + static_cast<int>(threadIdx.x);
    const int c = t / kPerRow, p = t % kPerRow * kVec;
    const T* e = reinterpret_cast<const T*>(&v[i]);
#pragma unroll
    for (int k = 0; k < kVec; ++k) tile[(p + k) * kCopyPitch<T> + c] = e[k];
  }
}
// One V of pixel p of image n, at channel c of the destination. kPad: rows carry zero pixels, and whoever writes a row's first or
// last pixel writes those beside it. (A template argument, and one division: as run-time branches with three of them, copies
// without padding took 0.2 us longer, of 8.6 for a one-image call.)
template <bool kPad, typename T, typename V>
__device__ __forceinline__ void copy_store(const CopyJob& j, T* dst, long long n, int p, int c, const V& v) {
  if constexpr (!kPad) {
    *reinterpret_cast<V*>(dst + (n * j.P + p) * j.Cp + c) = v;
  } else {
    const int h = p / j.W, w = p - h * j.W;
    T* at = dst + ((n * j.H + h) * (j.W + j.pad_lo + j.pad_hi) + j.pad_lo + w) * j.Cp + c;
    *reinterpret_cast<V*>(at) = v;
    if (w == 0)
      for (int k = 1; k <= j.pad_lo; ++k) *reinterpret_cast<V*>(at - static_cast<long long>(k) * j.Cp) = V{};
    if (w == j.W - 1)
      for (int k = 1; k <= j.pad_hi; ++k) *reinterpret_cast<V*>(at + static_cast<long long>(k) * j.Cp) = V{};
  }
}
// 16 bytes of one tile row (4-byte aligned).
template <typename T>
__device__ __forceinline__ uint4 tile_chunk(const T* row, int chunk) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(row) + chunk * 4;
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Layout adapters of one call -- the activations, the filter bank, or both -- as one launch: a small call's time is the
// number of dependent launches in front of its convolution, not their bytes.
template <typename T, bool kPad>
__global__ void __launch_bounds__(kCopyThreads) copy_channels_last_kernel(const __grid_constant__ CopyJobs jobs) {
  // the convolution behind this launch may bring up its CTAs; the sources may come from, and the scratch may still be read
  // by, the launch in front of it
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ __align__(16) T tile[kCopyTileP * kCopyPitch<T>];
  constexpr int kChunk = 16 / sizeof(T);               // elements per 16 bytes
  long long b = blockIdx.x;
  const bool second = b >= jobs.job[0].blocks;
  if (second) b -= jobs.job[0].blocks;
  const CopyJob& j = jobs.job[second ? 1 : 0];
  const T* src = static_cast<const T*>(j.src);
  T* dst = static_cast<T*>(j.dst);
  const int tid = static_cast<int>(threadIdx.x);
  if (j.mode == kCopyPlanes) {
    const int tiles_p = (j.P + kCopyTileP - 1) / kCopyTileP, tiles_c = (j.Cp + kCopyTileC<T> - 1) / kCopyTileC<T>;
    const int tp = static_cast<int>(b % tiles_p);
    const long long t = b / tiles_p;
    const int c0 = static_cast<int>(t % tiles_c) * kCopyTileC<T>, p0 = tp * kCopyTileP;
    const long long n = t / tiles_c;
    const T* s = src + n * j.sn;
    if (j.vec == 1) copy_tile_in<T, 1>(j, tile, s, c0, p0);
    else if (j.vec == 2) copy_tile_in<T, 2>(j, tile, s, c0, p0);
    else if (j.vec == 4) copy_tile_in<T, 4>(j, tile, s, c0, p0);
    else if constexpr (sizeof(T) == 2) copy_tile_in<T, 8>(j, tile, s, c0, p0);
    __syncthreads();
    for (int i = tid; i < kCopyTileP * 8; i += kCopyThreads) {   // 8 lanes write one pixel's 128 bytes
      const int p = i >> 3, c = c0 + (i & 7) * kChunk;
      if (p0 + p < j.P && c < j.Cp) copy_store<kPad>(j, dst, n, p0 + p, c, tile_chunk(tile + p * kCopyPitch<T>, i & 7));
    }
  } else if (j.mode == kCopyTaps) {
    // one block: one group of 128 bytes of channels of as many images (output channels) as fill the tile
    const int tiles_c = (j.Cp + kCopyTileC<T> - 1) / kCopyTileC<T>;
    const int c0 = static_cast<int>(b % tiles_c) * kCopyTileC<T>;
    const int per = kCopyTileP / j.P;
    const long long n0 = b / tiles_c * per;
    const int run = min(kCopyTileC<T>, j.C - c0) * j.P;            // contiguous source elements (<= 0: padding only)
    const int full = kCopyTileC<T> * j.P;
#pragma unroll 4
    for (int i = tid; i < per * full; i += kCopyThreads) {
      const int k = i / full, e = i - k * full;
      const int c = e / j.P, p = e - c * j.P;
      T v = T(0);
      if (n0 + k < j.N && e < run) v = src[(n0 + k) * j.sn + static_cast<long long>(c0) * j.P + e];
      tile[(k * j.P + p) * kCopyPitch<T> + c] = v;
    }
    __syncthreads();
    for (int i = tid; i < per * j.P * 8; i += kCopyThreads) {
      const int r = i >> 3, c = c0 + (i & 7) * kChunk;
      if (n0 + r / j.P < j.N && c < j.Cp)
        *reinterpret_cast<uint4*>(dst + (n0 * j.P + r) * j.Cp + c) = tile_chunk(tile + r * kCopyPitch<T>, i & 7);
    }
  } else if (j.mode == kCopyRows) {
    const int per_row = j.Cp / kChunk;
    const long long total = j.N * j.P * per_row;
    const long long i = b * kCopyThreads + tid;
    if (i >= total) return;
    const long long row = i / per_row;
    const int c = static_cast<int>(i - row * per_row) * kChunk;
    const long long n = row / j.P;
    const int p = static_cast<int>(row - n * j.P), h = p / j.W;
    const T* s = src + n * j.sn + h * j.sh + (p - h * j.W) * j.sw + c;
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    T* e = reinterpret_cast<T*>(&out);
    if (c + kChunk <= j.C) {
      if (sizeof(T) == 2 && j.vec == 2) {
        uint32_t* w = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = reinterpret_cast<const uint32_t*>(s)[k];
      } else {
#pragma unroll
        for (int k = 0; k < kChunk; ++k) e[k] = s[k];
      }
    } else {
#pragma unroll
      for (int k = 0; k < kChunk; ++k)
        if (c + k < j.C) e[k] = s[k];
    }
    copy_store<kPad>(j, dst, n, p, c, out);
  } else {
    const int tiles_p = (j.P + 31) / 32, tiles_c = (j.Cp + 31) / 32;
    const int p0 = static_cast<int>(b % tiles_p) * 32;
    const long long t = b / tiles_p;
    const int c0 = static_cast<int>(t % tiles_c) * 32;
    const long long n = t / tiles_c;
    const int tx = tid & 31, ty = tid >> 5;
    const int p = p0 + tx;
    const long long poff = p < j.P ? static_cast<long long>(p / j.W) * j.sh + (p % j.W) * j.sw : 0;
    for (int i = ty; i < 32; i += kCopyThreads / 32) {
      const int c = c0 + i;
      T v = T(0);
      if (p < j.P && c < j.C) v = src[n * j.sn + c * j.sc + poff];
      tile[i * 33 + tx] = v;
    }
    __syncthreads();
    const int c = c0 + tx;
    for (int i = ty; i < 32; i += kCopyThreads / 32)
      if (p0 + i < j.P && c < j.Cp) copy_store<kPad>(j, dst, n, p0 + i, c, tile[tx * 33 + i]);
  }
}

// Small-channel inputs (one pixel = 16 bytes after channel padding, e.g. RGB as 8 x bf16): x -> dst[n][h][Wp][Cp]
// with `pad` zero pixels in front of every row and zeros up to the row pitch Wp behind it. With the
// horizontal padding materialised, the S taps of one filter row are adjacent in memory, so the conv
// kernel fetches a whole filter row of a pixel (8 pixels x 16 B = one 128-byte k-chunk) with one copy.
// One thread writes one destination pixel (16 bytes).
template <typename T, int kCp>
__global__ void to_channels_last_wpad_kernel(const T* __restrict__ src, T* __restrict__ dst, int C, int H, int W,
                                             int Wp, int pad, long long total_pixels, long long sn, long long sc,
                                             long long sh, long long sw) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= total_pixels) return;
  const int wp = static_cast<int>(i % Wp);
  const long long t = i / Wp;
  const int h = static_cast<int>(t % H);
  const long long n = t / H;
  const int w = wp - pad;
  T v[kCp];
#pragma unroll
  for (int c = 0; c < kCp; ++c) v[c] = T(0);
  if (w >= 0 && w < W) {
    const T* p = src + n * sn + h * sh + w * sw;
#pragma unroll
    for (int c = 0; c < kCp; ++c)
      if (c < C) v[c] = p[c * sc];
  }
  if constexpr (kCp * sizeof(T) == 16) *reinterpret_cast<uint4*>(dst + i * kCp) = *reinterpret_cast<const uint4*>(v);
  else *reinterpret_cast<uint2*>(dst + i * kCp) = *reinterpret_cast<const uint2*>(v);   // 8-byte pixels (4 x 16 bit)
}

// w[k, c, r, s] (element strides) -> dst[k][r][s][Cp], zero-padded channels: the K-major B operand
// whose Kgemm axis runs (r, s, c), the order the reference walks it (conv.rs:209-210).
// `Sd` >= S is the number of tap slots per filter row in the destination (slots s >= S are zero).
template <typename T>
__global__ void pack_weights_krsc_kernel(const T* __restrict__ src, T* __restrict__ dst,
                                         long long total, int C, int R, int S, int Sd, int Cp, long long sk,
                                         long long sc, long long sr, long long ss) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= total) return;
  const int c = static_cast<int>(i % Cp);
  long long t = i / Cp;
  const int s = static_cast<int>(t % Sd);
  t /= Sd;
  const int r = static_cast<int>(t % R);
  const long long k = t / R;
  dst[i] = (c < C && s < S) ? src[k * sk + c * sc + r * sr + s * ss] : T(0);
}

// The padded copy of a channels-last RGB image of 16-bit values (pixel pitch 3 elements) as 4-channel pixels, and its filter bank
// packed [K][R][Sd][4], in one programmatic launch in front of the row-band kernel. Bound by the memory system: a thread turns the
// source of two neighbouring destination pixels into one 16-byte store, so that a warp's store covers 512 consecutive bytes (as
// four 8-byte stores a thread, 32 bytes apart, a store touched every sector a quarter at a time); kStemRows rows a block, their
// loads in flight together. Pixels outside the image are zeros. Rows of the source start on 4-byte boundaries, W and Wp are even.
// Whole calls of the 7x7/2 stem at 224x224, bf16, with the copy and the packing as two ordinary launches (four pixels a thread) and
// with this one: 1 image 9.2 -> 9.0 us replayed and 15.8 -> 12.2 issued one by one, 32 images 29.7 -> 28.8, 256 173 -> 163, 512 337 -> 316.
// The launch behind it may only come up beside its last blocks while the copy is about a wave (`early`): with more, calls issued one
// behind another took 181 us at 256 images and 350 at 512 (1 image without: 9.4). Why is not established.
constexpr int kStemThreads = 128, kStemRows = 8;
struct StemCopy {
  const uint16_t* src;
  uint16_t* dst;
  int H, W, Wp, pad, rows, image_blocks;   // rows: N * H
  int early;                               // let the next launch start before this one is done
  long long src_img, src_row;
  const uint16_t* w;
  uint16_t* w_dst;
  int C, R, S, Sd, w_total;                // w_total: K * R * Sd * 4
  long long sk, sc, sr, ss;
};
// Pixel i of a source row as {e0 | e1 << 16, e2}, zeros outside the row.
__device__ __forceinline__ uint2 rgb16_pixel(const uint32_t* row, int i, int W) {
  if (i < 0 || i >= W) return make_uint2(0u, 0u);
  const uint32_t* w = row + ((3 * i) >> 1);
  const uint32_t a = w[0], b = w[1];
  return (i & 1) != 0 ? make_uint2((a >> 16) | (b << 16), b >> 16) : make_uint2(a, b & 0xffffu);
}
__global__ void __launch_bounds__(kStemThreads) rgb16_stem_copy_kernel(const __grid_constant__ StemCopy c) {
  if (c.early != 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = static_cast<int>(threadIdx.x);
  if (static_cast<int>(blockIdx.x) >= c.image_blocks) {
    const int i = (static_cast<int>(blockIdx.x) - c.image_blocks) * kStemThreads + tid;
    if (i >= c.w_total) return;
    const int ch = i & 3, s = (i >> 2) % c.Sd, t = (i >> 2) / c.Sd, r = t % c.R, k = t / c.R;
    c.w_dst[i] = ch < c.C && s < c.S ? c.w[k * c.sk + ch * c.sc + r * c.sr + s * c.ss] : uint16_t(0);
    return;
  }
  const int row0 = static_cast<int>(blockIdx.x) * kStemRows;
  const int count = min(kStemRows, c.rows - row0);
  const int n0 = row0 / c.H, h0 = row0 - n0 * c.H;
  for (int j = tid; j < c.Wp / 2; j += kStemThreads) {
    int n = n0, h = h0;
    uint4* d = reinterpret_cast<uint4*>(c.dst + static_cast<long long>(row0) * c.Wp * 4) + j;
    for (int r0 = 0; r0 < count; r0 += kStemRows / 2) {
      uint4 v[kStemRows / 2];
#pragma unroll
      for (int k = 0; k < kStemRows / 2; ++k) {
        if (r0 + k >= count) break;
        const uint32_t* row = reinterpret_cast<const uint32_t*>(c.src + n * c.src_img + h * c.src_row);
        const uint2 a = rgb16_pixel(row, 2 * j - c.pad, c.W), b = rgb16_pixel(row, 2 * j + 1 - c.pad, c.W);
        v[k] = make_uint4(a.x, a.y, b.x, b.y);
        if (++h == c.H) { h = 0; ++n; }
      }
#pragma unroll
      for (int k = 0; k < kStemRows / 2; ++k) {
        if (r0 + k >= count) break;
        *d = v[k];
        d += c.Wp / 2;
      }
    }
  }
}

}  // namespace tb200
