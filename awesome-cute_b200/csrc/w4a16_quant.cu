// Device-side Layer.pack: fake-quantised (or plain) fp16 weights + scales -> Marlin-packed int4 words and permuted
// scales, bit-exact with the host packer (w4a16_pack.cpp) and therefore with the reference's numpy packer
// (gemm/marlin_gemm/marlin.py:92-131).  Elementwise work, HBM-bound when done right: 2 bytes read and 0.5 byte written
// per weight.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/w4a16.h"

namespace {

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }

// The reference's quantiser as it is written (marlin.py:108-110): fp16 quotient, round half to even, + 8, clamp.
__device__ __noinline__ uint32_t quantize_exact(__half w, float s) {
  const float quo = __half2float(__float2half_rn(__half2float(w) / s));
  const int code = (int)rintf(quo) + 8;
  return (uint32_t)(code < 0 ? 0 : (code > 15 ? 15 : code));
}

// Two weights of one column (k, k + 1) -> their codes in bits 0..3 and 16..19.
//
// Quotient without a divide: with rs = 1 / s rounded correctly, q0 = w * rs, r = w - q0 * s (one fma: exact, q0 * s
// and w agree to within a few units in the last place) and q = q0 + r * rs, q is within 0.51 units in the last place
// of w / s (Markstein's correction step).  That gives the SAME fp16 quotient as a correctly rounded fp32 one: the
// fp16 rounding changes only at midpoints m of fp16 values; writing w = W 2^a, s = S 2^b, m = M 2^c with W, S < 2^11 and
// M < 2^12, a quotient that is not m itself is off m by a relative 2^-23 at least (w - m s is a multiple of the smaller
// of 2^a and 2^(b+c), and m s < 2^(23+b+c)), more than q's error; and for w / s = m the correction returns m.
// Integer part without conversions: clamped to [-8, 7] (integers, so clamping before rounding is the same), adding
// 1544 = 1536 + 8 rounds to the nearest integer, ties to even, in the mantissa of a number in [1024, 2048).
// `bad` turns NaN when a quotient is not finite (zero or non-finite scale, overflow): the caller then redoes the word
// with quantize_exact.
__device__ __forceinline__ uint32_t quantize_pair(uint32_t w2, float s, float rs, __half2 &bad) {
  const float2 w = __half22float2(bits_h2(w2));
  const float qx = w.x * rs, qy = w.y * rs;
  const float x = fmaf(fmaf(-qx, s, w.x), rs, qx), y = fmaf(fmaf(-qy, s, w.y), rs, qy);
  const __half2 q = __floats2half2_rn(x, y);
  bad = __hfma2(q, bits_h2(0u), bad);
  const __half2 c = __hmax2(__hmin2(q, bits_h2(0x47004700u)), bits_h2(0xc800c800u));   // [-8, 7]
  return h2_bits(__hadd2(c, bits_h2(0x66086608u))) & 0x000f000fu;
}

// One warp packs 64 columns x 64 k (half a scale group of a 64-column block), without shared memory: lane 4 g + 2 r + u
// owns the columns g, g + 8, ..., g + 56 at k 4u..4u+3 and 8 + 4u..8 + 4u+3 of the 16-k rows r and r + 2.  Those are all the
// weights of the eight words t = 2u, 2u + 1 x j = 0..3, which lie next to each other (32 bytes): word (t, j) takes the
// pairs k = 2t, 2t+1 and 2t+8, 2t+9 of columns g + 16 j and g + 16 j + 8 (closed form of marlin.py:29-47), each pair one
// register of an 8-byte load.  The four warps of a block take neighbouring ranges of k: 512 contiguous bytes of each of
// 64 rows.  80 registers: six blocks, 96 KB of loads in flight per SM.
// Bound by HBM, with the conversions (15 instructions per two weights) close behind.  Measured, 22016 x 4096 (228 MB):
// 157 us -> 44 us (5.2 TB/s), 28672 x 16384 193 us (6.1 TB/s, 0.94 of the copy rate), 1024 x 3840 12.3 -> 7.0 us; the kernel
// before it gathered halves from shared memory and divided (its time depended on the data: 85 us without zeros).
// 128-k ranges per warp leave a longer last wave (45.6 / 9.0 us at the first and last size), 256-thread blocks
// 47 us; 16-byte loads of whole 16-k rows need 128 registers, 60 us.
constexpr int PACK_THREADS = 128, PACK_K = 64;

__global__ void __launch_bounds__(PACK_THREADS, 6)
    quantize_pack_kernel(const __half *__restrict__ w_nk, const __half *__restrict__ scales, int k, int n, int group, int groups,
                         bool vec_out, uint32_t *__restrict__ B, __half *__restrict__ s_packed) {
  const int k0 = (blockIdx.x * (PACK_THREADS / 32) + (threadIdx.x >> 5)) * PACK_K;
  if (k0 >= k) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, r = (lane >> 1) & 1, u = lane & 1;
  const int blk = blockIdx.y, n0 = blk * 64;
  const int sg = k0 / group;                            // group is 128 or k
  const __half *src = w_nk + (size_t)(n0 + g) * k + k0 + 16 * r + 4 * u;
  uint32_t *dst = B + (size_t)(k0 / 16 + r) * 2 * n + 128 * blk + 16 * g + 8 * u;
  uint2 lo[8], hi[8];
  auto load = [&](int h) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint2 *p = reinterpret_cast<const uint2 *>(src + (size_t)(8 * i) * k + 32 * h);
      lo[i] = __ldg(p), hi[i] = __ldg(p + 2);
    }
  };
  load(0);
  float s[8], rs[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __half sh = scales[(size_t)sg * n + n0 + g + 8 * i];
    s[i] = __half2float(sh), rs[i] = 1.0f / s[i];
    if (k0 == sg * group && (i & 3) == (lane & 3)) {
      // the first warp of a group: its scales, permuted (marlin.py:49-54): inside 64-column blocks, or 32 for a single row
      const int c64 = g + 8 * i, c32 = c64 & 31;
      const int pos = groups > 1 ? 8 * g + i : (c64 & 32) + 8 * ((c32 & 7) >> 1) + 2 * (c32 >> 3) + (c32 & 1);
      s_packed[(size_t)sg * n + n0 + pos] = sh;
    }
  }
#pragma unroll 1
  for (int h = 0; h < PACK_K / 32; ++h) {
    if (h) load(h);
    uint32_t word[2][4];   // [t - 2u][j]
    __half2 bad = bits_h2(0u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = 2 * j, b = 2 * j + 1;
      word[0][j] = quantize_pair(lo[a].x, s[a], rs[a], bad) | quantize_pair(hi[a].x, s[a], rs[a], bad) << 4 |
                   quantize_pair(lo[b].x, s[b], rs[b], bad) << 8 | quantize_pair(hi[b].x, s[b], rs[b], bad) << 12;
      word[1][j] = quantize_pair(lo[a].y, s[a], rs[a], bad) | quantize_pair(hi[a].y, s[a], rs[a], bad) << 4 |
                   quantize_pair(lo[b].y, s[b], rs[b], bad) << 8 | quantize_pair(hi[b].y, s[b], rs[b], bad) << 12;
    }
    if (!(__low2float(bad) == 0.0f && __high2float(bad) == 0.0f)) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          uint32_t v = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int col = 2 * j + (i >> 1);
            const uint2 q = i & 1 ? hi[col] : lo[col];
            const __half2 pair = bits_h2(t ? q.y : q.x);
            v |= quantize_exact(__low2half(pair), s[col]) << (4 * i);
            v |= quantize_exact(__high2half(pair), s[col]) << (4 * i + 16);
          }
          word[t][j] = v;
        }
    }
    uint32_t *out = dst + (size_t)(2 * h) * 2 * n;
    if (vec_out) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
        *reinterpret_cast<uint4 *>(out + 4 * t) = make_uint4(word[t][0], word[t][1], word[t][2], word[t][3]);
    } else {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[4 * t + j] = word[t][j];
    }
  }
}

}  // namespace

extern "C" int w4a16_quantize_pack_device(const void *weight_nk, const void *scales, int k, int n, int groupsize,
                                          void *B, void *s_packed, void *stream) {
  if (!weight_nk || !scales || !B || !s_packed) return W4A16_ERR_ARG;
  if (groupsize != -1 && groupsize != 128) return W4A16_ERR_KERN_SHAPE;      // marlin.py:70-71
  if (k <= 0 || n <= 0 || k % 128 || n % 256) return W4A16_ERR_PROB_SHAPE;   // marlin.py:72-73
  const int group = groupsize == -1 ? k : groupsize;
  const int groups = k / group;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (reinterpret_cast<uintptr_t>(weight_nk) & 15) return W4A16_ERR_ARG;   // the library's alignment of operands (rows are read 8 bytes at a time)
  quantize_pack_kernel<<<dim3((unsigned)((k / PACK_K + PACK_THREADS / 32 - 1) / (PACK_THREADS / 32)), (unsigned)(n / 64)), PACK_THREADS, 0, st>>>(
      static_cast<const __half *>(weight_nk), static_cast<const __half *>(scales), k, n, group, groups,
      !(reinterpret_cast<uintptr_t>(B) & 15), static_cast<uint32_t *>(B), static_cast<__half *>(s_packed));
  return cudaGetLastError() == cudaSuccess ? W4A16_OK : W4A16_ERR_CUDA;
}
