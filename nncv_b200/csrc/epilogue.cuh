// Shared parts of the tensor-core convolutions' epilogue.
//
// The accumulator of a tile leaves through EIGHT INDEPENDENT WARPS: each owns 32 accumulator rows (its TMEM lane
// quadrant) of every second 128-byte-wide slab and has its own staging buffers, its own bulk-store group and its own
// barriers for residual rows that TMA brings into the staging buffer ahead of time.  Nothing in the loop synchronises
// more than one warp.  (With block-wide barriers around every slab -- the earlier form: 256 threads converting one
// 128 x 64 slab, a store by one thread, and a barrier on either side -- a slab cost 1.7 to 1.8 us of latency whatever
// its size, and that, not HBM or the tensor pipe, set the time of every convolution with a short reduction.)
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {
namespace epi {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kBufBytes = 32 * 128;    // 32 rows of 128 bytes: one warp's part of a slab
constexpr int kMaxBufs = 3;

__device__ __forceinline__ unsigned long long pk(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpk(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// two fused multiply-adds in one instruction, each rounded like fmaf
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ float2 unpack16(uint32_t w, bool bf16) {
  if (bf16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// 16-bit pair with optional ReLU folded into the conversion (negative -> +0, a NaN stays NaN, like cmpf ugt + select);
// fp16 saturates.
__device__ __forceinline__ uint32_t pack16(float a, float b, bool bf16, bool relu) {
  if (bf16) {
    if (relu) return ptx::pack_bf162_relu(a, b);
    const __nv_bfloat162 x = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&x);
  }
  return relu ? ptx::pack_half2_sat_relu(a, b) : ptx::pack_half2_sat(a, b);
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Scale and shift of a slab, fetched by the warp before it needs them (lane l: columns 2l and 2l + 1) and spread
// through shared memory as {scale, scale, shift, shift} of a column pair: the operands of one packed multiply-add.
struct ColParams { float s0, s1, h0, h1; };
__device__ __forceinline__ ColParams fetch_cols(const float* scale, const float* shift, int col, int Kout, int lane) {
  ColParams c{1.0f, 1.0f, 0.0f, 0.0f};
  const int n = col + 2 * lane;
  if (n < Kout) {
    if (scale) c.s0 = __ldg(scale + n);
    if (shift) c.h0 = __ldg(shift + n);
  }
  if (n + 1 < Kout) {
    if (scale) c.s1 = __ldg(scale + n + 1);
    if (shift) c.h1 = __ldg(shift + n + 1);
  }
  return c;
}
__device__ __forceinline__ void put_cols(uint32_t tab, const ColParams& c, int lane) {
  sts128(tab + (uint32_t)lane * 16u, __float_as_uint(c.s0), __float_as_uint(c.s1), __float_as_uint(c.h0), __float_as_uint(c.h1));
}

// What happens to a row between the accumulator and the staging buffer.  Each combination is a function of its own: with
// the choices tested per element the conversion of a 128 x 64 slab took 840 instructions a warp and, at two warps a
// scheduler, 6000 clocks; this bound every convolution with a short reduction.
enum Mode : int { kModeBf16 = 1, kModeRes = 2, kModeActShift = 2 };   // act: 0 none, 1 ReLU, 2 hard-swish, 3 SiLU
inline __host__ __device__ int mode_of(bool bf16, bool res, bool relu, int act) {
  const int a = act == kActHardSwish ? 2 : (act == kActSilu ? 3 : (relu ? 1 : 0));
  return (bf16 ? kModeBf16 : 0) | (res ? kModeRes : 0) | (a << kModeActShift);
}

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// One row's 64 accumulator columns -> scale / shift (+ residual, read from the staging row) (+ activation) -> the 128-byte
// staging row, 16-byte chunks XOR-swizzled by the row.  Sixteen columns at a time, the next sixteen's scale, shift and
// residual on their way from shared memory meanwhile.
template <bool BF16, bool RES, int ACT>
__device__ __forceinline__ void row64(const uint32_t (&acc)[64], uint32_t tab, uint32_t srow, uint32_t sw) {
  uint4 t[2][8], r[2][2];
  auto load = [&](int c, int s) {
#pragma unroll
    for (int h = 0; h < 8; ++h) t[s][h] = lds128(tab + (uint32_t)(c * 8 + h) * 16u);
    if (RES) {
      r[s][0] = lds128(srow + (((uint32_t)(2 * c) ^ sw) << 4));
      r[s][1] = lds128(srow + (((uint32_t)(2 * c + 1) ^ sw) << 4));
    }
  };
  load(0, 0);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int s = c & 1;
    if (c < 3) load(c + 1, s ^ 1);
    uint32_t o[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const uint4 q = t[s][h];
      unsigned long long v = fma2(pk(__uint_as_float(acc[c * 16 + 2 * h]), __uint_as_float(acc[c * 16 + 2 * h + 1])),
                                  pk(__uint_as_float(q.x), __uint_as_float(q.y)), pk(__uint_as_float(q.z), __uint_as_float(q.w)));
      if (RES) {
        const uint4 w4 = r[s][h >> 2];
        const uint32_t w = (h & 3) == 0 ? w4.x : ((h & 3) == 1 ? w4.y : ((h & 3) == 2 ? w4.z : w4.w));
        const float2 f = unpack16(w, BF16);
        v = add2(v, pk(f.x, f.y));
      }
      float a, b;
      unpk(v, a, b);
      // hard-swish x * min(max(x + 3, 0), 6) / 6 or SiLU x / (1 + exp(-x)); a NaN stays NaN through the product with x
      if (ACT == 2) {
        a *= __saturatef(fmaf(a, 0.16666667f, 0.5f));
        b *= __saturatef(fmaf(b, 0.16666667f, 0.5f));
      } else if (ACT == 3) {
        a *= __fdividef(1.0f, __expf(-a) + 1.0f);
        b *= __fdividef(1.0f, __expf(-b) + 1.0f);
      }
      o[h] = pack16(a, b, BF16, ACT == 1);
    }
    sts128(srow + (((uint32_t)(2 * c) ^ sw) << 4), o[0], o[1], o[2], o[3]);
    sts128(srow + (((uint32_t)(2 * c + 1) ^ sw) << 4), o[4], o[5], o[6], o[7]);
  }
}

// ACTS: the highest activation a kernel needs (1: none or ReLU, 3: all).
template <int ACTS>
__device__ __forceinline__ void row64_by_mode(int mode, const uint32_t (&acc)[64], uint32_t tab, uint32_t srow, uint32_t sw) {
#define NNCV_ROW(B_, R_, A_) \
  case (B_ ? kModeBf16 : 0) | (R_ ? kModeRes : 0) | (A_ << kModeActShift): row64<B_, R_, A_>(acc, tab, srow, sw); break;
  switch (mode) {
    NNCV_ROW(false, false, 0) NNCV_ROW(false, false, 1) NNCV_ROW(false, true, 0) NNCV_ROW(false, true, 1)
    NNCV_ROW(true, false, 0) NNCV_ROW(true, false, 1) NNCV_ROW(true, true, 0) NNCV_ROW(true, true, 1)
    default:
      if constexpr (ACTS > 1) {
        switch (mode) {
          NNCV_ROW(false, false, 2) NNCV_ROW(false, true, 2) NNCV_ROW(true, false, 2) NNCV_ROW(true, true, 2)
          NNCV_ROW(false, false, 3) NNCV_ROW(false, true, 3) NNCV_ROW(true, false, 3) NNCV_ROW(true, true, 3)
          default: break;
        }
      }
      break;
  }
#undef NNCV_ROW
}

// fp32 results: 32 columns fill the 128-byte row.
template <bool RELU>
__device__ __forceinline__ void row32_f32(const uint32_t (&acc)[32], uint32_t tab, uint32_t srow, uint32_t sw) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint4 t[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) t[h] = lds128(tab + (uint32_t)(c * 8 + h) * 16u);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float v[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 q = t[2 * g + h];
        const int e = c * 16 + g * 4 + 2 * h;
        unpk(fma2(pk(__uint_as_float(acc[e]), __uint_as_float(acc[e + 1])), pk(__uint_as_float(q.x), __uint_as_float(q.y)),
                  pk(__uint_as_float(q.z), __uint_as_float(q.w))),
             v[2 * h], v[2 * h + 1]);
      }
      if (RELU) {
#pragma unroll
        for (int h = 0; h < 4; ++h) v[h] = !(v[h] <= 0.0f) ? v[h] : 0.0f;
      }
      sts128(srow + (((uint32_t)(c * 4 + g) ^ sw) << 4), __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]),
             __float_as_uint(v[3]));
    }
  }
}

// A row that is a pad slot leaves as zeros.
__device__ __forceinline__ void zero_row(uint32_t srow) {
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) sts128(srow + (c << 4), 0u, 0u, 0u, 0u);
}

// n / d for 0 <= n < 2^31 without a division.
struct FastDiv {
  uint32_t d, mul, shift;
};
inline FastDiv fast_div(uint32_t d) {
  FastDiv f{d, 0, 0};
  if (d > 1) {
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;                                   // ceil(log2 d) >= 1
    f.mul = (uint32_t)(((1ull << (31 + l)) / d) + 1);
    f.shift = l - 1;
  }
  return f;
}
__device__ __forceinline__ uint32_t div_by(uint32_t n, const FastDiv& f) { return f.d == 1 ? n : __umulhi(n, f.mul) >> f.shift; }

// Host: staging buffers per epilogue warp.  With a residual three (its rows are requested two slabs ahead of their use)
// or two, without one two or one, the larger count only while `want` bytes of operand stages stay beside it; where not
// even `need` bytes would, a single buffer (a residual row is then waited for in full).
inline int pick_bufs(bool residual, size_t limit, size_t want, size_t need) {
  const int least = residual ? 2 : 1;
  for (int bufs = residual ? 3 : 2; bufs >= least; --bufs)
    if ((size_t)bufs * kWarps * kBufBytes + want <= limit) return bufs;
  return (size_t)least * kWarps * kBufBytes + need <= limit ? least : 1;
}

}  // namespace epi
}  // namespace nncv_b200
