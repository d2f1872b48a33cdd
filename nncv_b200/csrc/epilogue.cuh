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
__device__ __forceinline__ float lds32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
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

// A warp's 32 x 64 accumulator slab -> scale / shift (+ residual, read from the staging buffer) (+ activation) -> the staging
// buffer's rows of 128 bytes, 16-byte chunks XOR-swizzled by the row.
//
// The slab is held as matrix fragments (ptx::tmem_ld_16x64, rows 0-15 in acc[0..31], rows 16-31 after), so a thread owns the
// same sixteen columns in all of its four rows and reads 8 x 16 bytes of scale and shift a slab; residual and result pass
// through ldmatrix / stmatrix.  With a row a thread (32 lanes x 64 columns) every thread read all 32 x 16 bytes: at four clocks
// a 16-byte read 2048 clocks of the shared-memory port for a 128 x 256 tile, beside which TMA and the tensor core, which use the
// same port, waited.  ResNet-50 at batch 512, before and now, us: 64 -> 256 pointwise 219 185, with residual 301 285, 128 -> 512
// 180 163, 256 -> 1024 116 103, 512 -> 2048 70 64, 64 -> 64 3x3 107 105.
__device__ __forceinline__ void load_slab(uint32_t taddr, uint32_t (&acc)[64]) {
  ptx::tmem_ld_16x64<0>(taddr, acc);
  ptx::tmem_ld_16x64<32>(taddr + (16u << 16), acc);
}
template <bool BF16, bool RES, int ACT>
__device__ __forceinline__ void slab64(const uint32_t (&acc)[64], uint32_t tab, uint32_t buf, int lane) {
  const uint32_t row = buf + (uint32_t)(lane & 15) * 128u, hi = (uint32_t)(lane >> 4), sw = (uint32_t)(lane & 7);
  const uint32_t t0 = tab + (uint32_t)(lane & 3) * 16u;
  uint4 t[2][2];
  uint32_t r[2][2][4];
  auto load = [&](int c, int s) {   // column groups 2c and 2c + 1
    t[s][0] = lds128(t0 + (uint32_t)(2 * c) * 64u);
    t[s][1] = lds128(t0 + (uint32_t)(2 * c + 1) * 64u);
    if (RES) {
      ptx::ldmatrix4(row + ((((uint32_t)(2 * c)) | hi) ^ sw) * 16u, r[s][0]);
      ptx::ldmatrix4(row + 16u * 128u + ((((uint32_t)(2 * c)) | hi) ^ sw) * 16u, r[s][1]);
    }
  };
  load(0, 0);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int s = c & 1;
    if (c < 3) load(c + 1, s ^ 1);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {   // group 2c: rows 0-7, rows 8-15; group 2c + 1 likewise
        const uint4 q = t[s][e >> 1];
        const int at = h * 32 + (2 * c + (e >> 1)) * 4 + (e & 1) * 2;
        unsigned long long v = fma2(pk(__uint_as_float(acc[at]), __uint_as_float(acc[at + 1])), pk(__uint_as_float(q.x), __uint_as_float(q.y)),
                                    pk(__uint_as_float(q.z), __uint_as_float(q.w)));
        if (RES) {
          const float2 f = unpack16(r[s][h][e], BF16);
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
        o[e] = pack16(a, b, BF16, ACT == 1);
      }
      ptx::stmatrix4(row + (uint32_t)h * 16u * 128u + ((((uint32_t)(2 * c)) | hi) ^ sw) * 16u, o[0], o[1], o[2], o[3]);
    }
  }
}

// ACTS: the highest activation a kernel needs (1: none or ReLU, 3: all).
template <int ACTS>
__device__ __forceinline__ void slab64_by_mode(int mode, const uint32_t (&acc)[64], uint32_t tab, uint32_t buf, int lane) {
#define NNCV_SLAB(B_, R_, A_) \
  case (B_ ? kModeBf16 : 0) | (R_ ? kModeRes : 0) | (A_ << kModeActShift): slab64<B_, R_, A_>(acc, tab, buf, lane); break;
  switch (mode) {
    NNCV_SLAB(false, false, 0) NNCV_SLAB(false, false, 1) NNCV_SLAB(false, true, 0) NNCV_SLAB(false, true, 1)
    NNCV_SLAB(true, false, 0) NNCV_SLAB(true, false, 1) NNCV_SLAB(true, true, 0) NNCV_SLAB(true, true, 1)
    default:
      if constexpr (ACTS > 1) {
        switch (mode) {
          NNCV_SLAB(false, false, 2) NNCV_SLAB(false, true, 2) NNCV_SLAB(true, false, 2) NNCV_SLAB(true, true, 2)
          NNCV_SLAB(false, false, 3) NNCV_SLAB(false, true, 3) NNCV_SLAB(true, false, 3) NNCV_SLAB(true, true, 3)
          default: break;
        }
      }
      break;
  }
#undef NNCV_SLAB
}

// fp32 results: 32 columns fill the 128-byte row.  Rows 0-15 of the slab in acc[0..15], rows 16-31 in acc[16..31].
__device__ __forceinline__ void load_slab_f32(uint32_t taddr, uint32_t (&acc)[64]) {
  ptx::tmem_ld_16x32<0>(taddr, acc);
  ptx::tmem_ld_16x32<16>(taddr + (16u << 16), acc);
}
template <bool RELU>
__device__ __forceinline__ void slab32_f32(const uint32_t (&acc)[64], uint32_t tab, uint32_t buf, int lane) {
  const uint32_t row = buf + (uint32_t)(lane & 15) * 128u, hi = (uint32_t)(lane >> 4), sw = (uint32_t)(lane & 7);
  const uint32_t t0 = tab + (uint32_t)((lane >> 1) & 1) * 16u + (uint32_t)(lane & 1) * 4u;
  float s[8], h[8];
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    s[g] = lds32(t0 + (uint32_t)g * 32u);
    h[g] = lds32(t0 + (uint32_t)g * 32u + 8u);
  }
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int c = 0; c < 4; ++c) {   // column groups 2c and 2c + 1 of four
      float v[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int g = 2 * c + e, at = half * 16 + 2 * g;
        unpk(fma2(pk(__uint_as_float(acc[at]), __uint_as_float(acc[at + 1])), pk(s[g], s[g]), pk(h[g], h[g])), v[2 * e], v[2 * e + 1]);
      }
      if (RELU) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = !(v[e] <= 0.0f) ? v[e] : 0.0f;
      }
      ptx::stmatrix4(row + (uint32_t)half * 16u * 128u + ((((uint32_t)(2 * c)) | hi) ^ sw) * 16u, __float_as_uint(v[0]), __float_as_uint(v[1]),
                     __float_as_uint(v[2]), __float_as_uint(v[3]));
    }
}

// Rows that are pad slots (keep: lane l's row l is none) leave as zeros.
__device__ __forceinline__ void zero_pads(uint32_t buf, int lane, bool keep) {
  if (__all_sync(0xffffffffu, keep)) return;
  __syncwarp();   // other lanes wrote the row
  if (keep) return;
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) sts128(buf + (uint32_t)lane * 128u + (c << 4), 0u, 0u, 0u, 0u);
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
