// First convolution of a small-channel network: 3x3 (any stride) on the 3-channel NCHW network input,
// 16 .. 64 output channels, folded batch-norm / bias and activation, written as NHWC in the
// executor's layout (MobileNetV3's `conv 3 -> 16, 3x3 stride 2 + BN + hard-swish`,
// tests/Nets/MobileNetV3.mlir:240-295).
//
// With 27 multiply-adds per output value and 3 input channels this layer is bound by HBM (one read
// of the NCHW input, one write of the output), and it does not fit the tensor-core kernels: as an
// implicit GEMM its K of 27 would be padded to 9 x 64 and its N of 16 to 64 (measured on the TMA-fed
// kernel: 821 us at batch 256, plus 109 us for the NCHW -> NHWC conversion in front of it).  Here one
// thread computes 16 output channels of one pixel straight from the NCHW input (a warp reads
// consecutive columns of a row), filter / scale / shift in shared memory read as broadcast vectors,
// fp32 accumulation on register pairs, and the conversion pass disappears.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "epilogue.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {

namespace {

constexpr int kCG = 16;   // output channels per thread

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long ra, rb, rc, rd;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}

template <typename T> __device__ __forceinline__ float ld(const T* p);
template <> __device__ __forceinline__ float ld<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ld<__half>(const __half* p) { return __half2float(__ldg(p)); }

__device__ __forceinline__ float act16(float x, int act) {
  switch (act) {
    case kActRelu: return !(x <= 0.0f) ? x : 0.0f;
    case kActHardSwish: {
      float t = (x + 3.0f) * 0.16666667f;
      t = (1.0f < t) ? 1.0f : t;
      t = (0.0f > t) ? 0.0f : t;
      return x * t;
    }
    case kActSilu: return x * __fdividef(1.0f, __expf(-x) + 1.0f);
    default: return x;
  }
}

template <typename TI, bool BF16>
__global__ void __launch_bounds__(256) stem3x3_kernel(const TI* __restrict__ src, const float* __restrict__ w,
                                                      const float* __restrict__ scale, const float* __restrict__ shift,
                                                      void* __restrict__ dst, Layout ol, int N, int H, int W, int OH, int OW, int Cout,
                                                      int stride, int pad, int act) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  extern __shared__ __align__(16) float sw[];     // [27][Cout] filter, [Cout] scale, [Cout] shift
  float* ssc = sw + 27 * Cout;
  float* ssh = ssc + Cout;
  for (int i = threadIdx.x; i < 27 * Cout; i += blockDim.x) {
    const int k = i / 27, t = i - k * 27;           // source [Cout][3][3][3]: t = (ci*3 + ky)*3 + kx
    sw[t * Cout + k] = w[i];
  }
  for (int c = threadIdx.x; c < Cout; c += blockDim.x) {
    ssc[c] = scale ? scale[c] : 1.0f;
    ssh[c] = shift ? shift[c] : 0.0f;
  }
  __syncthreads();
  const int groups = Cout / kCG;
  const unsigned total = (unsigned)N * OH * OW * groups;      // kept below 2^31 by the launcher
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    // the channel group is the slowest index: the threads of a warp share it and walk along a row
    const unsigned per = (unsigned)N * OH * OW;
    const int g = (int)(i / per);
    unsigned t = i - (unsigned)g * per;
    const unsigned t2 = t / (unsigned)OW;
    const int ox = (int)(t - t2 * OW);
    const int n = (int)(t2 / (unsigned)OH);
    const int oy = (int)(t2 - (unsigned)n * OH);
    float2 acc[kCG / 2];
#pragma unroll
    for (int e = 0; e < kCG / 2; ++e) acc[e] = make_float2(0.0f, 0.0f);
    const int ix0 = ox * stride - pad, iy0 = oy * stride - pad;
    // all 27 input values first (out-of-range taps read as zero without a branch), so that the loads are in
    // flight together; then the multiply-adds
    float in[27];
#pragma unroll
    for (int ci = 0; ci < 3; ++ci) {
      const TI* plane = src + ((size_t)n * 3 + ci) * H * W;
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        const int iy = iy0 + ky;
        const bool yin = (unsigned)iy < (unsigned)H;
        const TI* rowp = plane + (size_t)(yin ? iy : 0) * W;
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const int ix = ix0 + kx;
          const bool inb = yin && (unsigned)ix < (unsigned)W;
          const float v = ld<TI>(rowp + (inb ? ix : 0));
          in[(ci * 3 + ky) * 3 + kx] = inb ? v : 0.0f;
        }
      }
    }
#pragma unroll
    for (int t9 = 0; t9 < 27; ++t9) {
      const float2 v2 = make_float2(in[t9], in[t9]);
      const float* wp = sw + t9 * Cout + g * kCG;
#pragma unroll
      for (int e = 0; e < kCG / 2; e += 2) {
        const float4 w4 = *reinterpret_cast<const float4*>(wp + 2 * e);
        acc[e] = fma2(v2, make_float2(w4.x, w4.y), acc[e]);
        acc[e + 1] = fma2(v2, make_float2(w4.z, w4.w), acc[e + 1]);
      }
    }
    uint32_t o[kCG / 2];
#pragma unroll
    for (int e = 0; e < kCG / 2; ++e) {
      const float2 sc = *reinterpret_cast<const float2*>(ssc + g * kCG + 2 * e);
      const float2 sh = *reinterpret_cast<const float2*>(ssh + g * kCG + 2 * e);
      const float2 a = fma2(acc[e], sc, sh);
      const float x = act16(a.x, act), y = act16(a.y, act);
      if (BF16) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
        o[e] = *reinterpret_cast<const uint32_t*>(&b);
      } else {
        o[e] = ptx::pack_half2_sat(x, y);
      }
    }
    uint4* out = reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(dst) +
                                          (((size_t)n * ol.img_rows + oy + ol.off) * ol.pitch + ox + ol.off) * Cout + g * kCG);
    out[0] = make_uint4(o[0], o[1], o[2], o[3]);
    out[1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

// The same for stride 1 and 2, FOUR adjacent output pixels a thread.  With one pixel a thread the layer was bound by
// instructions: a broadcast load of the filter for every four packed multiply-adds, 27 guarded loads of the input and their
// addresses (146 us for MobileNetV3's first layer at batch 256, 180 MB: 28 us of HBM; the whole network 1234 us, with this
// kernel 1177).  Here a filter value serves four pixels, the input comes as one row of 3 * STRIDE + 3 values per (channel,
// filter row), and where rows are 16-byte aligned (VEC: stride 2, pad 1, W a multiple of 8) as 16-byte loads whose left
// neighbour arrives by shuffle.
constexpr int kPX = 4;

template <typename TI, bool VEC, int STRIDE>
__device__ __forceinline__ void input_row(const TI* rowp, bool yin, int ix0, int W, int gx, int lane, float (&v)[(kPX - 1) * STRIDE + 3]) {
  constexpr int NC = (kPX - 1) * STRIDE + 3;
  if constexpr (VEC) {
    // columns 8 gx - 1 .. 8 gx + 7; the first one is the last value of the lane before, a pad at the row's start
    if constexpr (sizeof(TI) == 2) {
      uint4 q = make_uint4(0, 0, 0, 0);
      if (yin) q = __ldg(reinterpret_cast<const uint4*>(rowp + 8 * gx));
      const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(h[e]);
        v[1 + 2 * e] = f.x;
        v[2 + 2 * e] = f.y;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (yin) q = __ldg(reinterpret_cast<const float4*>(rowp + 8 * gx) + e);
        v[1 + 4 * e] = q.x; v[2 + 4 * e] = q.y; v[3 + 4 * e] = q.z; v[4 + 4 * e] = q.w;
      }
    }
    float left = __shfl_up_sync(0xffffffffu, v[8], 1);
    if (lane == 0) left = yin && gx > 0 ? ld<TI>(rowp + 8 * gx - 1) : 0.0f;
    v[0] = gx > 0 ? left : 0.0f;
  } else {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const bool in = yin && (unsigned)(ix0 + c) < (unsigned)W;
      v[c] = in ? ld<TI>(rowp + ix0 + c) : 0.0f;
    }
  }
}

template <typename TI, bool BF16, bool VEC, int STRIDE>
__global__ void __launch_bounds__(256, 2) stem3x3_row_kernel(const TI* __restrict__ src, const float* __restrict__ w, const float* __restrict__ scale,
                                                          const float* __restrict__ shift, void* __restrict__ dst, Layout ol, int N, int H, int W,
                                                          int OH, int OW, int Cout, int pad, int act, int xgroups, long long total) {
  constexpr int NC = (kPX - 1) * STRIDE + 3;
  extern __shared__ __align__(16) float sw[];     // [27][Cout] filter, [Cout] scale, [Cout] shift
  float* ssc = sw + 27 * Cout;
  float* ssh = ssc + Cout;
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  for (int i = threadIdx.x; i < 27 * Cout; i += blockDim.x) {
    const int k = i / 27, t = i - k * 27;           // source [Cout][3][3][3]: t = (ci*3 + ky)*3 + kx
    sw[t * Cout + k] = w[i];
  }
  for (int c = threadIdx.x; c < Cout; c += blockDim.x) {
    ssc[c] = scale ? scale[c] : 1.0f;
    ssh[c] = shift ? shift[c] : 0.0f;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned per = (unsigned)(total / (Cout / kCG));   // pixel groups of one channel group
  // whole warps stay in the loop: the shuffle needs every lane
  for (long long i0 = (long long)blockIdx.x * blockDim.x; i0 < total; i0 += (long long)gridDim.x * blockDim.x) {
    const bool live = i0 + threadIdx.x < total;
    const unsigned i = (unsigned)(live ? i0 + threadIdx.x : total - 1);
    const int g = (int)(i / per);
    const unsigned t = i - (unsigned)g * per;
    const unsigned t2 = t / (unsigned)xgroups;
    const int gx = (int)(t - t2 * xgroups);
    const int n = (int)(t2 / (unsigned)OH), oy = (int)(t2 - (unsigned)n * OH);
    float2 acc[kPX][kCG / 2];
#pragma unroll
    for (int x = 0; x < kPX; ++x)
#pragma unroll
      for (int e = 0; e < kCG / 2; ++e) acc[x][e] = make_float2(0.0f, 0.0f);
    const int ix0 = gx * kPX * STRIDE - pad;
    const TI* img = src + (size_t)n * 3 * H * W;
#pragma unroll 1
    for (int ky = 0; ky < 3; ++ky) {
      const int iy = oy * STRIDE - pad + ky;
      const bool yin = (unsigned)iy < (unsigned)H;
      float v[3][NC];
#pragma unroll
      for (int ci = 0; ci < 3; ++ci) input_row<TI, VEC, STRIDE>(img + ((size_t)ci * H + (yin ? iy : 0)) * W, yin, ix0, W, gx, lane, v[ci]);
#pragma unroll
      for (int ci = 0; ci < 3; ++ci)
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const float* wp = sw + ((ci * 3 + ky) * 3 + kx) * Cout + g * kCG;
#pragma unroll
          for (int e = 0; e < kCG / 2; e += 2) {
            const float4 w4 = *reinterpret_cast<const float4*>(wp + 2 * e);
#pragma unroll
            for (int x = 0; x < kPX; ++x) {
              const float2 v2 = make_float2(v[ci][x * STRIDE + kx], v[ci][x * STRIDE + kx]);
              acc[x][e] = fma2(v2, make_float2(w4.x, w4.y), acc[x][e]);
              acc[x][e + 1] = fma2(v2, make_float2(w4.z, w4.w), acc[x][e + 1]);
            }
          }
        }
    }
    if (!live) continue;
#pragma unroll
    for (int x = 0; x < kPX; ++x) {
      const int ox = gx * kPX + x;
      if (ox >= OW) break;
      uint32_t o[kCG / 2];
#pragma unroll
      for (int e = 0; e < kCG / 2; ++e) {
        const float2 sc = *reinterpret_cast<const float2*>(ssc + g * kCG + 2 * e);
        const float2 sh = *reinterpret_cast<const float2*>(ssh + g * kCG + 2 * e);
        float2 a = fma2(acc[x][e], sc, sh);
        if (act == kActHardSwish) {   // a NaN stays NaN through the product
          a.x *= __saturatef(fmaf(a.x, 0.16666667f, 0.5f));
          a.y *= __saturatef(fmaf(a.y, 0.16666667f, 0.5f));
        } else {
          a.x = act16(a.x, act);
          a.y = act16(a.y, act);
        }
        if (BF16) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(a.x, a.y);
          o[e] = *reinterpret_cast<const uint32_t*>(&b);
        } else {
          o[e] = ptx::pack_half2_sat(a.x, a.y);
        }
      }
      ptx::stg_256(reinterpret_cast<unsigned short*>(dst) + (((size_t)n * ol.img_rows + oy + ol.off) * ol.pitch + ox + ol.off) * Cout + g * kCG, o);
    }
  }
}

// fp16 images and an fp16 filter, stride 2, pad 1, W a multiple of 8: the tensor cores' (mma.sync) work.  On the fma pipe the 27 x 16
// multiply-adds of a pixel bound the layer: 80 us at batch 256 (224 x 224 -> 16 channels, 180 MB, 28 us of HBM), 46 us here.  tcgen05
// would need the windows laid out in shared memory; an A fragment of mma.sync takes them as they lie in the rows of the image.
// K: the nine (channel, filter row) pairs, four columns of the input each -- two aligned words, of which the first value is no tap and
// is cleared, so that an infinity or NaN there does not reach the sum.  A warp computes 16 adjacent pixels x 16 channels: the columns of
// the two 8-channel halves are dealt so that a thread ends up with four adjacent channels, 8 bytes to store.  Products are exact, sums
// fp32, as before.  The rows come to shared memory as bulk copies, three (one a channel) for kRowsOut rows of output, the next ones while
// these are computed: read straight from global memory, in words, too few bytes were on their way (77 us).
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b));
}

constexpr int kRowsOut = 4, kRowsIn = 2 * kRowsOut + 1;   // rows of output and input a block works on at a time
constexpr int kMmaThreads = 256;

__device__ __forceinline__ uint32_t lds(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

template <bool BF16, bool HSWISH>
__global__ void __launch_bounds__(kMmaThreads, 4) stem3x3_mma_kernel(const __half* __restrict__ src, const float* __restrict__ w, const float* __restrict__ scale,
                                                          const float* __restrict__ shift, void* __restrict__ dst, Layout ol, int H, int W,
                                                          int OH, int OW, int Cout, int act, epi::FastDiv div_groups, epi::FastDiv div_x, int units,
                                                          int* error_flag) {
  extern __shared__ __align__(128) uint8_t rows_raw[];   // 16 bytes, two stages of [channel][kRowsIn][W] halves, 128 bytes
  __shared__ __align__(8) unsigned long long s_full[2];
  const uint32_t rows0 = ptx::smem_u32(rows_raw) + 16u, full = ptx::smem_u32(s_full);
  const int row_bytes = 2 * W, stage_bytes = 3 * kRowsIn * row_bytes;
  if (threadIdx.x == 0) {
    ptx::mbar_init(full, 1);
    ptx::mbar_init(full + 8, 1);
    ptx::mbar_fence_init();
  }
  __syncthreads();
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, c0 = (int)blockIdx.y * kCG;
  // step s (16 k values), half h (8 of them): k = 2t, 2t + 1 of the half are columns 2 (t & 1), + 1 of input row j = 4s + 2h + t / 2
  uint32_t b[5][2];       // [2s + h][half of the channels]
  int row[5];             // where row j lies in a stage, bytes from the output row's first input row
  unsigned top = 0, bottom = 0;   // bit 2s + h: row j is the one above, the one below
#pragma unroll
  for (int sh = 0; sh < 5; ++sh) {
    const int j = 2 * sh + (t >> 1), ci = j / 3, ky = j - 3 * ci;
    row[sh] = j < 9 ? (ci * kRowsIn + ky) * row_bytes : 0;   // there is no tenth: what is read there is cleared
    if (ky == 0) top |= 1u << sh;
    if (ky == 2) bottom |= 1u << sh;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int ch = c0 + 4 * (g >> 1) + 2 * q + (g & 1);   // column g of half q
      __half2 v = __floats2half2_rn(0.0f, 0.0f);
      if (j < 9) {
        const float* wp = w + ch * 27 + j * 3;
        v = (t & 1) ? __floats2half2_rn(wp[1], wp[2]) : __floats2half2_rn(0.0f, wp[0]);
      }
      b[sh][q] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
  const bool ninth = t < 2;   // the last step holds one row: the other threads' is none
  const uint32_t taps = (t & 1) ? 0xffffffffu : 0xffff0000u;
  float sc[4], sf[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    sc[e] = scale ? scale[c0 + 4 * t + e] : 1.0f;
    sf[e] = shift ? shift[c0 + 4 * t + e] : 0.0f;
  }
  unsigned short* const out_first = reinterpret_cast<unsigned short*>(dst) + ((long long)ol.off * ol.pitch + ol.off) * Cout + c0 + 4 * t;
  const int warp = threadIdx.x >> 5;
  auto fetch = [&](int u, int st) {   // one thread: the rows under output rows oy0 ..
    const int n = (int)epi::div_by((uint32_t)u, div_groups), iy = 2 * kRowsOut * (u - n * (int)div_groups.d) - 1;
    const int lo = max(iy, 0), hi = min(iy + kRowsIn, H);
    const uint32_t bytes = (uint32_t)((hi - lo) * row_bytes);
    ptx::mbar_arrive_expect_tx(full + 8 * st, 3 * bytes);
    for (int ci = 0; ci < 3; ++ci)
      ptx::bulk_g2s(rows0 + (uint32_t)(st * stage_bytes + (ci * kRowsIn + lo - iy) * row_bytes), src + ((size_t)(n * 3 + ci) * H + lo) * W, bytes, full + 8 * st);
  };
  if (threadIdx.x == 0 && (int)blockIdx.x < units) fetch((int)blockIdx.x, 0);
  uint32_t turn = 0;   // stages waited for
  for (int u = (int)blockIdx.x; u < units; u += (int)gridDim.x, ++turn) {
    const uint32_t st = turn & 1u;
    if (threadIdx.x == 0 && u + (int)gridDim.x < units) fetch(u + (int)gridDim.x, (int)(st ^ 1u));
    if (__syncthreads_or(!ptx::mbar_wait(full + 8 * st, (turn >> 1) & 1u))) {
      if (threadIdx.x == 0) {
        if (error_flag) atomicCAS(error_flag, 0, (int)kErrWaitProducer);
        ptx::mbar_wait(full + 8 * st, (turn >> 1) & 1u);   // once more: no copy may outlive its shared memory
        if (u + (int)gridDim.x < units) ptx::mbar_wait(full + 8 * (st ^ 1u), ((turn + 1) >> 1) & 1u);
      }
      break;
    }
    const int n = (int)epi::div_by((uint32_t)u, div_groups), oy0 = kRowsOut * (u - n * (int)div_groups.d), rows = min(kRowsOut, OH - oy0);
    const int tiles = rows * (int)div_x.d;
    const uint32_t stage = rows0 + st * (uint32_t)stage_bytes + 4u * (uint32_t)(g + (t & 1)) - 4u;
    // the warps take turns with the first tile, so that a remainder does not always fall to the same ones
    for (int k = (warp + (int)turn * 4) & 7; k < tiles; k += kMmaThreads / 32) {
      const int ry = (int)epi::div_by((uint32_t)k, div_x), oy = oy0 + ry, x0 = (k - ry * (int)div_x.d) * 16, px = x0 + g;
      // words px - 1 (t even) and px (t odd) of a row; pixel px + 8 eight words on.  Past the right edge lies other data, which only
      // reaches pixels that are not stored; on the left edge and in rows outside the image zeros take its place.
      const uint32_t at = stage + (uint32_t)(2 * ry * row_bytes + 4 * x0);
      uint32_t v[5][2];
#pragma unroll
      for (int sh = 0; sh < 5; ++sh) {
        v[sh][0] = lds(at + (uint32_t)row[sh]);
        v[sh][1] = lds(at + (uint32_t)row[sh] + 32u);
      }
      const uint32_t left = px == 0 && !(t & 1) ? 0u : taps;
#pragma unroll
      for (int sh = 0; sh < 4; ++sh) {
        v[sh][0] &= left;
        v[sh][1] &= taps;
      }
      v[4][0] &= ninth ? left : 0u;
      v[4][1] &= ninth ? taps : 0u;
      if (oy == 0 || 2 * oy + 1 >= H) {
        const unsigned out = (oy == 0 ? top : 0u) | (2 * oy + 1 >= H ? bottom : 0u);
#pragma unroll
        for (int sh = 0; sh < 5; ++sh)
          if (out >> sh & 1u) v[sh][0] = v[sh][1] = 0u;
      }
      float d[2][4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        d[q][0] = d[q][1] = d[q][2] = d[q][3] = 0.0f;
#pragma unroll
        for (int s = 0; s < 2; ++s)
          mma16(d[q], {v[2 * s][0], v[2 * s][1], v[2 * s + 1][0], v[2 * s + 1][1]}, {b[2 * s][q], b[2 * s + 1][q]});
        mma8(d[q], v[4][0], v[4][1], b[4][q]);
      }
      unsigned short* to = out_first + (((long long)n * ol.img_rows + oy) * ol.pitch + px) * Cout;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float a = fmaf(d[e >> 1][2 * h + (e & 1)], sc[e], sf[e]);
          y[e] = HSWISH ? a * __saturatef(fmaf(a, 0.16666667f, 0.5f)) : act16(a, act);
        }
        uint2 o;
        if (BF16) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[1]), hi = __floats2bfloat162_rn(y[2], y[3]);
          o = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
          o = make_uint2(ptx::pack_half2_sat(y[0], y[1]), ptx::pack_half2_sat(y[2], y[3]));
        }
        if (px + 8 * h < OW) *reinterpret_cast<uint2*>(to + 8 * h * Cout) = o;
      }
    }
    __syncthreads();   // the stage may be filled again
  }
}

template <typename TI, bool BF16>
cudaError_t launch_row(const TI* src, const float* w, const float* scale, const float* shift, void* dst, Layout ol, int N, int H, int W, int OH,
                       int OW, int Cout, int stride, int pad, int act, cudaStream_t st) {
  const int xg = (OW + kPX - 1) / kPX;
  const long long total = (long long)N * OH * xg * (Cout / kCG);
  const bool vec = stride == 2 && pad == 1 && W % 8 == 0 && !(reinterpret_cast<uintptr_t>(src) & 15);   // then OW == W / 2
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 2) blocks = 148 * 2;   // two blocks a SM (registers): the filter is loaded once
  const size_t smem = (size_t)29 * Cout * sizeof(float);
  auto go = [&](auto kern) {
    return launch_pdl(kern, dim3((unsigned)blocks), dim3(256), smem, st, src, w, scale, shift, dst, ol, N, H, W, OH, OW, Cout, pad, act, xg, total);
  };
  if (vec) return go(stem3x3_row_kernel<TI, BF16, true, 2>);
  return stride == 2 ? go(stem3x3_row_kernel<TI, BF16, false, 2>) : go(stem3x3_row_kernel<TI, BF16, false, 1>);
}

}  // namespace

bool stem3x3_supported(int Cin, int Cout, int R, int S, DType act_dt, int act) {
  return Cin == 3 && R == 3 && S == 3 && Cout % kCG == 0 && Cout >= kCG && Cout <= 64 && act_dt != kF32 &&
         (act == kActNone || act == kActRelu || act == kActHardSwish || act == kActSilu);
}

cudaError_t launch_stem3x3(const void* src, DType src_dt, const float* w, const float* scale, const float* shift, void* dst, DType dt,
                           Layout out_l, int N, int H, int W, int Cout, int stride, int pad, int act, int w_f16, int* error_flag, cudaStream_t st) {
  if (!stem3x3_supported(3, Cout, 3, 3, dt, act) || src_dt == kBF16 || stride < 1 || pad < 0) return cudaErrorInvalidValue;
  const int OH = (H + 2 * pad - 3) / stride + 1, OW = (W + 2 * pad - 3) / stride + 1;
  if (OH <= 0 || OW <= 0) return cudaErrorInvalidValue;
  if (out_l.pitch == 0) out_l = dense_layout(OH, OW);
  const long long total = (long long)N * OH * OW * (Cout / kCG);
  if (total >= (1LL << 31) - (1LL << 21)) return cudaErrorInvalidValue;
  // operands that fp16 holds exactly, rows that bulk copies can take (then OW == W / 2), two stages of them in a quarter of an SM's memory
  const size_t rows_smem = (size_t)2 * 3 * kRowsIn * 2 * W + 144;
  if (src_dt == kF16 && w_f16 && stride == 2 && pad == 1 && W % 8 == 0 && rows_smem <= 48 * 1024 && !(reinterpret_cast<uintptr_t>(src) & 15)) {
    const int groups = (OH + kRowsOut - 1) / kRowsOut, units = N * groups;
    const dim3 grid((unsigned)(units < 148 * 4 ? units : 148 * 4), (unsigned)(Cout / kCG));
    auto go = [&](auto kern) {
      return launch_pdl(kern, grid, dim3(kMmaThreads), rows_smem, st, (const __half*)src, w, scale, shift, dst, out_l, H, W, OH, OW, Cout, act,
                        epi::fast_div((uint32_t)groups), epi::fast_div((uint32_t)((OW + 15) / 16)), units, error_flag);
    };
    if (act == kActHardSwish) return dt == kBF16 ? go(stem3x3_mma_kernel<true, true>) : go(stem3x3_mma_kernel<false, true>);
    return dt == kBF16 ? go(stem3x3_mma_kernel<true, false>) : go(stem3x3_mma_kernel<false, false>);
  }
  if (stride <= 2) {   // wider strides share no input between neighbours
    if (src_dt == kF32)
      return dt == kBF16 ? launch_row<float, true>((const float*)src, w, scale, shift, dst, out_l, N, H, W, OH, OW, Cout, stride, pad, act, st)
                         : launch_row<float, false>((const float*)src, w, scale, shift, dst, out_l, N, H, W, OH, OW, Cout, stride, pad, act, st);
    return dt == kBF16 ? launch_row<__half, true>((const __half*)src, w, scale, shift, dst, out_l, N, H, W, OH, OW, Cout, stride, pad, act, st)
                       : launch_row<__half, false>((const __half*)src, w, scale, shift, dst, out_l, N, H, W, OH, OW, Cout, stride, pad, act, st);
  }
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  const size_t smem = (size_t)29 * Cout * sizeof(float);
#define NNCV_ST(TI, BF) \
  launch_pdl(stem3x3_kernel<TI, BF>, dim3((unsigned)blocks), dim3(256), smem, st, (const TI*)src, w, scale, shift, dst, out_l, N, H, W, OH, OW, Cout, stride, pad, act)
  if (src_dt == kF32) { if (dt == kBF16) NNCV_ST(float, true); else NNCV_ST(float, false); }
  else { if (dt == kBF16) NNCV_ST(__half, true); else NNCV_ST(__half, false); }
#undef NNCV_ST
  return cudaGetLastError();
}

}  // namespace nncv_b200
