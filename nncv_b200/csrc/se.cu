// Squeeze-and-excitation of a network in one kernel, in place (tests/Nets/MobileNetV3.mlir:319-389):
//   pooled = mean over pixels;  gate = hard_sigmoid(W2 relu(W1 pooled + b1) + b2);  x *= gate.
//
// As three kernels (pool, gate, scaling) the nine blocks of MobileNetV3 took 361 of 1115 us at batch 256 and, at small
// batches, 27 launches of a few microseconds each; now 213 of 913.  Here a cluster of eight CTAs owns one, two or four images
// from beginning to end: the map is read from L2 twice and written once, and what the CTAs exchange (pixel sums, hidden values,
// gates) goes through distributed shared memory.  With few images each CTA keeps its eighth of both matrices in shared memory,
// copied before the previous kernel of the stream has ended (read from L2 as they were needed, 576 -> 144 -> 576 took 30 us at
// batch 4, most of it latency); with many they are read from L2, once for the images of the cluster (50 us at batch 256 with one
// row a warp at a time, now 29).
//
// An image's pixels are always cut into the same eight slices, the slices added pairwise, whatever the number of images a
// cluster owns: an image's result does not depend on the batch it came in.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "epilogue.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {

namespace cg = cooperative_groups;

namespace {

constexpr int kCluster = 8, kThreads = 256, kWarps = kThreads / 32;
constexpr size_t kMaxSmem = 200 * 1024, kShareSmem = 54 * 1024;   // of a CTA; of one of the four an SM holds

template <typename T> struct Vec8;   // a 16-byte vector as fp32 values
template <> struct Vec8<float> {
  static constexpr int V = 4;
  static __device__ __forceinline__ void load(const uint4& r, float (&f)[4]) {
    f[0] = __uint_as_float(r.x); f[1] = __uint_as_float(r.y); f[2] = __uint_as_float(r.z); f[3] = __uint_as_float(r.w);
  }
  static __device__ __forceinline__ uint4 store(const float (&f)[4]) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
};
template <bool BF16> struct Vec16 {
  static constexpr int V = 8;
  static __device__ __forceinline__ void load(const uint4& r, float (&f)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 p = epi::unpack16(w[e], BF16);
      f[2 * e] = p.x;
      f[2 * e + 1] = p.y;
    }
  }
  static __device__ __forceinline__ uint4 store(const float (&f)[8]) {
    return make_uint4(epi::pack16(f[0], f[1], BF16, false), epi::pack16(f[2], f[3], BF16, false), epi::pack16(f[4], f[5], BF16, false),
                      epi::pack16(f[6], f[7], BF16, false));
  }
};
template <> struct Vec8<__half> : Vec16<false> {};
template <> struct Vec8<__nv_bfloat16> : Vec16<true> {};

// The clamps pass a NaN on, as the fixture's cmpf / select pairs do.
template <typename T>
__device__ __forceinline__ float hard_sigmoid(float x) {
  float t = sizeof(T) == 4 ? (x + 3.0f) / 6.0f : (x + 3.0f) * 0.16666667f;
  t = (1.0f < t) ? 1.0f : t;
  return (0.0f > t) ? 0.0f : t;
}

struct SeParams {
  const float *w1, *b1, *w2, *b2;
  Layout l;
  int N, H, W, C, Cr;
  epi::FastDiv div_w;
  int* error_flag;
};

// `rows` rows of k values (a multiple of 4) times the G vectors at `vec` (pitch k): L lanes a row, R rows a thread at once, whose
// loads are in flight together and share what is read of the vectors.  (One row at a time, the two layers of 576 -> 144 -> 576 took
// 14000 and 12000 of 53000 clocks at batch 256: a load from L2 for every 16 multiply-adds, one after another; MobileNetV3
// 256x224 947 -> 927 us with this.)
template <int G, int L, bool SMEM, typename F>
__device__ __forceinline__ void matvec(const float* m, int rows, int k, const float* vec, F&& out) {
  constexpr int R = 3, kSubs = kThreads / L;
  const int sub = threadIdx.x / L, lane = threadIdx.x % L;
  for (int j0 = 0; j0 < rows; j0 += R * kSubs) {   // whole warps stay for the shuffles
    float s[R][G];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int im = 0; im < G; ++im) s[r][im] = 0.0f;
#pragma unroll(G == 4 ? 1 : 2)
    for (int i = 4 * lane; i < k; i += 4 * L) {
      float4 w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int j = min(j0 + r * kSubs + sub, rows - 1);   // past the last row: that one again, not used
        const float4* wp = reinterpret_cast<const float4*>(m + (size_t)j * k + i);
        w[r] = SMEM ? *wp : __ldg(wp);
      }
#pragma unroll
      for (int im = 0; im < G; ++im) {
        const float4 v = *reinterpret_cast<const float4*>(vec + im * k + i);
#pragma unroll
        for (int r = 0; r < R; ++r) s[r][im] = fmaf(v.x, w[r].x, fmaf(v.y, w[r].y, fmaf(v.z, w[r].z, fmaf(v.w, w[r].w, s[r][im]))));
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = j0 + r * kSubs + sub;
      if (j0 + r * kSubs >= rows) break;
#pragma unroll
      for (int im = 0; im < G; ++im)
#pragma unroll
        for (int d = L / 2; d > 0; d >>= 1) s[r][im] += __shfl_xor_sync(0xffffffffu, s[r][im], d);
      if (j < rows && lane < kCluster) {   // every lane has the sums: each sees to one CTA of the cluster
#pragma unroll
        for (int im = 0; im < G; ++im) out(j, im, s[r][im], lane);
      }
    }
  }
}

// first of the n rows that CTA `rank` of the cluster owns
__device__ __forceinline__ int row_of(int n, int rank) { return n * rank / kCluster; }
template <typename T, int G, bool STAGED>   // G images a cluster (1, 2 or 4); the matrices staged in shared memory
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads, 4) se_kernel(T* __restrict__ x, const SeParams p) {
  using VT = Vec8<T>;
  constexpr int V = VT::V;
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(8) unsigned long long w_bar;
  const int C = p.C, Cr = p.Cr, HW = p.H * p.W;
  float* part = smem;                          // [G][kThreads][V]: sums of the pixel slots of this CTA's slices
  float* slice_sum = part + G * kThreads * V;  // [C]: the sum of this CTA's slices (G of the G * 8 of the cluster)
  float* pooled = slice_sum + C;               // [G][C]; later the gates of its image
  float* hidden = pooled + G * C;              // [G][Cr]
  float* m1 = hidden + G * Cr;                 // its rows of W1 and W2
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int n0 = (int)(blockIdx.x / kCluster) * G;
  const int cv = C / V, ps = kThreads / cv;    // channel vectors, pixel slots
  const int slot = threadIdx.x / cv, vc = threadIdx.x - slot * cv;
  const int r1 = row_of(Cr, rank), n1 = row_of(Cr, rank + 1) - r1, r2 = row_of(C, rank), n2 = row_of(C, rank + 1) - r2;
  float* m2 = m1 + n1 * C;
  const uint32_t bar = ptx::smem_u32(&w_bar);
  if (STAGED && threadIdx.x == 0) {
    ptx::mbar_init(bar, 1);
    ptx::mbar_fence_init();
    const uint32_t b1 = (uint32_t)(n1 * C) * 4u, b2 = (uint32_t)(n2 * Cr) * 4u;
    ptx::mbar_arrive_expect_tx(bar, b1 + b2);
    if (b1) ptx::bulk_g2s(ptx::smem_u32(m1), p.w1 + (size_t)r1 * C, b1, bar);
    if (b2) ptx::bulk_g2s(ptx::smem_u32(m2), p.w2 + (size_t)r2 * Cr, b2, bar);
  }
  // CTA r works on image r / (8 / G), slices [(r % (8 / G)) * G, + G)
  const int per = kCluster / G, img = n0 + rank / per, first = (rank % per) * G;
  const bool live = slot < ps && img < p.N;
  T* base = x + ((size_t)img * p.l.img_rows * p.l.pitch) * C;
  auto at = [&](int px, int v) {
    const int y = (int)epi::div_by((uint32_t)px, p.div_w);
    return base + ((size_t)(y + p.l.off) * p.l.pitch + (px - y * p.W) + p.l.off) * C + (size_t)v * V;
  };
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  {
    // the slices side by side: G independent loads a step
    float s[G][V];
    int px[G], hi[G];
#pragma unroll
    for (int k = 0; k < G; ++k) {
      px[k] = (int)((long long)HW * (first + k) / kCluster) + slot;
      hi[k] = (int)((long long)HW * (first + k + 1) / kCluster);
#pragma unroll
      for (int e = 0; e < V; ++e) s[k][e] = 0.0f;
    }
    if (live) {
      const int steps = (HW / kCluster + 1 + ps - 1) / ps;
#pragma unroll(G == 1 ? 8 : (G == 2 ? 4 : 2))
      for (int t = 0; t < steps; ++t) {
#pragma unroll
        for (int k = 0; k < G; ++k) {
          uint4 r = make_uint4(0, 0, 0, 0);
          if (px[k] < hi[k]) r = __ldcg(reinterpret_cast<const uint4*>(at(px[k], vc)));
          px[k] += ps;
          float f[V];
          VT::load(r, f);
#pragma unroll
          for (int e = 0; e < V; ++e) s[k][e] += f[e];
        }
      }
    }
    if (slot < ps) {
#pragma unroll
      for (int k = 0; k < G; ++k)
#pragma unroll
        for (int e = 0; e < V; e += 4)
          *reinterpret_cast<float4*>(part + (size_t)k * kThreads * V + (slot * cv + vc) * V + e) = make_float4(s[k][e], s[k][e + 1], s[k][e + 2], s[k][e + 3]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C; i += kThreads) {
    float t[G];
#pragma unroll
    for (int k = 0; k < G; ++k) {
      t[k] = 0.0f;
      for (int q = 0; q < ps; ++q) t[k] += part[k * kThreads * V + q * C + i];
    }
#pragma unroll
    for (int d = 1; d < G; d <<= 1)
#pragma unroll
      for (int k = 0; k < G; k += 2 * d) t[k] += t[k + d];
    slice_sum[i] = t[0];
  }
  cluster.sync();
  for (int i = threadIdx.x; i < G * (C / 4); i += kThreads) {
    const int im = i / (C / 4), c = 4 * (i - im * (C / 4));
    float4 t[kCluster / G];
#pragma unroll
    for (int q = 0; q < kCluster / G; ++q) t[q] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&slice_sum[c], im * per + q));
#pragma unroll
    for (int d = 1; d < kCluster / G; d <<= 1)
#pragma unroll
      for (int q = 0; q < kCluster / G; q += 2 * d) {
        t[q].x += t[q + d].x; t[q].y += t[q + d].y; t[q].z += t[q + d].z; t[q].w += t[q + d].w;
      }
    const float n = (float)HW;
    *reinterpret_cast<float4*>(pooled + im * C + c) = make_float4(t[0].x / n, t[0].y / n, t[0].z / n, t[0].w / n);
  }
  __syncthreads();
  // bounded; every thread of the cluster takes the same way out of a copy that does not arrive: none, the sums are then
  // wrong and the status word says so
  if (STAGED && !ptx::mbar_wait(bar, 0) && p.error_flag && threadIdx.x == 0) atomicCAS(p.error_flag, 0, (int)kErrWaitLoader);
  // Hidden values and gates are stored into the CTAs that use them: nobody reads another's shared memory after the first exchange,
  // so that a CTA may leave when it is done.  (Collected by their readers, with a last barrier before anyone left, the exchanges took
  // 2500 clocks more, at two images a fifth of the kernel.)
  auto to_hidden = [&](int j, int im, float v, int q) {
    v += __ldg(p.b1 + r1 + j);
    *cluster.map_shared_rank(&hidden[im * Cr + r1 + j], q) = !(v <= 0.0f) ? v : 0.0f;
  };
  const float* w1 = STAGED ? m1 : p.w1 + (size_t)r1 * C;
  if (n1 <= 3 * kWarps) matvec<G, 32, STAGED>(w1, n1, C, pooled, to_hidden);
  else matvec<G, 8, STAGED>(w1, n1, C, pooled, to_hidden);
  cluster.sync();                              // also: nobody reads slice_sum or pooled any more
  auto to_gate = [&](int j, int im, float v, int q) {   // to the CTAs of image im
    if (q < per) *cluster.map_shared_rank(&pooled[r2 + j], im * per + q) = hard_sigmoid<T>(v + __ldg(p.b2 + r2 + j));
  };
  const float* w2 = STAGED ? m2 : p.w2 + (size_t)r2 * Cr;
  if (n2 <= 3 * kWarps) matvec<G, 32, STAGED>(w2, n2, Cr, hidden, to_gate);
  else matvec<G, 8, STAGED>(w2, n2, Cr, hidden, to_gate);
  cluster.sync();
  if (!live) return;
  float g[V];
#pragma unroll
  for (int e = 0; e < V; ++e) g[e] = pooled[vc * V + e];
  const int lo = (int)((long long)HW * first / kCluster), hi = (int)((long long)HW * (first + G) / kCluster);
#pragma unroll 4
  for (int px = lo + slot; px < hi; px += ps) {
    uint4* q = reinterpret_cast<uint4*>(at(px, vc));
    float f[V];
    VT::load(__ldcg(q), f);
#pragma unroll
    for (int e = 0; e < V; ++e) f[e] *= g[e];
    *q = VT::store(f);
  }
}

size_t se_smem(bool staged, int V, int G, int C, int Cr) {
  const size_t m = staged ? (size_t)((Cr + kCluster - 1) / kCluster) * C + (size_t)((C + kCluster - 1) / kCluster) * Cr : 0;
  return ((size_t)G * kThreads * V + (size_t)(C + G * C) + (size_t)G * Cr + m) * sizeof(float);
}

template <typename T, int G, bool STAGED>
cudaError_t launch_images(void* x, const SeParams& p, cudaStream_t st) {
  const size_t smem = se_smem(STAGED, Vec8<T>::V, G, p.C, p.Cr);
  cudaError_t e = cudaFuncSetAttribute(se_kernel<T, G, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(se_kernel<T, G, STAGED>, dim3((unsigned)((p.N + G - 1) / G * kCluster)), dim3(kThreads), smem, st, static_cast<T*>(x), p);
}

// More images per cluster read the matrices less often, as long as three CTAs an SM remain (four fit); the matrices are
// staged where that costs no residency: they are small, or the CTAs few.
template <typename T, int G>
cudaError_t launch_staged(void* x, const SeParams& p, int sms, cudaStream_t st) {
  const size_t smem = se_smem(true, Vec8<T>::V, G, p.C, p.Cr);
  const long long ctas = (long long)((p.N + G - 1) / G) * kCluster;
  if (smem <= kShareSmem || (ctas <= sms && smem <= kMaxSmem)) return launch_images<T, G, true>(x, p, st);
  return launch_images<T, G, false>(x, p, st);
}
template <typename T>
cudaError_t launch_typed(void* x, const SeParams& p, int sms, cudaStream_t st) {
  auto take = [&](int g) { return (long long)((p.N + g - 1) / g) * kCluster >= 3LL * sms && se_smem(false, Vec8<T>::V, g, p.C, p.Cr) <= kMaxSmem; };
  if (take(4)) return launch_staged<T, 4>(x, p, sms, st);
  if (take(2)) return launch_staged<T, 2>(x, p, sms, st);
  return launch_staged<T, 1>(x, p, sms, st);
}

}  // namespace

// One channel vector a thread; rows of the matrices are read 16 bytes at a time.
bool se_supported(DType dt, int C, int Cr) {
  const int V = 16 / (int)dtype_size(dt);
  return C % V == 0 && C / V <= kThreads && Cr % 4 == 0 && Cr >= kCluster && Cr <= 2048;
}

cudaError_t launch_se(void* x, Layout l, const float* w1, const float* b1, const float* w2, const float* b2, DType dt, int N, int H, int W, int C,
                      int Cr, int sm_count, int* error_flag, cudaStream_t st) {
  if (!se_supported(dt, C, Cr) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w1) & 15) ||
      (reinterpret_cast<uintptr_t>(w2) & 15) || (long long)N * kCluster > 0x7fffffffLL)
    return cudaErrorInvalidValue;
  if (l.pitch == 0) l = dense_layout(H, W);
  const SeParams p{w1, b1, w2, b2, l, N, H, W, C, Cr, epi::fast_div((uint32_t)W), error_flag};
  if (dt == kF32) return launch_typed<float>(x, p, sm_count, st);
  if (dt == kF16) return launch_typed<__half>(x, p, sm_count, st);
  return launch_typed<__nv_bfloat16>(x, p, sm_count, st);
}

}  // namespace nncv_b200
