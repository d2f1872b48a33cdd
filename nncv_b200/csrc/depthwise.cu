// Depthwise convolution + folded batch-norm + activation, NHWC, staged through shared memory by TMA
// (linalg.depthwise_conv_2d_nchw_chw followed by the batch-norm and hard-swish / ReLU generics,
// tests/Nets/MobileNetV3.mlir:301,426,486 ...).
//
// The operator is bound by HBM: 2 bytes in and 2 bytes out per element, 9 or 25 multiply-adds.  A
// kernel that fetches its taps with per-thread global loads spends its time waiting for them (a
// few loads in flight per thread, bounds checks between them), so here a persistent CTA walks
// tiles of 4 or 8 output rows x TW output columns x CB channels and one thread issues, one or two tiles
// ahead, ONE tensor copy per tile: the input patch with its halo, out-of-range pixels filled with zeros by
// the copy engine (no bounds checks on the input side at all).  The block's threads (up to 128, in fp32
// 256) then read the patch from shared memory: thread = (four channels, one or two output columns),
// computing a column strip of output rows in fp32 pairs (fma.rn.f32x2), so that each input value is
// loaded once per input column and reused down the strip, and each filter value serves the strip.
// What bounds the 16-bit kernels is the pipe of the packed multiply-adds, on which the conversions to
// fp32 run too (64x112x112x96 hard-swish: 64 % of its rate with one column a thread, 15 conversions
// beside 18 multiply-adds for an output of four channels; two columns share four of six input columns:
// 10).  An fp16 map is converted by multiply-adds with 1, which run at twice the rate of conversions and give the same values (that layer
// 69.2 -> 65.4 us; MobileNetV3, 256 images, 906 -> 876).  A filter that fp16 holds could be multiplied as it is, too (fma.rn.f32.f16 takes
// map and filter; 845), but then without the scale in it, which gives other sums, and it pays only with more than one tile an SM: an
// image's result came to depend on its batch.
// With eight channels a thread and strips of four rows the 5x5 layers were bound by
// shared memory: a filter vector of eight fp32 is two loads at a stride of 32 bytes, two-way bank conflicts, and those loads
// were two thirds of the traffic (14x14x240 at batch 256: 9.8 M wavefronts, 48 us); now a lane's four filter values are 16
// contiguous bytes and are read half as often.  Filter, scale and shift sit in shared memory: for the 16-bit types as the
// filter times the scale and the shift the sums start at; for fp32, where the product's rounding would be one more error of
// the size of the others (and the same for every pixel, so that it survives averaging: MobileNetV3's fp32 logits were
// 4.3e-7 off the result in 64 bits instead of 3.3e-7), one by one.
// Every wait on a copy is bounded; a wait that gives up sets the status word and the CTA leaves.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "depthwise_shape.h"
#include "epilogue.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {

namespace {

// What a thread computes: KP output rows x PX adjacent output columns of four channels (depthwise_shape.h).
template <typename T, int KP> constexpr int kTH = sizeof(T) == 4 ? 8 : KP;   // output rows of a tile
template <typename T> constexpr bool kFold = sizeof(T) == 2;   // the scale multiplied into the filter
using dw::kMaxStages;

struct DwParams {
  const void* w;       // [C][KS*KS], fp32 or fp16
  int w_half;
  const float* scale;  // [C] or null
  const float* shift;  // [C] or null
  void* y;             // [N,OH,OW,C]
  int N, H, W, C, OH, OW, pad, act;
  Layout in_l, out_l;  // input coordinates and output pixels are shifted by the layouts' pad offsets
  int tw, cbv;         // output columns per tile, 16-byte channel vectors per chunk
  int tiles_x, tiles_y, n_tiles;   // spatial tiles (n_tiles = N * tiles_y * tiles_x)
  epi::FastDiv div_tx, div_ty;
  int stages;
  uint32_t stage_bytes, stage_stride;
  int* error_flag;
};

typedef unsigned long long u64;   // two fp32 in a register pair
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// a * b + c of two fp16 values and an fp32 one, the product exact, rounded once
__device__ __forceinline__ void fma_halves(float& d0, float& d1, uint32_t a, uint32_t b) {
  asm("{\n.reg .b16 al, ah, bl, bh;\nmov.b32 {al, ah}, %2;\nmov.b32 {bl, bh}, %3;\nfma.rn.f32.f16 %0, al, bl, %0;\nfma.rn.f32.f16 %1, ah, bh, %1;\n}\n"
      : "+f"(d0), "+f"(d1) : "r"(a), "r"(b));
}

// A thread's vector: four channels, 8 bytes of a 16-bit type or 16 of fp32.
template <typename T> struct Vec { using type = uint2; };
template <> struct Vec<float> { using type = uint4; };
__device__ __forceinline__ void unpack(const uint4& raw, u64 (&f)[2], float) {
  f[0] = epi::pk(__uint_as_float(raw.x), __uint_as_float(raw.y));
  f[1] = epi::pk(__uint_as_float(raw.z), __uint_as_float(raw.w));
}
__device__ __forceinline__ void unpack(const uint2& raw, u64 (&f)[2], __half) {
  // x * 1 - 0: conversions run at half the rate of multiply-adds
  float a[4] = {-0.0f, -0.0f, -0.0f, -0.0f};
  fma_halves(a[0], a[1], raw.x, 0x3c003c00u);
  fma_halves(a[2], a[3], raw.y, 0x3c003c00u);
  f[0] = epi::pk(a[0], a[1]);
  f[1] = epi::pk(a[2], a[3]);
}
__device__ __forceinline__ void unpack(const uint2& raw, u64 (&f)[2], __nv_bfloat16) {   // a bf16 is the upper half of an fp32
  f[0] = epi::pk(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u));
  f[1] = epi::pk(__uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
}
__device__ __forceinline__ uint4 pack(const float (&v)[4], float) {
  return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
}
__device__ __forceinline__ uint2 pack(const float (&v)[4], __half) {   // saturating, NaN stays NaN
  return make_uint2(epi::pack16(v[0], v[1], false, false), epi::pack16(v[2], v[3], false, false));
}
__device__ __forceinline__ uint2 pack(const float (&v)[4], __nv_bfloat16) {
  return make_uint2(epi::pack16(v[0], v[1], true, false), epi::pack16(v[2], v[3], true, false));
}

// The activations of MobileNetV3.mlir:345-383 and Yolov5s.mlir:158-169.  EXACT (fp32 tensors) keeps
// IEEE division and expf; 16-bit results take the multiply by 1/6 and the hardware exponential.
// Compare-and-select clamps pass a NaN on, as the fixtures' cmpf/select pairs do.
template <bool EXACT>
__device__ __forceinline__ float act1(float x, int act) {
  switch (act) {
    case kActRelu: return !(x <= 0.0f) ? x : 0.0f;
    case kActHardSigmoid:
    case kActHardSwish: {
      float t = EXACT ? (x + 3.0f) / 6.0f : (x + 3.0f) * 0.16666667f;
      t = (1.0f < t) ? 1.0f : t;
      t = (0.0f > t) ? 0.0f : t;
      return act == kActHardSwish ? x * t : t;
    }
    case kActSigmoid:
    case kActSilu: {
      const float s = EXACT ? 1.0f / (expf(-x) + 1.0f) : __fdividef(1.0f, __expf(-x) + 1.0f);
      return act == kActSilu ? x * s : s;
    }
    default: return x;
  }
}

template <typename T, int KS, int STRIDE, int PX, int kP>
__global__ void __launch_bounds__(dw::max_threads(sizeof(T)), dw::ctas(sizeof(T), KS, PX)) depthwise_tma_kernel(const __grid_constant__ CUtensorMap tm_in, const DwParams p) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  constexpr int V = 4;                                  // channels of a thread
  constexpr int TH = kTH<T, kP>;
  constexpr int kPer = 16 / (V * sizeof(T));            // threads of a 16-byte vector
  using Raw = typename Vec<T>::type;
  constexpr int NR = (kP - 1) * STRIDE + KS, NC = (PX - 1) * STRIDE + KS;   // input rows and columns under a thread's outputs
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) unsigned long long full_bar[kMaxStages];
  __shared__ int abort_flag;
  __shared__ int4 tile_info[kMaxStages];                 // (image, first output row, first output column) of the tile in a stage

  const int tid = threadIdx.x;
  const int cbv = p.cbv, tw = p.tw;
  const int CB = cbv * kPer * V;                         // channels per chunk
  const int IW = (tw - 1) * STRIDE + KS;
  const int c0 = blockIdx.y * CB;
  float* sw = reinterpret_cast<float*>(smem + (size_t)p.stages * p.stage_stride);   // [KS*KS][CB] filter, shift[CB], scale[CB] unless folded
  float* ssh = sw + KS * KS * CB;
  float* ssc = ssh + CB;

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 1);
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_in);
  }
  const int my_tiles = ((int)blockIdx.x < p.n_tiles) ? (p.n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto issue = [&](int k) {      // thread 0: the copy of this CTA's k-th tile into stage k % stages
    const int sp = blockIdx.x + k * gridDim.x;
    const int t2 = (int)epi::div_by((uint32_t)sp, p.div_tx), tx = sp - t2 * p.tiles_x;
    const int n = (int)epi::div_by((uint32_t)t2, p.div_ty), ty = t2 - n * p.tiles_y;
    const int s = k % p.stages;
    const uint32_t bar = ptx::smem_u32(&full_bar[s]);
    tile_info[s] = make_int4(n, ty * TH, tx * tw, 0);   // read by the others after they have seen the barrier complete
    ptx::mbar_arrive_expect_tx(bar, p.stage_bytes);
    ptx::tma_load_4d(ptx::smem_u32(smem + (size_t)s * p.stage_stride), &tm_in, c0, tx * tw * STRIDE - p.pad + p.in_l.off,
                     ty * TH * STRIDE - p.pad + p.in_l.off, n, bar);
  };
  int issued = 0;
  if (tid == 0)
    for (; issued < p.stages - 1 && issued < my_tiles; ++issued) issue(issued);

  // filter, scale and shift: all loads of a channel in flight together, behind the first copies
  for (int c = tid; c < CB; c += (int)blockDim.x) {
    const bool in = c0 + c < p.C;
    float v[KS * KS];
#pragma unroll
    for (int tap = 0; tap < KS * KS; ++tap) {
      const size_t idx = (size_t)(c0 + c) * (KS * KS) + tap;
      v[tap] = !in ? 0.0f : p.w_half ? __half2float(reinterpret_cast<const __half*>(p.w)[idx]) : reinterpret_cast<const float*>(p.w)[idx];
    }
    const float scale = in && p.scale ? p.scale[c0 + c] : 1.0f;
    ssh[c] = in && p.shift ? p.shift[c0 + c] : 0.0f;
    if (!kFold<T>) ssc[c] = scale;
#pragma unroll
    for (int tap = 0; tap < KS * KS; ++tap) sw[tap * CB + c] = kFold<T> ? v[tap] * scale : v[tap];
  }
  __syncthreads();

  const int xs = tid / (kPer * cbv), cvec = tid - xs * (kPer * cbv), pairs = tw / PX;
  const int ys = TH == kP ? 0 : xs / pairs, x = (xs - ys * pairs) * PX;   // strip of rows, first column
  int k = 0;
  for (; k < my_tiles; ++k) {
    const int s = k % p.stages;
    bool ok = ptx::mbar_wait_abortable(ptx::smem_u32(&full_bar[s]), (uint32_t)((k / p.stages) & 1), &abort_flag);
    // one barrier per tile: past it every thread has finished tile k - 1, whose stage the next copy overwrites
    if (__syncthreads_or(!ok)) break;
    if (tid == 0 && issued < my_tiles) { issue(issued); ++issued; }

    if (xs >= pairs * (TH / kP)) continue;   // no strip of the tile is this thread's
    const unsigned char* st = smem + (size_t)s * p.stage_stride;
    // folded: the sums start at the shift, the filter carries the scale
    u64 acc[PX][kP][2];
    {
      const ulonglong2 sh = kFold<T> ? *reinterpret_cast<const ulonglong2*>(ssh + cvec * V) : make_ulonglong2(0, 0);
#pragma unroll
      for (int px = 0; px < PX; ++px)
#pragma unroll
        for (int o = 0; o < kP; ++o) { acc[px][o][0] = sh.x; acc[px][o][1] = sh.y; }
    }
    ulonglong2 wr[KS][KS];   // filter column kx in wr[kx], live while an output column needs it
#pragma unroll
    for (int ix = 0; ix < NC; ++ix) {
      if (ix < KS) {
#pragma unroll
        for (int q = 0; q < KS; ++q) wr[ix][q] = *reinterpret_cast<const ulonglong2*>(sw + (q * KS + ix) * CB + cvec * V);
      }
      const unsigned char* col = st + (size_t)(ys * kP * STRIDE * IW + x * STRIDE + ix) * cbv * 16 + cvec * sizeof(Raw);
#pragma unroll
      for (int ry = 0; ry < NR; ++ry) {
        u64 f[2];
        unpack(*reinterpret_cast<const Raw*>(col + (size_t)ry * IW * cbv * 16), f, T{});
#pragma unroll
        for (int px = 0; px < PX; ++px) {
          const int kx = ix - px * STRIDE;
          if (kx < 0 || kx >= KS) continue;
#pragma unroll
          for (int o = 0; o < kP; ++o) {
            const int q = ry - o * STRIDE;               // compile-time after unrolling
            if (q >= 0 && q < KS) {
              acc[px][o][0] = epi::fma2(f[0], wr[kx][q].x, acc[px][o][0]);
              acc[px][o][1] = epi::fma2(f[1], wr[kx][q].y, acc[px][o][1]);
            }
          }
        }
      }
    }
    // epilogue: activation, store
    const int4 ti = tile_info[s];
    const int c = c0 + cvec * V, rows = min(kP, p.OH - ti.y - ys * kP);
    if (c >= p.C) continue;
#pragma unroll
    for (int px = 0; px < PX; ++px) {
      const int ox = ti.z + x + px;
      if (ox >= p.OW) break;
      if (!kFold<T>) {
        const ulonglong2 sc = *reinterpret_cast<const ulonglong2*>(ssc + cvec * V), sh = *reinterpret_cast<const ulonglong2*>(ssh + cvec * V);
#pragma unroll
        for (int o = 0; o < kP; ++o) {
          acc[px][o][0] = epi::fma2(acc[px][o][0], sc.x, sh.x);
          acc[px][o][1] = epi::fma2(acc[px][o][1], sc.y, sh.y);
        }
      }
      T* yp = reinterpret_cast<T*>(p.y) + (((size_t)ti.x * p.out_l.img_rows + ti.y + ys * kP + p.out_l.off) * p.out_l.pitch + ox + p.out_l.off) * p.C + c;
      const size_t row_step = (size_t)p.out_l.pitch * p.C;
      auto finish = [&](auto f4) {
#pragma unroll
        for (int o = 0; o < kP; ++o) {
          if (o >= rows) break;
          float v[4];
          f4(acc[px][o][0], v[0], v[1]);
          f4(acc[px][o][1], v[2], v[3]);
          *reinterpret_cast<Raw*>(yp + o * row_step) = pack(v, T{});
        }
      };
      if (p.act == kActNone) {
        finish([](u64 a, float& r, float& t) { epi::unpk(a, r, t); });
      } else if (sizeof(T) == 2 && p.act == kActHardSwish) {
        // clamp of (x + 3) / 6 to [0, 1]: a NaN still comes out as NaN because the clamped factor multiplies x itself
        finish([](u64 a, float& r, float& t) {
          epi::unpk(a, r, t);
          epi::unpk(mul2(a, epi::pk(__saturatef(fmaf(r, 0.16666667f, 0.5f)), __saturatef(fmaf(t, 0.16666667f, 0.5f)))), r, t);
        });
      } else {
        finish([&](u64 a, float& r, float& t) {
          epi::unpk(a, r, t);
          r = act1<sizeof(T) == 4>(r, p.act);
          t = act1<sizeof(T) == 4>(t, p.act);
        });
      }
    }
  }
  if (k < my_tiles && tid == 0) {
    // a wait gave up: record it, then give the copies still in flight a bounded time to land before
    // the CTA's shared memory is released
    if (p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    for (int j = k; j < issued; ++j)
      ptx::mbar_wait_limit(ptx::smem_u32(&full_bar[j % p.stages]), (uint32_t)((j / p.stages) & 1), 1LL << 24);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 dw_get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  });
  return fn;
}

template <typename T, int KS, int STRIDE, int PX, int KP>
cudaError_t launch_one(const CUtensorMap& tm, const DwParams& p, dim3 grid, int threads, size_t smem, cudaStream_t st) {
  auto kern = depthwise_tma_kernel<T, KS, STRIDE, PX, KP>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  launch_pdl(kern, grid, dim3((unsigned)threads), smem, st, tm, p);
  return cudaGetLastError();
}

template <typename T, int PX, int KP>
cudaError_t launch_typed(const CUtensorMap& tm, const DwParams& p, int ks, int stride, dim3 grid, int threads, size_t smem, cudaStream_t st) {
  if (ks == 3 && stride == 1) return launch_one<T, 3, 1, PX, KP>(tm, p, grid, threads, smem, st);
  if (ks == 3 && stride == 2) return launch_one<T, 3, 2, PX, KP>(tm, p, grid, threads, smem, st);
  if (ks == 5 && stride == 1) return launch_one<T, 5, 1, PX, KP>(tm, p, grid, threads, smem, st);
  return launch_one<T, 5, 2, PX, KP>(tm, p, grid, threads, smem, st);
}
template <typename T>
cudaError_t launch_shape(int px, const CUtensorMap& tm, const DwParams& p, int ks, int stride, dim3 grid, int threads, size_t smem, cudaStream_t st) {
  if (px == 1) return launch_typed<T, 1, 8>(tm, p, ks, stride, grid, threads, smem, st);
  if (ks == 3) return stride == 1 ? launch_one<T, 3, 1, 2, 8>(tm, p, grid, threads, smem, st) : launch_one<T, 3, 2, 2, 4>(tm, p, grid, threads, smem, st);
  return stride == 1 ? launch_one<T, 5, 1, 2, 8>(tm, p, grid, threads, smem, st) : launch_one<T, 5, 2, 2, 4>(tm, p, grid, threads, smem, st);
}

}  // namespace

bool depthwise_tma_supported(DType dt, int N, int H, int W, int C, int R, int S, int stride, int pad) {
  const int V = 16 / (int)dtype_size(dt);
  if (R != S || (R != 3 && R != 5) || (stride != 1 && stride != 2) || pad > R) return false;
  if (C % V != 0 || C / V < 2) return false;
  const int OH = (H + 2 * pad - R) / stride + 1, OW = (W + 2 * pad - S) / stride + 1;
  if (OH <= 0 || OW <= 0) return false;
  return (long long)N * ((OH + 3) / 4) * ((OW + 1) / 2) < (1LL << 30);
}

cudaError_t launch_depthwise_tma(const void* x, const void* w, DType w_dt, const float* scale, const float* shift, void* y, DType dt,
                                 int N, int H, int W, int C, int R, int S, int stride, int pad, int act, Layout in_l, Layout out_l,
                                 int sm_count, int* error_flag, cudaStream_t st) {
  if (!depthwise_tma_supported(dt, N, H, W, C, R, S, stride, pad) || (reinterpret_cast<uintptr_t>(x) & 15) ||
      (reinterpret_cast<uintptr_t>(y) & 15))
    return cudaErrorInvalidValue;
  const int es = (int)dtype_size(dt), V = 16 / es, cv = C / V;   // cv: 16-byte channel vectors
  const int OH = (H + 2 * pad - R) / stride + 1, OW = (W + 2 * pad - S) / stride + 1;
  DwParams p{};
  const int sms = sm_count > 0 ? sm_count : 148;
  const dw::Shape d = dw::shape_of(N, C, OH, OW, R, stride, es, sms);
  if (d.cbv == 0) return cudaErrorInvalidValue;
  const int tw = d.tw, cbv = d.cbv, px = d.px, kp = d.kp, th = es == 2 ? kp : 8, IH = (th - 1) * stride + R, IW = (tw - 1) * stride + R;
  p.tw = tw; p.cbv = cbv;
  p.stage_bytes = (uint32_t)IW * IH * cbv * 16;
  p.stage_stride = (p.stage_bytes + 127u) & ~127u;
  p.stages = d.stages;
  const size_t smem = d.smem;
  p.w = w; p.w_half = w_dt == kF16; p.scale = scale; p.shift = shift; p.y = y;
  p.N = N; p.H = H; p.W = W; p.C = C; p.OH = OH; p.OW = OW; p.pad = pad; p.act = act;
  if (in_l.pitch == 0) in_l = dense_layout(H, W);
  if (out_l.pitch == 0) out_l = dense_layout(OH, OW);
  // a padded layout's pad row / column is zero and everything beyond the map is out of the tensor map's range
  // (zero-filled), so the halo reads the same values as over a dense map
  if (in_l.off != 0 && (in_l.off != 1 || in_l.pitch != W + 1 || in_l.img_rows != H + 1)) return cudaErrorInvalidValue;
  p.in_l = in_l; p.out_l = out_l;
  p.tiles_x = (OW + tw - 1) / tw; p.tiles_y = (OH + th - 1) / th;
  p.n_tiles = N * p.tiles_y * p.tiles_x;
  p.div_tx = epi::fast_div((uint32_t)p.tiles_x); p.div_ty = epi::fast_div((uint32_t)p.tiles_y);
  p.error_flag = error_flag;

  auto enc = dw_get_encode();
  if (!enc) return cudaErrorNotSupported;
  CUtensorMap tm;
  const CUtensorMapDataType tdt = dt == kF32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                  : dt == kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  cuuint64_t gdim[4] = {(cuuint64_t)C, (cuuint64_t)in_l.pitch, (cuuint64_t)in_l.img_rows, (cuuint64_t)N};
  cuuint64_t gstr[3] = {(cuuint64_t)C * es, (cuuint64_t)in_l.pitch * C * es, (cuuint64_t)in_l.img_rows * in_l.pitch * C * es};
  cuuint32_t box[4] = {(cuuint32_t)(cbv * V), (cuuint32_t)IW, (cuuint32_t)IH, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  if (enc(&tm, tdt, 4, const_cast<void*>(x), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;

  const int chunks = (cv + cbv - 1) / cbv;
  int gx = sms * d.per_sm / chunks;
  if (gx < 1) gx = 1;
  if (gx > p.n_tiles) gx = p.n_tiles;
  const dim3 grid((unsigned)gx, (unsigned)chunks);
  if (chunks > 65535) return cudaErrorInvalidValue;
  if (dt == kF32) return launch_typed<float, 1, 4>(tm, p, R, stride, grid, d.threads, smem, st);
  if (dt == kF16) return launch_shape<__half>(px, tm, p, R, stride, grid, d.threads, smem, st);
  return launch_shape<__nv_bfloat16>(px, tm, p, R, stride, grid, d.threads, smem, st);
}

}  // namespace nncv_b200
