// Convolutions and fully connected layers of small batches: the implicit GEMM of tconv.cu on 64 x 32 tiles.
//
// What bounds a layer of one or a few images is one chain: launch, first copies, R*S*C/64 blocks one after another on a few
// SMs, epilogue, stores (counters of 14x14x256 -> 256 3x3: 32 CTAs, the tensor pipe 13 % busy on the busiest SM, an instruction
// issued every sixth clock).  The MMAs of a block of a 128 x 64 tile read 6 KB of operands each through the shared-memory port,
// 48 clocks; those of a 64 x 32 tile read 3 KB.  Four times the tiles also spread the weights, of which every CTA brings its own
// rows from L2, over four times the SMs.  Sums are formed in the order of the other 16-bit kernels (channel block outermost, tap,
// 16 channels a step), so the results are the same bits and the tile may be chosen by timing.
// One image, us a layer in a row of launches, 128-row tiles before and this: 512 -> 512 3x3 on 7x7 12.4 9.7, 256 -> 256 on 14x14
// 8.1 7.0, with the 1x1 branch 256 -> 512 11.8 8.1, 2048 -> 512 pointwise 9.3 7.2, 1024 -> 256 7.1 5.5; a layer of one block takes
// 4.1 either way.  Forwards of one image: ResNet-18 141 -> 96, ResNet-50 326 -> 222, MobileNetV3 275 -> 200.
//
// One tile a CTA.  Warp 0 issues the MMAs.  Warps 1-4 copy, step j by warp j mod 4 (TMA; weights before the previous kernel
// ends): to see a free stage, announce the bytes and issue two copies takes a warp longer than a block's MMAs take (512 -> 512
// on 7x7: one copying warp 18.1 us, four 11.3).  A step is two blocks, so that the issuing warp waits and commits once for
// eight MMAs (9.7 us; four blocks: no better).  Both test their barriers without a pause.  Then they drain 16 rows x 32 columns
// each, from registers straight to global memory: a staging tile and a TMA store would make the chain longer, and few bytes
// leave.  For M = 64 the accumulator's rows 16w .. 16w + 15 lie in the first sixteen lanes of warp w's quadrant.
// DUAL: the 1x1 branch on the centre tap of tconv.cu, a second accumulator.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "epilogue.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {

namespace {

constexpr int kCopyWarps = 4, kThreads = (1 + kCopyWarps) * 32;
constexpr int kBM = 64, kBN = 32;
constexpr int kABytes = kBM * 128, kWBytes = kBN * 128, kBlockBytes = kABytes + kWBytes;
constexpr int kPer = 2;          // blocks a stage: one wait and one commit for eight MMAs
constexpr int kStageBytes = kPer * kBlockBytes;
constexpr int kMaxStages = 8;

struct SmallParams {
  const uint8_t* wpack;
  const uint8_t* wpack2;
  const float *scale, *shift, *scale2, *shift2;
  const void* residual;   // layout and type of out, or null
  void *out, *out2;
  int* error_flag;
  int Kout, CB, taps, S, stride, pad, in_off, out_off;
  int OH, OW, NB, out_pitch, out_rows;
  int tw, th;                          // tile: tn images x th rows x tw columns = 64 pixels
  int tw_log, th_log;
  int tiles_x, tiles_y, n_tiles;
  epi::FastDiv div_taps, div_s;        // by the taps of a channel block, the branch's included, and by the filter's width
  int stages_log, relu, bf16, out_f32, w_ready;
  int mode;                            // of the epilogue (epi::mode_of)
};

// A load that stays where it stands: the compiler moves plain ones down to their use, behind the wait for the accumulator, where
// their latency is bare (0.5 us a layer).
__device__ __forceinline__ float2 load_now(const float* v) {   // one by one: scale and shift may lie on any float's boundary
  float2 r;
  asm volatile("ld.global.nc.f32 %0, [%2];\n ld.global.nc.f32 %1, [%2 + 4];" : "=&f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint32_t load_now(const unsigned short* v) {
  uint32_t r;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(r) : "l"(v));
  return r;
}

// A thread's 2 x 8 values -> memory.  Each combination is a function of its own, as in epilogue.cuh: with the choices tested for
// every pair by a warp alone on its scheduler, ResNet-18 took 114 us for one image, now 99.
template <bool BF16, bool RES, int ACT>
__device__ __forceinline__ void finish(const uint32_t (&acc)[16], const float2 (&sc)[4], const float2 (&sh)[4], const uint32_t (&res)[2][4],
                                       unsigned short* out, const long long (&at)[2], int cols0, int Kout) {
  uint32_t o[2][4];
#pragma unroll
  for (int g = 0; g < 4; ++g)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unsigned long long v = epi::fma2(epi::pk(__uint_as_float(acc[4 * g + 2 * h]), __uint_as_float(acc[4 * g + 2 * h + 1])),
                                       epi::pk(sc[g].x, sc[g].y), epi::pk(sh[g].x, sh[g].y));
      if (RES) {
        const float2 f = epi::unpack16(res[h][g], BF16);
        v = epi::add2(v, epi::pk(f.x, f.y));
      }
      float a, b;
      epi::unpk(v, a, b);
      if (ACT == 2) {
        a *= __saturatef(fmaf(a, 0.16666667f, 0.5f));
        b *= __saturatef(fmaf(b, 0.16666667f, 0.5f));
      } else if (ACT == 3) {
        a *= __fdividef(1.0f, __expf(-a) + 1.0f);
        b *= __fdividef(1.0f, __expf(-b) + 1.0f);
      }
      o[h][g] = epi::pack16(a, b, BF16, ACT == 1);
    }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int g = 0; g < 4; ++g)
      if (at[h] >= 0 && cols0 + 8 * g < Kout) *reinterpret_cast<uint32_t*>(out + at[h] + cols0 + 8 * g) = o[h][g];
}
__device__ __forceinline__ void finish_f32(const uint32_t (&acc)[16], const float2 (&sc)[4], const float2 (&sh)[4], bool relu, float* out,
                                           const long long (&at)[2], int cols0, int Kout) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float a, b;
      epi::unpk(epi::fma2(epi::pk(__uint_as_float(acc[4 * g + 2 * h]), __uint_as_float(acc[4 * g + 2 * h + 1])), epi::pk(sc[g].x, sc[g].y),
                          epi::pk(sh[g].x, sh[g].y)),
                a, b);
      if (relu) {
        a = !(a <= 0.0f) ? a : 0.0f;
        b = !(b <= 0.0f) ? b : 0.0f;
      }
      if (at[h] >= 0 && cols0 + 8 * g < Kout) *reinterpret_cast<float2*>(out + at[h] + cols0 + 8 * g) = make_float2(a, b);
    }
}

template <bool DUAL>
__global__ void __launch_bounds__(kThreads)
conv_small_kernel(const __grid_constant__ CUtensorMap tm_in, const SmallParams p) {
  constexpr int kCols = DUAL ? 64 : 32;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_bars[2 * kMaxStages + 1];
  const uint32_t ring = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t full = ptx::smem_u32(s_bars), empty = full + 8 * kMaxStages, acc_full = empty + 8 * kMaxStages;
  const int warp = ptx::warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < 2 * kMaxStages + 1; ++i) ptx::mbar_init(full + 8 * i, 1);
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_in);
  }
  if (warp == 0) {
    ptx::tmem_alloc(ptx::smem_u32(&s_tmem), kCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = (uint32_t)ptx::warp_uniform((int)*reinterpret_cast<volatile uint32_t*>(&s_tmem));
  volatile int* abort_flag = &s_abort;

  const int m_item = (int)blockIdx.x / p.n_tiles, n_tile = (int)blockIdx.x - m_item * p.n_tiles;
  const int t2 = m_item / p.tiles_x, tx = m_item - t2 * p.tiles_x, t3 = t2 / p.tiles_y, ty = t2 - t3 * p.tiles_y;
  const int n0 = t3 * (kBM >> (p.tw_log + p.th_log)), oy0 = ty * p.th, ox0 = tx * p.tw;
  const int taps_x = p.taps + (DUAL ? 1 : 0), KB = p.taps * p.CB;

  const uint32_t blocks = (uint32_t)(p.CB * taps_x), steps = (blocks + kPer - 1) / kPer, stages = 1u << p.stages_log;
  if (warp == 0) {
    // ------------------------------------------------------------------ MMAs ------------
    const uint32_t issue = ptx::elect_one();
    const uint32_t idesc = ptx::umma_idesc(kBM, kBN, p.bf16 ? 1 : 0);
    bool okw = true;
    uint32_t tap = 0, seen = 0;
    for (uint32_t j = 0; j < steps; ++j) {
      const uint32_t st = j & (stages - 1);
      if (!ptx::warp_all(seen) && !ptx::warp_spin(full + 8 * st, (j >> p.stages_log) & 1u, abort_flag)) { okw = false; break; }
      ptx::tc_fence_after();
      seen = ptx::mbar_peek(full + 8 * ((j + 1) & (stages - 1)), ((j + 1) >> p.stages_log) & 1u);
#pragma unroll
      for (uint32_t b = 0; b < kPer; ++b) {
        const uint32_t i = j * kPer + b;
        if (i >= blocks) break;
        const bool second = DUAL && tap == (uint32_t)p.taps;
        const uint32_t at = ring + st * kStageBytes + b * kBlockBytes;
        const uint32_t a_lo = ptx::smem_desc_k128_lo(at), b_lo = ptx::smem_desc_k128_lo(at + kABytes);
        const uint32_t first = second ? i - tap : i;   // 0: the accumulator starts here
#pragma unroll
        for (uint32_t k4 = 0; k4 < 4; ++k4)
          ptx::umma_f16(second ? tmem + kBN : tmem, ptx::desc_from_halves(a_lo + k4 * 2, ptx::kSmemDescK128Hi),
                        ptx::desc_from_halves(b_lo + k4 * 2, ptx::kSmemDescK128Hi), idesc, first | k4, issue);
        if (++tap == (uint32_t)taps_x) tap = 0;
      }
      ptx::tc_commit(empty + 8 * st, issue);
    }
    if (okw) ptx::tc_commit(acc_full, issue);
    else if (lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitMma);
    ptx::grid_dependency_wait();
  } else {
    // ------------------------------------------------------------------ copies ----------
    const uint32_t issue = ptx::elect_one(), me = (uint32_t)warp - 1u;
    auto load_weights = [&](uint32_t cb, uint32_t tap, uint32_t at, uint32_t bar) {
      const uint8_t* src = DUAL && tap == (uint32_t)p.taps ? p.wpack2 + ((size_t)n_tile * p.CB + cb) * kWBytes
                                                           : p.wpack + ((size_t)n_tile * KB + (size_t)tap * p.CB + cb) * kWBytes;
      ptx::bulk_g2s(at + kABytes, src, kWBytes, bar, issue);
    };
    auto expect = [&](uint32_t j, uint32_t st) {
      ptx::mbar_arrive_expect_tx(full + 8 * st, j * kPer + kPer <= blocks ? kStageBytes : (blocks - j * kPer) * kBlockBytes, issue);
    };
    const uint32_t early = p.w_ready ? (stages < steps ? stages : steps) : 0u;   // nobody writes packed weights once they are made
    for (uint32_t j = me; j < early; j += kCopyWarps) {
      expect(j, j);
      for (uint32_t i = j * kPer; i < (j + 1) * kPer && i < blocks; ++i) {
        const uint32_t cb = epi::div_by(i, p.div_taps);
        load_weights(cb, i - cb * p.div_taps.d, ring + i * kBlockBytes, full + 8 * j);
      }
    }
    ptx::grid_dependency_wait();   // before this, the input, scale, shift and residual may still be written and out still be read
    ptx::grid_launch_dependents();
    const int xb = p.stride * ox0 - p.pad + p.in_off, yb = p.stride * oy0 - p.pad + p.in_off;
    bool okc = true;
    for (uint32_t j = me; j < steps; j += kCopyWarps) {
      const uint32_t st = j & (stages - 1);
      if (j >= stages && !ptx::warp_spin(empty + 8 * st, ((j >> p.stages_log) & 1u) ^ 1u, abort_flag)) { okc = false; break; }
      if (j >= early) expect(j, st);
#pragma unroll
      for (uint32_t b = 0; b < kPer; ++b) {
        const uint32_t i = j * kPer + b, at = ring + st * kStageBytes + b * kBlockBytes;
        if (i >= blocks) break;
        const uint32_t cb = epi::div_by(i, p.div_taps), tap = i - cb * p.div_taps.d;
        const uint32_t pixel = DUAL && tap == (uint32_t)p.taps ? tap / 2 : tap;   // the branch reads the centre tap's pixels
        const uint32_t r = epi::div_by(pixel, p.div_s), s = pixel - r * p.div_s.d;
        ptx::tma_load_4d(at, &tm_in, (int)cb * 64, xb + (int)s, yb + (int)r, n0, full + 8 * st, issue);
        if (j >= early) load_weights(cb, tap, at, full + 8 * st);
      }
    }
    if (!okc && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    // ------------------------------------------------------------------ epilogue --------
    const int quad = warp & 3, cols0 = n_tile * kBN + 2 * (lane & 3);
    long long at[2];   // element offset of the thread's two rows; -1: outside
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = quad * 16 + h * 8 + (lane >> 2);
      const int x = ox0 + (r & (p.tw - 1)), y = oy0 + ((r >> p.tw_log) & (p.th - 1)), n = n0 + (r >> (p.tw_log + p.th_log));
      at[h] = x < p.OW && y < p.OH && n < p.NB ? (((long long)n * p.out_rows + y + p.out_off) * p.out_pitch + x + p.out_off) * p.Kout : -1;
    }
    auto columns = [&](const float* v, float one, float2 (&c)[4]) {
#pragma unroll
      for (int g = 0; g < 4; ++g)
        c[g] = v && cols0 + 8 * g < p.Kout ? load_now(v + cols0 + 8 * g) : make_float2(one, one);
    };
    float2 sc[4], sh[4];
    uint32_t res[2][4];
    auto load = [&](const float* scale, const float* shift) {
      columns(scale, 1.0f, sc);
      columns(shift, 0.0f, sh);
    };
    load(p.scale, p.shift);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int g = 0; g < 4; ++g)
        res[h][g] = p.residual && at[h] >= 0 && cols0 + 8 * g < p.Kout
                        ? load_now(static_cast<const unsigned short*>(p.residual) + at[h] + cols0 + 8 * g) : 0u;
    const bool okw = ptx::warp_spin(acc_full, 0, abort_flag);
    if (okw) {
      ptx::tc_fence_after();
#pragma unroll
      for (int o = 0; o < (DUAL ? 2 : 1); ++o) {
        if (o == 1) load(p.scale2, p.shift2);
        uint32_t acc[16];
        ptx::tmem_ld_16x32_f(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(o * kBN), acc);
        ptx::tmem_ld_wait();
        if (p.out_f32) {
          finish_f32(acc, sc, sh, p.relu != 0, static_cast<float*>(p.out), at, cols0, p.Kout);
          continue;
        }
        unsigned short* out = static_cast<unsigned short*>(o ? p.out2 : p.out);
#define NNCV_FINISH(B_, R_, A_) \
  case (B_ ? epi::kModeBf16 : 0) | (R_ ? epi::kModeRes : 0) | (A_ << epi::kModeActShift): finish<B_, R_, A_>(acc, sc, sh, res, out, at, cols0, p.Kout); break;
        switch (o ? (p.mode & epi::kModeBf16) : p.mode) {
          NNCV_FINISH(false, false, 0) NNCV_FINISH(false, false, 1) NNCV_FINISH(false, true, 0) NNCV_FINISH(false, true, 1)
          NNCV_FINISH(true, false, 0) NNCV_FINISH(true, false, 1) NNCV_FINISH(true, true, 0) NNCV_FINISH(true, true, 1)
          default:
            if constexpr (!DUAL) {
              switch (p.mode) {
                NNCV_FINISH(false, false, 2) NNCV_FINISH(false, true, 2) NNCV_FINISH(true, false, 2) NNCV_FINISH(true, true, 2)
                NNCV_FINISH(false, false, 3) NNCV_FINISH(false, true, 3) NNCV_FINISH(true, false, 3) NNCV_FINISH(true, true, 3)
                default: break;
              }
            }
        }
#undef NNCV_FINISH
      }
    } else if (lane == 0 && p.error_flag) {
      atomicCAS(p.error_flag, 0, (int)kErrWaitEpilogue);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_dealloc(tmem, kCols);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  });
  return fn;
}

}  // namespace

long long conv_small_tiles(int N, int OH, int OW, int Kout) {
  int tw, th, tn;
  conv_small_tile(N, OH, OW, &tw, &th, &tn);
  return (long long)((OW + tw - 1) / tw) * ((OH + th - 1) / th) * ((N + tn - 1) / tn) * ((Kout + kBN - 1) / kBN);
}

// The width of 64, 32 or 16 pixels that leaves the least of a row's last tile empty, 8 for narrow maps; then rows, then images.
void conv_small_tile(int N, int OH, int OW, int* tw, int* th, int* tn) {
  int w = 8;
  if (N == 1 && OH == 1) {
    w = kBM;   // a matrix
  } else if (OW > 8) {
    int waste = 1 << 30;
    for (int c : {64, 32, 16}) {
      const int ws = (OW + c - 1) / c * c - OW;
      if (ws < waste) { w = c; waste = ws; }
    }
  }
  int h = 1;
  while (h * w < kBM && h < OH) h *= 2;
  *tw = w; *th = h; *tn = kBM / (w * h);
}

cudaError_t launch_conv_small(const TconvArgs& args, cudaStream_t stream) {
  TconvArgs a = args;
  pointwise_as_matrix(&a);
  if (a.ab == kF32 || a.b_rowmajor || !tconv_supported(a.C, a.Kout, a.out_dtype, a.Kout) || (a.residual && a.out_dtype == kF32) || a.stride > 4)
    return cudaErrorInvalidValue;
  if (a.wpack2 && (!a.out2 || a.out_dtype == kF32 || a.R != a.S || a.R % 2 == 0 || a.pad != a.R / 2)) return cudaErrorInvalidValue;
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.wpack) |
                       reinterpret_cast<uintptr_t>(a.wpack2) | reinterpret_cast<uintptr_t>(a.out2);
  if ((al & 15) || (reinterpret_cast<uintptr_t>(a.residual) & 31)) return cudaErrorMisalignedAddress;
  SmallParams p;
  p.wpack = static_cast<const uint8_t*>(a.wpack); p.wpack2 = static_cast<const uint8_t*>(a.wpack2);
  p.scale = a.scale; p.shift = a.shift; p.scale2 = a.scale2; p.shift2 = a.shift2;
  p.residual = a.residual; p.out = a.out; p.out2 = a.out2; p.error_flag = a.error_flag;
  p.Kout = a.Kout; p.CB = (a.C + 63) / 64; p.taps = a.R * a.S; p.S = a.S; p.stride = a.stride; p.pad = a.pad;
  p.in_off = a.in_l.off; p.out_off = a.out_l.off;
  p.OH = a.OH; p.OW = a.OW; p.NB = a.N; p.out_pitch = a.out_l.pitch; p.out_rows = a.out_l.img_rows;
  int tn;
  conv_small_tile(a.N, a.OH, a.OW, &p.tw, &p.th, &tn);
  if (p.tw * a.stride > 256 || p.th * a.stride > 256) return cudaErrorInvalidConfiguration;
  p.tw_log = __builtin_ctz(p.tw); p.th_log = __builtin_ctz(p.th);
  p.tiles_x = (a.OW + p.tw - 1) / p.tw;
  p.tiles_y = (a.OH + p.th - 1) / p.th;
  p.n_tiles = (a.Kout + kBN - 1) / kBN;
  const long long tiles = conv_small_tiles(a.N, a.OH, a.OW, a.Kout);
  if (tiles <= 0 || tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
  p.relu = a.relu; p.bf16 = a.ab == kBF16; p.out_f32 = a.out_dtype == kF32; p.w_ready = a.weights_ready;
  p.mode = epi::mode_of(a.ab == kBF16, a.residual != nullptr, a.relu != 0, a.act);
  const int taps_x = p.taps + (a.wpack2 ? 1 : 0);
  p.div_taps = epi::fast_div((uint32_t)taps_x); p.div_s = epi::fast_div((uint32_t)a.S);
  p.stages_log = 1;
  while ((1 << p.stages_log) < kMaxStages && (kPer << p.stages_log) < taps_x * p.CB) ++p.stages_log;
  const size_t smem = 1024 + ((size_t)kStageBytes << p.stages_log);

  auto enc = get_encode();
  if (!enc) return cudaErrorInvalidValue;
  // [N][rows][pitch][C], box 64 channels x tw x th x tn, taken at every stride-th pixel; past the edges it reads zeros
  CUtensorMap tm_in;
  cuuint64_t gdim[4] = {(cuuint64_t)a.C, (cuuint64_t)a.in_l.pitch, (cuuint64_t)a.in_l.img_rows, (cuuint64_t)a.N};
  cuuint64_t gstr[3] = {(cuuint64_t)a.C * 2, (cuuint64_t)a.in_l.pitch * a.C * 2, (cuuint64_t)a.in_l.img_rows * a.in_l.pitch * a.C * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)(p.tw * a.stride), (cuuint32_t)(p.th * a.stride), (cuuint32_t)tn};
  cuuint32_t estr[4] = {1, (cuuint32_t)a.stride, (cuuint32_t)a.stride, 1};
  if (enc(&tm_in, p.bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(a.in), gdim, gstr, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  auto kern = a.wpack2 ? conv_small_kernel<true> : conv_small_kernel<false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(kern, dim3((unsigned)tiles), dim3(kThreads), smem, stream, tm_in, p);
}

}  // namespace nncv_b200
