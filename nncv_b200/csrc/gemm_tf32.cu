// fp32 GEMM on the tensor cores: C[M,N] = A[M,K] * B[K,N] (+ bias[N]) (+ ReLU), all row-major fp32, with
// fp32-level accuracy from three tcgen05.mma.kind::tf32 products per k step ("3xTF32").
//
// linalg.matmul on f32 is nncv's SGEMM case (tests/MatMulOptimization/MatMulDeafult.mlir:6-9 1024^3,
// MatMulNv.mlir:6-9 8192^3); its own CUDA kernel for it is an unfinished SIMT stub
// (src/libnncv/kernel/sgemm.cu:13-100) and its GPU lowering aims at 16^3 wmma tiles
// (src/nncv/compiler/Conversion/MatMulOptimize/MatMul2NvMMA.cpp:37-90).
//
// A tf32 operand keeps 10 mantissa bits, so one product is good to about 1e-3.  Every operand x is
// split into hi = x rounded to the nearest tf32 value and lo = x - hi (exact in fp32, then rounded
// to tf32 as well); A*B ~= Ahi*Bhi + Ahi*Blo + Alo*Bhi with fp32 accumulation in TMEM, the dropped
// Alo*Blo term being about 2^-24 of the product.
// Data path: kind::tf32 takes K-major operands only (an MN-major B, which the 16-bit kinds accept,
// gives wrong products -- measured), so the row-major B[K,N] is transposed on the way in.  TMA lands
// 128 x 32 fp32 tiles of A with the 128-byte swizzle and 32 x 128 tiles of B as they lie; three groups of four
// converter warps take the stages in turn.  A thread owns one row of A, which it splits into TENSOR MEMORY: the MMAs then
// read only B from shared memory, 4 KB instead of 8 in the 64 clocks that 128 bytes a clock allow for.  It also owns one column
// n of B; when the whole group has its values in registers, the hi and lo parts go, K-major and swizzled, where B and A
// came, so that a stage is 32 KB and six fit.  (With global loads of B by its thread the group stood 2000 clocks of 3450
// issuing them, 32 a block; with a place of its own for the lo part four stages fit, as long as the way from one use of a
// stage to the next.)  One warp issues
// 3 x 4 MMAs per stage; four epilogue warps drain the accumulator through a swizzled staging slab and TMA
// stores.  TMEM holds one pair of accumulators and the A parts of four blocks: a second pair would hide
// the 2 us of an epilogue, but leaves no room for A (2048 x 2048 x 256 takes as long either way).
// With fewer tiles than SMs, clusters share a tile's k blocks (see the launch).  What bounds it now: 880 clocks a block of 32, where its
// MMAs take 780; for small matrices the 3500 clocks to the first MMA and, with clusters, the 5000 after the last one: 32 KB of partial
// sums come from the other CTA at about 16 bytes a clock.  Out-of-range rows/columns read as zero and are clipped on store, so N and K
// need only be multiples of 4 (16-byte row pitches of A, B and C).
// us, with B by global loads and now, inputs in L2 and (from memory): 1024^3 20.6 16.0 (26.6 22.5); 2048^3 113 76 (125 88); 100x1000x2048
// 14.0 12.4 (20.5 18.4); 1900x1500x520 37.8 29.1 (43.0 34.8); 4096x4096x512 112 89 (123 100); 128x128x4096 20.0 15.7 (24.6 22.5).
// Every wait is bounded and abortable; a timed-out wait sets the device status word.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <mutex>

#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {

namespace {

constexpr int kBN = 128;                   // N tile
constexpr int kConvWarps = 4, kConvGroups = 3, kEpiWarps = 4;
constexpr int kConvThreads = kConvWarps * 32, kEpiThreads = kEpiWarps * 32;
constexpr int kThreads = 64 + kConvGroups * kConvThreads + kEpiThreads;
static_assert(64 <= 4 * (kThreads / 32), "four rows a warp finish half of a tile");
constexpr int kTile = 128 * 128;           // bytes of one operand tile: 128 rows (pixels of A / columns of B) x 32 fp32
constexpr int kStageBytes = 2 * kTile;     // A and B as they came, then B lo and B hi in their places
constexpr int kStages = 6, kAStages = 4;   // and parts of A in tensor memory
// TMEM: the accumulators of the hi*hi products and of the cross terms, then A hi and A lo of kAStages blocks
constexpr uint32_t kTmemA = 2 * kBN, kTmemStage = 64;
constexpr int kSlabBytes = 128 * 128;      // 128 rows x 32 fp32

// Nearest tf32 value (10 mantissa bits; ties away from zero): rounding, unlike cutting the low bits,
// leaves no error of one sign to pile up over a long k loop (cutting gave rel-L2 1.5e-5 at K = 2048).
__device__ __forceinline__ float tf32_round(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}

// A load that is under way until its value is used (as `inside ? load : 0` the value is waited for where it is chosen).
__device__ __forceinline__ float load_or_zero(const float* q, bool inside) {
  float v;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.u32 p, %2, 0;\n"
      "mov.f32 %0, 0f00000000;\n"
      "@p ld.global.nc.f32 %0, [%1];\n"
      "}\n"
      : "=&f"(v)
      : "l"(q), "r"((uint32_t)inside));
  return v;
}

struct GtParams {
  const float* bias;
  float* C;
  int* error_flag;
  int M, N, K;
  int m_tiles, n_tiles, k_blocks;
  int relu;
  int splits_log;   // (as a power of two) CTAs of a cluster that share a tile's k blocks (then every cluster has one tile); 1: no clusters
};

__global__ void __launch_bounds__(kThreads, 1)
gemm_tf32x3_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_c,
                   const GtParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_abort;
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t sRing = base;
  const uint32_t sStage = sRing + kStages * kStageBytes;
  const uint32_t bars = sStage + 2 * kSlabBytes;
  const uint32_t full = bars, conv = bars + 8 * kStages, empty = conv + 8 * kStages;
  const uint32_t a_empty = empty + 8 * kStages, acc_full = a_empty + 8 * kAStages, acc_empty = acc_full + 8;
  const uint32_t tmem_slot = acc_empty + 8;
  {
    uint32_t dyn_bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    if (tmem_slot + 4 > raw + dyn_bytes) {
      if (threadIdx.x == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrBounds);
      return;
    }
  }
  const int warp = ptx::warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(full + 8 * i, 1);
      ptx::mbar_init(conv + 8 * i, kConvThreads);
      ptx::mbar_init(empty + 8 * i, 1);
    }
    for (int i = 0; i < kAStages; ++i) ptx::mbar_init(a_empty + 8 * i, 1);
    ptx::mbar_init(acc_full, 1);
    ptx::mbar_init(acc_empty, kEpiThreads);
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_a);
    ptx::prefetch_tensormap(&tm_b);
    if (p.splits_log == 0) ptx::prefetch_tensormap(&tm_c);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, kTmemA + kAStages * kTmemStage);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = (uint32_t)ptx::warp_uniform(*reinterpret_cast<volatile int*>(smem_raw + (tmem_slot - raw)));
  volatile int* abort_flag = &s_abort;

  // all of this before the wait for the previous kernel: with 64-bit divisions behind it the first copy left 1700 clocks later
  const int total = p.m_tiles * p.n_tiles;
  const int S = 1 << p.splits_log, first = (int)blockIdx.x >> p.splits_log, step = (int)gridDim.x >> p.splits_log;
  const int rank = S > 1 ? (int)ptx::cluster_ctarank() : 0;
  const int kb_lo = (p.k_blocks * rank) >> p.splits_log, kb_hi = (p.k_blocks * (rank + 1)) >> p.splits_log;
  const int first_mt = first / p.n_tiles;
  auto item_of = [&](int i, int& m0, int& n0) {
    const int w = first + i * step;
    if (w >= total) return false;
    const int mt = i == 0 ? first_mt : w / p.n_tiles;
    m0 = mt * 128;
    n0 = (w - mt * p.n_tiles) * kBN;
    return true;
  };
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer ----
    if (lane == 0) {
      uint32_t cnt = 0;
      bool okw = true;
      for (int i = 0; okw; ++i) {
        int m0, n0;
        if (!item_of(i, m0, n0)) break;
        for (int kb = kb_lo; kb < kb_hi; ++kb, ++cnt) {
          const uint32_t st = cnt % kStages;
          if (!ptx::mbar_wait_abortable(empty + 8 * st, ((cnt / kStages) & 1u) ^ 1u, abort_flag)) { okw = false; break; }
          ptx::mbar_arrive_expect_tx(full + 8 * st, 2 * kTile);
          ptx::tma_load_2d(sRing + st * kStageBytes, &tm_a, kb * 32, m0, full + 8 * st);
          ptx::tma_load_2d(sRing + st * kStageBytes + kTile, &tm_b, n0, kb * 32, full + 8 * st);
        }
      }
      if (!okw && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer ------
    {
      const uint32_t issue = ptx::elect_one();
      const uint32_t idesc = ptx::umma_idesc(128, kBN, 2);   // kind::tf32, fp32 accumulate, both operands K-major
      uint32_t cnt = 0, acc_cnt = 0;
      bool okw = true;
      for (int i = 0; okw; ++i) {
        int m0, n0;
        if (!item_of(i, m0, n0)) break;
        if (!ptx::warp_wait(acc_empty, (acc_cnt & 1u) ^ 1u, abort_flag)) { okw = false; break; }
        ptx::tc_fence_after();
        // two accumulators: the hi*hi products, and the two small cross terms.  The tensor core
        // cuts (does not round) every accumulation into TMEM, an error of one sign per step: keeping the
        // large sum to one step per k block of 8 instead of three makes it three times smaller
        const uint32_t d = tmem_base, dl = d + kBN;
        for (int kb = kb_lo; kb < kb_hi; ++kb, ++cnt) {
          const uint32_t st = cnt % kStages, ta = cnt % kAStages;
          if (!ptx::warp_wait(conv + 8 * st, (cnt / kStages) & 1u, abort_flag)) { okw = false; break; }
          ptx::tc_fence_after();
          const uint32_t s0 = sRing + st * kStageBytes;
          const uint32_t a_hi = tmem_base + kTmemA + ta * kTmemStage, a_lo = a_hi + 32;
          const uint32_t b_hi = ptx::smem_desc_k128_lo(s0 + kTile), b_lo = ptx::smem_desc_k128_lo(s0);
#pragma unroll
          for (uint32_t k4 = 0; k4 < 4; ++k4) {   // k step of 8 fp32: 8 columns of A, 32 bytes along the rows of B
            const uint64_t bh = ptx::desc_from_halves(b_hi + k4 * 2, ptx::kSmemDescK128Hi);
            const uint64_t bl = ptx::desc_from_halves(b_lo + k4 * 2, ptx::kSmemDescK128Hi);
            ptx::umma_tf32_ts(dl, a_lo + k4 * 8, bh, idesc, kb != kb_lo || k4 != 0 ? 1u : 0u, issue);
            ptx::umma_tf32_ts(dl, a_hi + k4 * 8, bl, idesc, 1u, issue);
            ptx::umma_tf32_ts(d, a_hi + k4 * 8, bh, idesc, kb != kb_lo || k4 != 0 ? 1u : 0u, issue);
          }
          ptx::tc_commit(empty + 8 * st, issue);
          ptx::tc_commit(a_empty + 8 * ta, issue);
        }
        if (!okw) break;
        ptx::tc_commit(acc_full, issue);
        ++acc_cnt;
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitMma);
    }
  } else if (warp < 2 + kConvGroups * kConvWarps) {
    // ------------------------------------------------------------------ transpose B, hi / lo split ----
    const int grp = (warp - 2) / kConvWarps;           // this group takes every kConvGroups-th block
    const int t = (threadIdx.x - 64) % kConvThreads;   // 0..127: column of the B tile / share of the A tile
    const uint32_t swz = (uint32_t)(t & 7);
    const int quad = warp & 3;                         // tensor-memory lanes this warp may write
    bool okw = true;
    // blocks of all tiles of this CTA
    const uint32_t tiles = (uint32_t)(first < total ? (total - first - 1) / step + 1 : 0);
    const uint32_t blocks = tiles * (uint32_t)(kb_hi - kb_lo);
    {
      for (uint32_t cnt = (uint32_t)grp; cnt < blocks; cnt += kConvGroups) {
        const uint32_t st = cnt % kStages, ta = cnt % kAStages;
        // the stage has come, and the MMAs that read these columns of A last have finished
        bool got = ptx::mbar_wait_abortable(full + 8 * st, (cnt / kStages) & 1u, abort_flag);
        got = got && ptx::mbar_wait_abortable(a_empty + 8 * ta, ((cnt / kAStages) & 1u) ^ 1u, abort_flag);
        if (!ptx::named_bar_and(4 + grp, kConvThreads, got)) { okw = false; break; }
        const uint32_t s0 = sRing + st * kStageBytes;
        ptx::tc_fence_after();
        float bv[32];   // column t of B: 32 rows of 128 columns, a warp's loads of one row meet no bank twice
#pragma unroll
        for (int k = 0; k < 32; ++k)
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(bv[k]) : "r"(s0 + kTile + (uint32_t)k * (kBN * 4) + (uint32_t)t * 4u));
        // row (quad, lane) of A: out of shared memory, in two parts into tensor memory
        const uint32_t arow = s0 + (uint32_t)(quad * 32 + lane) * 128u;
        const uint32_t acol = tmem_base + ((uint32_t)(quad * 32) << 16) + kTmemA + ta * kTmemStage;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float hi[16], lo[16];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                         : "r"(arow + (((uint32_t)(h * 4 + c) ^ (uint32_t)(lane & 7)) << 4)));
            const float in[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              hi[c * 4 + e] = tf32_round(in[e]);
              lo[c * 4 + e] = tf32_round(in[e] - hi[c * 4 + e]);
            }
          }
          ptx::tmem_st_32x16(acol + h * 16, hi);
          ptx::tmem_st_32x16(acol + 32 + h * 16, lo);
        }
        // every thread of the group has its values in registers: the parts of B go where A and B were
        ptx::named_bar_sync(4 + grp, kConvThreads);
        // column n of B becomes row t of the K-major tiles: 8 chunks of 4 k values, chunk index XOR (row % 8)
        const uint32_t brow = s0 + (uint32_t)t * 128u;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            hi[e] = tf32_round(bv[4 * j + e]);
            lo[e] = tf32_round(bv[4 * j + e] - hi[e]);
          }
          const uint32_t dst = brow + (((uint32_t)j ^ swz) << 4);
          asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(dst + kTile), "f"(hi[0]), "f"(hi[1]), "f"(hi[2]), "f"(hi[3]) : "memory");
          asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "f"(lo[0]), "f"(lo[1]), "f"(lo[2]), "f"(lo[3]) : "memory");
        }
        ptx::fence_proxy_async_smem();
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        ptx::mbar_arrive(conv + 8 * st);
      }
    }
    if (!okw && p.error_flag && t == 0) atomicCAS(p.error_flag, 0, (int)kErrWaitLoader);
  } else {
    // ------------------------------------------------------------------ epilogue --------
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const bool elected = threadIdx.x == 64 + kConvGroups * kConvThreads;
    const uint32_t sw = (uint32_t)(row & 7);
    uint32_t acc_cnt = 0;
    int jglob = 0;
    bool okw = true;
    for (int i = 0; okw; ++i) {
      int m0, n0;
      if (!item_of(i, m0, n0)) break;
      const bool got = ptx::mbar_wait_abortable(acc_full, acc_cnt & 1u, abort_flag);
      if (!ptx::named_bar_and(3, kEpiThreads, got)) { okw = false; break; }
      ptx::tc_fence_after();
      if (S > 1) {   // partial sums into the ring, which nothing reads or fills any more: the tile's MMAs are complete
        for (int sl = 0; sl < kBN / 32; ++sl) {
          uint32_t acc[32], accl[32];
          __syncwarp();
          ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(sl * 32), acc);
          ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + kBN + (uint32_t)(sl * 32), accl);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4) {
            float o[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) o[h] = __uint_as_float(acc[c4 * 4 + h]) + __uint_as_float(accl[c4 * 4 + h]);
            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(sRing + (uint32_t)row * (kBN * 4) + (((uint32_t)(sl * 8 + c4) ^ sw) << 4)),
                         "f"(o[0]), "f"(o[1]), "f"(o[2]), "f"(o[3])
                         : "memory");
          }
        }
        break;
      }
      for (int sl = 0; sl < kBN / 32; ++sl, ++jglob) {
        const uint32_t sb = (uint32_t)jglob & 1u;
        const int ncol = n0 + sl * 32;
        uint32_t acc[32], accl[32];
        __syncwarp();
        ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(sl * 32), acc);
        ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + kBN + (uint32_t)(sl * 32), accl);
        ptx::tmem_ld_wait();
        if (sl == kBN / 32 - 1) {
          ptx::tc_fence_before();
          ptx::mbar_arrive(acc_empty);
        }
        const uint32_t srow = sStage + sb * kSlabBytes + (uint32_t)row * 128u;
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4) {
          float o[4];
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int n = ncol + c4 * 4 + h;
            float a = __uint_as_float(acc[c4 * 4 + h]) + __uint_as_float(accl[c4 * 4 + h]);
            if (p.bias && n < p.N) a += __ldg(p.bias + n);
            o[h] = p.relu ? (!(a <= 0.0f) ? a : 0.0f) : a;
          }
          asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(srow + (((uint32_t)c4 ^ sw) << 4)), "f"(o[0]), "f"(o[1]),
                       "f"(o[2]), "f"(o[3])
                       : "memory");
        }
        ptx::fence_proxy_async_smem();
        ptx::named_bar_sync(1, kEpiThreads);
        if (elected) {
          if (ncol < p.N) ptx::tma_store_2d(&tm_c, ncol, m0, sStage + sb * kSlabBytes);
          ptx::bulk_commit();
          ptx::bulk_wait_read<1>();
        }
        ptx::named_bar_sync(2, kEpiThreads);
      }
      ++acc_cnt;
    }
    if (elected) ptx::bulk_wait<0>();
    if (!okw && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitEpilogue);
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (S > 1) {
    // every CTA finishes its share of the rows from all partial sums, in rank order: the result does not depend on timing
    int m0, n0;
    item_of(0, m0, n0);
    const int n = n0 + lane * 4, rows = 128 / S;
    float bias[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) bias[e] = load_or_zero(p.bias + n + e, p.bias != nullptr && n < p.N);
    ptx::cluster_sync_all();
    // a warp's rows, at most 8 / S of them: the parts of all are asked for before the first is added
    float4 part[8];
    auto row_of = [&](int e) { return rank * rows + warp + (e >> p.splits_log) * (kThreads / 32); };
    auto mine = [&](int r) { return r < (rank + 1) * rows && m0 + r < p.M && !s_abort; };   // the same for the whole warp
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = row_of(e), q = e & (S - 1);
      if (!mine(r)) continue;
      const uint32_t at = sRing + (uint32_t)r * (kBN * 4) + (((uint32_t)lane ^ (uint32_t)(r & 7)) << 4);
      if (q == rank) asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(part[e].x), "=f"(part[e].y), "=f"(part[e].z), "=f"(part[e].w) : "r"(at));
      else part[e] = ptx::ld_cluster_f4(ptx::map_to_cta(at, (uint32_t)q));
    }
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = row_of(e);
      if (!mine(r)) continue;
      if ((e & (S - 1)) == 0) v = part[e];
      else { v.x += part[e].x; v.y += part[e].y; v.z += part[e].z; v.w += part[e].w; }
      if ((e & (S - 1)) != S - 1) continue;
      v.x += bias[0]; v.y += bias[1]; v.z += bias[2]; v.w += bias[3];
      if (p.relu) {
        v.x = !(v.x <= 0.0f) ? v.x : 0.0f; v.y = !(v.y <= 0.0f) ? v.y : 0.0f;
        v.z = !(v.z <= 0.0f) ? v.z : 0.0f; v.w = !(v.w <= 0.0f) ? v.w : 0.0f;
      }
      if (n < p.N) *reinterpret_cast<float4*>(p.C + (size_t)(m0 + r) * p.N + n) = v;
    }
    __syncwarp();
    ptx::cluster_sync_all();   // the peers' reads of this CTA's partial sums are over
  }
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, kTmemA + kAStages * kTmemStage);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 gt_get_encode() {
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

// 2-D map over a row-major fp32 [rows, cols] matrix; swizzle: rows of 128 bytes (32 columns) with the 128-byte swizzle.
bool gt_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, int box_cols, int box_rows, bool swizzle) {
  auto enc = gt_get_encode();
  if (!enc) return false;
  cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t gstr[1] = {(cuuint64_t)cols * 4};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool gemm_tf32x3_supported(int M, int N, int K) { return M > 0 && N >= 32 && K >= 32 && N % 4 == 0 && K % 4 == 0; }

cudaError_t launch_gemm_tf32x3(const float* A, const float* B, float* C, int M, int N, int K, const float* bias, int relu,
                               int sm_count, int* error_flag, cudaStream_t stream) {
  if (!gemm_tf32x3_supported(M, N, K)) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (reinterpret_cast<uintptr_t>(C) & 15))
    return cudaErrorMisalignedAddress;
  GtParams p{};
  p.bias = bias; p.C = C; p.error_flag = error_flag; p.M = M; p.N = N; p.K = K; p.relu = relu;
  p.m_tiles = (M + 127) / 128; p.n_tiles = (N + kBN - 1) / kBN; p.k_blocks = (K + 31) / 32;
  if ((long long)p.m_tiles * p.n_tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
  CUtensorMap tm_a, tm_b, tm_c = {};   // shared tiles are written without a map
  if (!gt_map(&tm_a, A, M, K, 32, 128, true) || !gt_map(&tm_b, B, K, N, kBN, 32, false)) return cudaErrorInvalidValue;
  const size_t smem = 1024 + (size_t)kStages * kStageBytes + 2 * kSlabBytes + 256;
  cudaError_t e = cudaFuncSetAttribute(gemm_tf32x3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int sms = sm_count > 0 ? sm_count : 148;
  const int items = p.m_tiles * p.n_tiles;
  // Fewer tiles than SMs: clusters split the k blocks of a tile, as far as all of them run at once and each CTA keeps four
  // blocks (a block takes about 0.5 us, the exchange of partial sums 2.5).
  static const ClusterFit fit = cluster_fit(gemm_tf32x3_kernel, kThreads, smem, sms);
  int splits = 1;
  for (int s = 2; s <= 8; s *= 2) {
    if (items > fit.of[s] || p.k_blocks < 4 * s) break;
    splits = s;
    ++p.splits_log;
  }
  if (splits == 1 && !gt_map(&tm_c, C, M, N, 32, 128, true)) return cudaErrorInvalidValue;
  if (splits == 1) return launch_pdl(gemm_tf32x3_kernel, dim3(items < sms ? items : sms), dim3(kThreads), smem, stream, tm_a, tm_b, tm_c, p);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(items * splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, gemm_tf32x3_kernel, tm_a, tm_b, tm_c, p);
}

}  // namespace nncv_b200
