// 3x3 stride-1 pad-1 convolution for sm_100a: implicit GEMM on tcgen05 whose A operand is
// nine SHIFTED VIEWS of one shared-memory halo tile, so every input element crosses the
// L2->SM path once per tile instead of nine times.
//
// Replaces, for the thirteen 3x3 stride-1 convolutions of ResNet-18 (tests/Nets/Res18.mlir:157,
// 180, 208, 231 ... 582, each preceded by a zero tensor.pad, :152-156), what nncv lowers to
// tiled scf.for nests (src/nncv/compiler/Conversion/CodeGen/LlvmCpu/ModernTile.cpp:184-199).
//
// Activation layout ("shared-pad NHWC"): a logical [N,H,W,C] tensor is stored as
// [N, H+1, W+1, C]; row 0 of every image and column 0 of every row are zero.  With the row
// pitch P = W+1 the pad column of row y+1 doubles as the right neighbour of the last pixel of
// row y, and row 0 of image n+1 doubles as the bottom pad of image n.  Flattening
// (n, y, x) -> slot q = (n*(H+1) + y)*P + x turns the convolution into
//     out[q] = sum_{r,s in 0..2} W[r][s] * in[q + (r-1)*P + (s-1)]
// for every slot; slots that are pads are computed too (4-23 % extra MMA work, depending on W)
// and stored as zeros, which keeps the output in the same layout with its pads clean.
//
// Kernel (persistent, 10 warps):
//   warp 0  one thread: TMA loads.  Per (tile, 64-channel block) ONE tiled copy brings rows
//           [q0-P-1, q0+MT*128+P+1) x 64 channels into shared memory (128-byte swizzle; rows
//           before slot 0 / past the end are zero-filled by TMA).  Weights are pre-packed
//           [Kout tile][tap][channel block] images: either all of them stay resident in shared
//           memory for the whole kernel, or they stream through a ring, one BN x 64 tile per tap.
//   warp 1  one thread: tcgen05.mma.  For tap (r,s) the A descriptor simply starts
//           (r*P+s)*128 bytes into the halo tile: the 128-byte swizzle is a function of the
//           absolute shared-memory address, so a view shifted by whole rows reads consistently.
//           MT accumulators of 128 x BN fp32 live in TMEM, double-buffered when they fit.
//   warps 2-9  epilogue (epilogue.cuh; two warps per TMEM lane quadrant, slabs in turn): tcgen05.ld, scale/shift
//           (+ residual, brought into the staging buffer by TMA) (+ ReLU), zero the pad slots, convert, TMA store.
// Every wait is bounded and abortable; a timed-out wait sets the device status word.
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

constexpr int kThreads = 64 + epi::kThreads;  // warp 0 TMA, warp 1 MMA, warps 2.. epilogue
constexpr int kMaxInStages = 4;
constexpr int kMaxWStages = 8;
constexpr size_t kBarBytes = 8 * (2 * kMaxInStages + 2 * kMaxWStages + 4 + epi::kWarps * epi::kMaxBufs) + 16;

struct C3Params {
  const uint8_t* wpack;
  const float* scale;
  const float* shift;
  int Kout;
  int* error_flag;
  int T;          // total slots
  int P;          // row pitch in slots (W + 1)
  int Himg;       // rows per image (H + 1)
  epi::FastDiv div_p, div_h, div_nt;   // by P, Himg, n_tiles
  int CB;         // channel blocks of 64
  int n_tiles;    // Kout / BN
  int m_items;    // ceil(T / (MT * 128))
  int box_rows;   // rows per TMA box of the input tile (multiple of 8)
  int in_boxes;   // boxes per input stage
  int in_stages;  // input ring depth
  int w_stages;   // weight ring depth (streamed mode)
  int relu, bf16;
  int has_res;    // tm_res holds a shared-pad [T, Kout] tensor that is added before the activation
  int epi_bufs;   // staging buffers per epilogue warp (1 .. epi::kMaxBufs)
};

template <int BN, int MT, bool RESIDENT>
__global__ void __launch_bounds__(kThreads, 1)
conv3x3_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out,
               const __grid_constant__ CUtensorMap tm_res, const C3Params p) {
  constexpr int AB = (2 * MT * BN <= 512) ? 2 : 1;  // accumulator buffers in TMEM
  constexpr int ACC_COLS = AB * MT * BN;
  constexpr int WTILE = BN * 128;
  constexpr int SLABS = BN / 64;       // 64-column slabs per 128-row sub-tile
  constexpr int SPI = MT * SLABS;      // slabs per work item

  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ __align__(16) float4 s_cols[epi::kWarps][32];   // scale / shift of the slab each epilogue warp works on
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const int in_stage_bytes = p.in_boxes * p.box_rows * 128;  // multiple of 1024
  const int kb_total = 9 * p.CB;
  const uint32_t sIn = base;
  const uint32_t sW = sIn + (uint32_t)p.in_stages * in_stage_bytes;
  const uint32_t sStage = sW + (uint32_t)(RESIDENT ? kb_total : p.w_stages) * WTILE;
  const uint32_t bars = sStage + (uint32_t)(epi::kWarps * p.epi_bufs) * epi::kBufBytes;
  const uint32_t in_full = bars, in_empty = bars + 8 * kMaxInStages;
  const uint32_t w_full = in_empty + 8 * kMaxInStages, w_empty = w_full + 8 * kMaxWStages;
  const uint32_t acc_full = w_empty + 8 * kMaxWStages, acc_empty = acc_full + 16;
  const uint32_t res_full = acc_empty + 16;
  const uint32_t tmem_slot = res_full + 8 * epi::kWarps * epi::kMaxBufs;
  {
    // the carve-up above must fit the dynamic shared memory of this launch: refuse to run otherwise
    uint32_t dyn_bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    if (tmem_slot + 4 > raw + dyn_bytes) {
      if (threadIdx.x == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrBounds);
      return;
    }
  }

  const int warp = ptx::warp_uniform((int)threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kMaxInStages; ++i) {
      ptx::mbar_init(in_full + 8 * i, 1);
      ptx::mbar_init(in_empty + 8 * i, 1);
    }
    for (int i = 0; i < kMaxWStages; ++i) {
      ptx::mbar_init(w_full + 8 * i, 1);
      ptx::mbar_init(w_empty + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(acc_full + 8 * i, 1);
      ptx::mbar_init(acc_empty + 8 * i, epi::kWarps);
    }
    for (int i = 0; i < epi::kWarps * epi::kMaxBufs; ++i) ptx::mbar_init(res_full + 8 * i, 1);
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_in);
    ptx::prefetch_tensormap(&tm_out);
    if (p.has_res) ptx::prefetch_tensormap(&tm_res);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, ACC_COLS);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = (uint32_t)ptx::warp_uniform(*reinterpret_cast<volatile int*>(smem_raw + (tmem_slot - raw)));
  volatile int* abort_flag = &s_abort;

  // Work items of this CTA.  Resident weights pin the CTA to one Kout tile (blockIdx.y) and it
  // strides over the slot tiles; streamed mode strides over (slot tile, Kout tile) pairs with the
  // Kout tiles of one slot tile adjacent, so that they share the input tile in L2.
  const int total_items = RESIDENT ? p.m_items : p.m_items * p.n_tiles;
  auto item_of = [&](int i, int& m_item, int& n_tile) {
    const int w = (int)blockIdx.x + i * (int)gridDim.x;
    if (RESIDENT) {
      m_item = w;
      n_tile = (int)blockIdx.y;
    } else {
      m_item = (int)epi::div_by((uint32_t)w, p.div_nt);
      n_tile = w - m_item * p.n_tiles;
    }
    return w < total_items;
  };

  // Packed weights never change, so their copies start before the previous kernel of the stream has finished.
  auto weight_tile = [&](int n_tile, int cb, int tap) { return p.wpack + ((size_t)n_tile * kb_total + (size_t)tap * p.CB + cb) * WTILE; };
  uint32_t early = 0;   // stages of the weight ring already on their way
  if (warp == 0) {
    const uint32_t issue = ptx::elect_one();
    if (RESIDENT) {
      const uint8_t* src = p.wpack + (size_t)blockIdx.y * kb_total * WTILE;
      ptx::mbar_arrive_expect_tx(w_full, (uint32_t)kb_total * WTILE, issue);
      for (int i = 0; i < kb_total; ++i)
        ptx::bulk_g2s(sW + (uint32_t)i * WTILE, src + (size_t)i * WTILE, WTILE, w_full, issue);
    } else {
      for (int i = 0; early < (uint32_t)p.w_stages; ++i) {
        int m_item, n_tile;
        if (!item_of(i, m_item, n_tile)) break;
        for (int cb = 0; cb < p.CB && early < (uint32_t)p.w_stages; ++cb)
          for (int tap = 0; tap < 9 && early < (uint32_t)p.w_stages; ++tap, ++early) {
            ptx::mbar_arrive_expect_tx(w_full + 8 * early, WTILE, issue);
            ptx::bulk_g2s(sW + early * WTILE, weight_tile(n_tile, cb, tap), WTILE, w_full + 8 * early, issue);
          }
      }
    }
  }
  // The rest reads what the previous kernel wrote, or writes what it may still be reading.
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer ----
    {
      const uint32_t issue = ptx::elect_one();
      uint32_t w_cnt = 0, st = 0, par = 1, ws = 0, wpar = 1, w_seen = 1;   // stages, parities of their rings' rounds
      bool okw = true;
      for (int i = 0; okw; ++i) {
        int m_item, n_tile;
        if (!item_of(i, m_item, n_tile)) break;
        const int row0 = m_item * (MT * 128) - p.P - 1;
        for (int cb = 0; cb < p.CB && okw; ++cb) {
          if (!ptx::warp_wait(in_empty + 8 * st, par, abort_flag)) { okw = false; break; }
          ptx::mbar_arrive_expect_tx(in_full + 8 * st, (uint32_t)in_stage_bytes, issue);
          for (int b = 0; b < p.in_boxes; ++b)
            ptx::tma_load_2d(sIn + st * in_stage_bytes + (uint32_t)b * p.box_rows * 128, &tm_in, cb * 64,
                             row0 + b * p.box_rows, in_full + 8 * st, issue);
          if (++st == (uint32_t)p.in_stages) { st = 0; par ^= 1u; }
          if (!RESIDENT) {
            for (int tap = 0; tap < 9; ++tap, ++w_cnt) {
              if (w_cnt >= early) {
                if (!ptx::warp_all(w_seen) && !ptx::warp_wait(w_empty + 8 * ws, wpar, abort_flag)) { okw = false; break; }
                ptx::mbar_arrive_expect_tx(w_full + 8 * ws, WTILE, issue);
                ptx::bulk_g2s(sW + ws * WTILE, weight_tile(n_tile, cb, tap), WTILE, w_full + 8 * ws, issue);
              }
              if (++ws == (uint32_t)p.w_stages) { ws = 0; wpar ^= 1u; }
              w_seen = ptx::mbar_peek(w_empty + 8 * ws, wpar);
            }
          }
        }
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer ------
    {
      const uint32_t issue = ptx::elect_one();
      const uint32_t idesc = ptx::umma_idesc(128, BN, p.bf16 ? 1 : 0);
      bool okw = true;
      if (RESIDENT) okw = ptx::warp_wait(w_full, 0, abort_flag);
      uint32_t in_st = 0, in_ring = 0, acc_cnt = 0;
      uint32_t ws = 0, w_ring = 0;   // weight stage, parity of the ring's round
      uint32_t w_seen = RESIDENT || !okw ? 0u : ptx::mbar_peek(w_full, 0);
      for (int i = 0; okw; ++i) {
        int m_item, n_tile;
        if (!item_of(i, m_item, n_tile)) break;
        const uint32_t ab = acc_cnt % AB;
        if (!ptx::warp_wait(acc_empty + 8 * ab, ((acc_cnt / AB) & 1u) ^ 1u, abort_flag)) { okw = false; break; }
        ptx::tc_fence_after();
        const uint32_t d_base = tmem_base + ab * (MT * BN);
        for (int cb = 0; cb < p.CB && okw; ++cb) {
          const uint32_t st = in_st;
          if (!ptx::warp_wait(in_full + 8 * st, in_ring, abort_flag)) { okw = false; break; }
          if (++in_st == (uint32_t)p.in_stages) { in_st = 0; in_ring ^= 1u; }
          ptx::tc_fence_after();
          const uint32_t a_stage = sIn + st * in_stage_bytes;
          for (int tap = 0; tap < 9; ++tap) {
            uint32_t w_addr;
            const uint32_t w_now = ws;
            if (RESIDENT) {
              w_addr = sW + (uint32_t)(tap * p.CB + cb) * WTILE;
            } else {
              if (!ptx::warp_all(w_seen) && !ptx::warp_wait(w_full + 8 * ws, w_ring, abort_flag)) { okw = false; break; }
              ptx::tc_fence_after();
              w_addr = sW + ws * WTILE;
              if (++ws == (uint32_t)p.w_stages) { ws = 0; w_ring ^= 1u; }
              w_seen = ptx::mbar_peek(w_full + 8 * ws, w_ring);
            }
            const int r = tap / 3, s = tap - 3 * r;
            // descriptors differ only in the address bits of the low word: one add per MMA
            const uint32_t a_lo = ptx::smem_desc_k128_lo(a_stage + (uint32_t)(r * p.P + s) * 128u);
            const uint32_t b_lo = ptx::smem_desc_k128_lo(w_addr);
            const uint32_t first = (cb | tap) != 0 ? 1u : 0u;
#pragma unroll
            for (int t = 0; t < MT; ++t) {
#pragma unroll
              for (int k4 = 0; k4 < 4; ++k4) {
                ptx::umma_f16(d_base + t * BN,
                              ptx::desc_from_halves(a_lo + (uint32_t)(t * (128 * 128) + k4 * 32) / 16u, ptx::kSmemDescK128Hi),
                              ptx::desc_from_halves(b_lo + (uint32_t)(k4 * 32) / 16u, ptx::kSmemDescK128Hi), idesc,
                              k4 == 0 ? first : 1u, issue);
              }
            }
            if (!RESIDENT) ptx::tc_commit(w_empty + 8 * w_now, issue);
          }
          ptx::tc_commit(in_empty + 8 * st, issue);
        }
        ptx::tc_commit(acc_full + 8 * ab, issue);
        ++acc_cnt;
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitMma);
    }
  } else {
    // ------------------------------------------------------------------ epilogue --------
    // Eight independent warps (epilogue.cuh); slabs of an item: sub-tile major, then 64 columns.
    const int ew = warp - 2, quad = warp & 3, half = ew >> 2;
    const int nb = p.epi_bufs;
    const uint32_t my_stage = sStage + (uint32_t)(ew * nb) * epi::kBufBytes;
    const uint32_t my_res = res_full + (uint32_t)(ew * epi::kMaxBufs) * 8u;
    const uint32_t tab = ptx::smem_u32(&s_cols[ew][0]);
    const int mode = epi::mode_of(p.bf16 != 0, p.has_res != 0, p.relu != 0, 0);
    // slab j -> first slot of this warp's rows, first column
    auto slab_of = [&](int j, int& q0, int& ncol) {
      const int i = j / SPI, rem = j - i * SPI;
      int m_item, n_tile;
      if (!item_of(i, m_item, n_tile)) return false;
      const int t = rem / SLABS, sl = rem - t * SLABS;
      q0 = m_item * (MT * 128) + t * 128 + quad * 32;
      ncol = n_tile * BN + sl * 64;
      return true;
    };
    uint32_t phase = 0, inflight = 0;   // per staging buffer: parity of its next residual, one on its way
    int ahead_j = half, ahead_b = 0;
    auto fetch_res = [&]() {   // residual rows of the next slab in line -> its staging buffer
      int q0, ncol;
      if (slab_of(ahead_j, q0, ncol) && q0 < p.T) {
        inflight |= 1u << ahead_b;
        if (lane == 0) {
          ptx::mbar_arrive_expect_tx(my_res + 8 * ahead_b, epi::kBufBytes);
          ptx::tma_load_2d(my_stage + (uint32_t)ahead_b * epi::kBufBytes, &tm_res, ncol, q0, my_res + 8 * ahead_b);
        }
      }
      ahead_j += 2;
      if (++ahead_b == nb) ahead_b = 0;
    };
    int j = half, b = 0;
    int q0 = 0, ncol = 0;
    bool have = slab_of(j, q0, ncol);
    epi::ColParams cols = epi::fetch_cols(p.scale, p.shift, have ? ncol : 0, p.Kout, lane);
    if (p.has_res)
      for (int k = 0; k + 1 < nb; ++k) fetch_res();
    bool okw = true;
    for (int i = 0; okw; ++i) {
      int m_item, n_tile;
      if (!item_of(i, m_item, n_tile)) break;
      const uint32_t ab = (uint32_t)i % AB;
      okw = ptx::mbar_wait_abortable(acc_full + 8 * ab, ((uint32_t)i / AB) & 1u, abort_flag);
      okw = __all_sync(0xffffffffu, okw);
      if (!okw) break;
      ptx::tc_fence_after();
      auto hand_back = [&]() {   // this warp has read its part of the accumulator
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(acc_empty + 8 * ab);
      };
      const int end_j = (i + 1) * SPI;
      if (j >= end_j) hand_back();   // no slab of this item is this warp's
      for (; j < end_j; j += 2) {
        const int rem = j - i * SPI;
        const int t = rem / SLABS, sl = rem - t * SLABS;
        const bool live = q0 < p.T;
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + ab * (MT * BN) + (uint32_t)(t * BN + sl * 64);
        uint32_t acc[64];
        epi::load_slab(taddr, acc);
        epi::put_cols(tab, cols, lane);
        if (p.has_res) {
          if (lane == 0) ptx::bulk_wait_read<0>();   // the buffer the next residual goes to was stored from one slab ago
          __syncwarp();
          fetch_res();
        } else if (lane == 0) {
          if (nb == 1) ptx::bulk_wait_read<0>();
          else ptx::bulk_wait_read<1>();
        }
        // pad slots (column 0 of a row, row 0 of an image) leave as zeros
        const int q = q0 + lane;
        const uint32_t yrow = epi::div_by((uint32_t)q, p.div_p), img = epi::div_by(yrow, p.div_h);
        const bool keep = (uint32_t)q != yrow * (uint32_t)p.P && yrow != img * (uint32_t)p.Himg;
        ptx::tmem_ld_wait();
        __syncwarp();
        if (j + 2 >= end_j) hand_back();
        int q0n = 0, ncoln = 0;
        have = slab_of(j + 2, q0n, ncoln);
        cols = epi::fetch_cols(p.scale, p.shift, have ? ncoln : 0, p.Kout, lane);
        if (live) {
          const uint32_t buf = my_stage + (uint32_t)b * epi::kBufBytes;
          if (p.has_res) {
            okw = ptx::mbar_wait_abortable(my_res + 8 * b, (phase >> b) & 1u, abort_flag);
            okw = __all_sync(0xffffffffu, okw);
            if (!okw) break;
            phase ^= 1u << b;
            inflight &= ~(1u << b);
          }
          epi::slab64_by_mode<1>(mode, acc, tab, buf, lane);
          epi::zero_pads(buf, lane, keep);
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_2d(&tm_out, ncol, q0, buf);
            ptx::bulk_commit();
          }
        }
        __syncwarp();
        q0 = q0n;
        ncol = ncoln;
        if (++b == nb) b = 0;
      }
    }
    if (!okw) {
      if (lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitEpilogue);
      for (int k = 0; k < nb; ++k)   // residual rows still on their way land before the block ends
        if ((inflight >> k) & 1u) ptx::mbar_wait_limit(my_res + 8 * k, (phase >> k) & 1u, 1LL << 24);
    }
    if (lane == 0) ptx::bulk_wait<0>();
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, ACC_COLS);
  }
}

// ------------------------------------------------------------------------ host side -----
PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
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

// 2-D map over a row-major [rows, cols] 16-bit tensor, box = 64 columns x box_rows rows,
// 128-byte swizzle, out-of-range elements read as zero.
bool make_map(CUtensorMap* m, const void* ptr, long long rows, int cols, int box_rows, bool bf16) {
  auto enc = get_encode();
  if (!enc) return false;
  cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t gstr[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
             const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr size_t kSmemLimit = 222 * 1024;   // dynamic part; the kernel also holds 4 KB of static shared memory

template <int BN, int MT, bool RESIDENT>
cudaError_t launch_cfg(const Conv3x3Args& a, cudaStream_t stream) {
  C3Params p;
  p.wpack = static_cast<const uint8_t*>(a.wpack);
  p.scale = a.scale; p.shift = a.shift; p.error_flag = a.error_flag;
  p.Kout = a.Kout; p.has_res = a.residual != nullptr;
  p.P = a.W + 1; p.Himg = a.H + 1;
  p.div_p = epi::fast_div((uint32_t)p.P); p.div_h = epi::fast_div((uint32_t)p.Himg);
  const long long T = (long long)a.N * p.Himg * p.P;
  if (T <= 0 || T > 0x7fffff00LL) return cudaErrorInvalidValue;
  p.T = (int)T;
  p.CB = a.C / 64;
  p.n_tiles = a.Kout / BN;
  p.div_nt = epi::fast_div((uint32_t)p.n_tiles);
  p.m_items = (int)((T + MT * 128 - 1) / (MT * 128));
  const int rows_in = MT * 128 + 2 * p.P + 2;
  p.in_boxes = (rows_in + 255) / 256;
  p.box_rows = ((rows_in + p.in_boxes - 1) / p.in_boxes + 7) & ~7;
  if (p.box_rows > 256) return cudaErrorInvalidValue;
  const size_t in_stage = (size_t)p.in_boxes * p.box_rows * 128;
  const size_t wtile = (size_t)BN * 128;
  const size_t wres = (size_t)9 * p.CB * wtile;
  p.epi_bufs = epi::pick_bufs(p.has_res != 0, kSmemLimit - 1024 - kBarBytes, (RESIDENT ? wres : 4 * wtile) + 2 * in_stage,
                              (RESIDENT ? wres : 2 * wtile) + 2 * in_stage);
  const size_t fixed = 1024 + (size_t)(epi::kWarps * p.epi_bufs) * epi::kBufBytes + kBarBytes;
  size_t wbytes;
  if (RESIDENT) {
    wbytes = (size_t)9 * p.CB * wtile;
    if (fixed + wbytes + in_stage > kSmemLimit) return cudaErrorInvalidConfiguration;
    p.w_stages = 0;
    size_t room = kSmemLimit - fixed - wbytes;
    p.in_stages = (int)(room / in_stage);
    if (p.in_stages > kMaxInStages) p.in_stages = kMaxInStages;
  } else {
    p.in_stages = fixed + 2 * in_stage + 2 * wtile <= kSmemLimit ? 2 : 1;   // very wide maps: one halo tile at a time
    if (fixed + p.in_stages * in_stage + 2 * wtile > kSmemLimit) return cudaErrorInvalidConfiguration;
    size_t room = kSmemLimit - fixed - p.in_stages * in_stage;
    p.w_stages = (int)(room / wtile);
    if (p.w_stages > kMaxWStages) p.w_stages = kMaxWStages;
    // spare room beyond a deep weight ring goes to a third input stage
    if (p.w_stages >= 5 && fixed + 3 * in_stage + 4 * wtile <= kSmemLimit) {
      p.in_stages = 3;
      room = kSmemLimit - fixed - 3 * in_stage;
      p.w_stages = (int)(room / wtile);
      if (p.w_stages > kMaxWStages) p.w_stages = kMaxWStages;
    }
    wbytes = (size_t)p.w_stages * wtile;
  }
  const size_t smem = fixed + wbytes + (size_t)p.in_stages * in_stage;
  p.relu = a.relu; p.bf16 = a.ab == kBF16;

  CUtensorMap tm_in, tm_out, tm_res;
  if (!make_map(&tm_in, a.in, T, a.C, p.box_rows, p.bf16) || !make_map(&tm_out, a.out, T, a.Kout, 32, p.bf16) ||
      !make_map(&tm_res, p.has_res ? a.residual : a.out, T, a.Kout, 32, p.bf16))
    return cudaErrorInvalidValue;

  auto kern = conv3x3_kernel<BN, MT, RESIDENT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int sms = a.sm_count > 0 ? a.sm_count : 148;
  dim3 grid;
  if (RESIDENT) {
    int gx = sms / p.n_tiles;
    if (gx < 1) gx = 1;
    if (gx > p.m_items) gx = p.m_items;
    grid = dim3(gx, p.n_tiles);
  } else {
    const int items = p.m_items * p.n_tiles;
    grid = dim3(items < sms ? items : sms, 1);
  }
  return launch_pdl(kern, grid, dim3(kThreads), smem, stream, tm_in, tm_out, tm_res, p);
}

}  // namespace


bool conv3x3_supported(int C, int Kout, int R, int S, int stride, int pad) {
  return R == 3 && S == 3 && stride == 1 && pad == 1 && C % 64 == 0 && Kout % 64 == 0 && C >= 64;
}

// Tile configuration, from timing every variant on the four ResNet-18 layer shapes at batch 256.
// With 64 input channels all nine weight tiles of a 64-wide Kout tile stay resident in shared
// memory; wider layers stream weights and favour the widest N tile (fewer passes over the input,
// and tcgen05.mma runs closer to its peak rate as N grows).
Conv3x3Config conv3x3_pick(int N, int H, int W, int C, int Kout, int has_res) {
  Conv3x3Config c;
  (void)N; (void)H; (void)W;
  if (C <= 64) {
    c.bn = 64; c.resident = 1; c.mt = has_res ? 1 : 2;
  } else if (C <= 128 || Kout % 256 != 0) {
    c.resident = 0; c.bn = Kout % 128 == 0 ? 128 : 64; c.mt = 2;
  } else if (C <= 256) {
    c.resident = 0; c.bn = 256; c.mt = 1;
  } else {
    c.resident = 0; c.bn = 256; c.mt = 2;
  }
  // Small batches: shrink the tile until the persistent grid has an item for every SM.
  const long long T = (long long)N * (H + 1) * (W + 1);
  auto items = [&]() { return ((T + c.mt * 128 - 1) / (c.mt * 128)) * (c.resident ? 1 : Kout / c.bn); };
  while (items() < 148) {
    if (c.mt > 1) c.mt >>= 1;
    else if (!c.resident && c.bn > 64) c.bn >>= 1;
    else break;
  }
  return c;
}

cudaError_t launch_conv3x3(const Conv3x3Args& a, cudaStream_t stream) {
  if (!conv3x3_supported(a.C, a.Kout, 3, 3, 1, 1) || a.ab == kF32) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(a.in) & 15) || (reinterpret_cast<uintptr_t>(a.out) & 15) ||
      (reinterpret_cast<uintptr_t>(a.residual) & 15) || (reinterpret_cast<uintptr_t>(a.wpack) & 15))
    return cudaErrorMisalignedAddress;
  if (a.Kout % a.bn != 0) return cudaErrorInvalidValue;
#define NNCV_C3(BN_, MT_, RES_) \
  if (a.bn == BN_ && a.mt == MT_ && (a.resident != 0) == RES_) return launch_cfg<BN_, MT_, RES_>(a, stream);
  NNCV_C3(64, 1, true)
  NNCV_C3(64, 2, true)
  NNCV_C3(64, 1, false)
  NNCV_C3(64, 2, false)
  NNCV_C3(128, 1, false)
  NNCV_C3(128, 2, false)
  NNCV_C3(128, 4, false)
  NNCV_C3(256, 1, false)
  NNCV_C3(256, 2, false)
#undef NNCV_C3
  return cudaErrorInvalidConfiguration;
}

}  // namespace nncv_b200
