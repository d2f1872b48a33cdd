// TMA-fed persistent implicit-GEMM convolution / GEMM for sm_100a (tcgen05 + TMEM).
//
// Covers the convolutions whose taps cannot share one halo tile -- 1x1 and 3x3 with stride 2
// (tests/Nets/Res18.mlir: the convs on %padded_107/111/115 and the 1x1 downsample convs on
// %cst_62/38/14), ResNet-50's 1x1 convs -- and plain linalg.matmul / the FC layer
// (Res18.mlir:617-628, tests/MatMulOptimization/MatMulNv.mlir:6-9).  nncv lowers strided convs
// with an extra {1,1} tile to near-scalar loops (ModernTile.cpp:201-209) and aims matmul at
// 16x16x16 wmma tiles (ModernTileGpu.cpp:427-525, PrepareModernVecGpu.cpp:43-48).
//
// GEMM view: D[pixels, Kout] = A[pixels, R*S*C] * W[Kout, R*S*C]^T.  The M tile is a block of
// tn images x th rows x tw columns of OUTPUT pixels (tn*th*tw = 128).  For every (tap, 64-channel
// block) ONE 4-D tiled TMA copy with element strides (1, stride, stride, 1) fetches exactly the
// input pixels that tile needs -- x = stride*ox + s - pad, y = stride*oy + r - pad -- as 128 rows
// of 128 bytes in the swizzled K-major layout tcgen05.mma reads; out-of-range pixels (padding,
// ragged tiles) arrive as zeros.  No thread touches the A operand.  A plain [M,K] matrix is the
// degenerate case tw = 128, th = tn = 1.
// Weights are the packed [Kout tile][k-block] images of launch_pack_weights(): resident in shared
// memory for the whole kernel when they fit, otherwise streamed with the A stage.
// Roles: warp 0 TMA producer, warp 1 MMA issuer (accumulator double-buffered in TMEM), warps 2-9
// epilogue (epilogue.cuh: residual rows in by TMA, scale/shift, ReLU, 128-byte rows in a staging buffer of
// the warp, 4-D TMA store, which clips ragged tiles and keeps the pads of shared-pad tensors untouched).
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

constexpr int kThreads = 64 + epi::kThreads;
constexpr int kABytes = 128 * 128;
constexpr int kMaxStages = 8;
constexpr size_t kBarBytes = 8 * (2 * kMaxStages + 2 + 2 + 1 + epi::kWarps * epi::kMaxBufs) + 16;

struct TcParams {
  const uint8_t* wpack;
  const float* scale;
  const float* shift;
  const uint8_t* wpack2;     // DUAL: packed 1x1 weights of the fused downsample branch
  const float* scale2;
  const float* shift2;
  int* error_flag;
  int Kout, CB, taps, S, stride, pad;
  int in_off;                // layout offset of the input (0 dense, 1 shared-pad)
  int out_off;
  int OH, OW, NB;            // logical output extent
  int out_pitch, out_rows;   // output layout: slots per row, rows per image
  int tw, th, tn;            // M tile shape
  int tiles_x, tiles_y, tiles_n, n_tiles, m_items;
  epi::FastDiv div_tx, div_ty, div_nt;   // by tiles_x, tiles_y, n_tiles
  int tail_start;   // matmul on pairs: items from here on are cut into halves by columns, one half a pair; -1: none
  int splits;       // matmul: CTAs of a cluster that share a tile's channel blocks (then every cluster has one tile); 1: no clusters
  void* out;        // the result, where it does not leave through tm_out
  int stages;                // A (+ streamed weight) ring depth
  int relu, bf16, out_f32;
  int w_ready;    // the packed weights were complete before this launch (not written by earlier work of its stream)
  int residual;   // tm_res holds a tensor of the output's layout and type, added before the activation
  int epi_bufs;   // staging buffers per epilogue warp (1 .. epi::kMaxBufs)
  int act;   // 0, or kActHardSwish / kActSilu applied after the residual add (16-bit outputs)
};

// DUAL: a ResNet block that changes resolution applies a 3x3 stride-2 pad-1 convolution and a 1x1
// stride-2 convolution to the SAME tensor (tests/Nets/Res18.mlir: the convs on %padded_107 and on
// %cst_62 both read the output of layer 1, and likewise for layers 3 and 4).  The 1x1 conv reads
// exactly the pixels of the 3x3 conv's centre tap, so it rides along as a tenth "tap" per channel
// block: the same A tile coordinates, its own weight tile, and a second accumulator beside the
// first.  Both results leave through the same epilogue (the second one with its own scale/shift,
// no ReLU, no residual) into a second output tensor.
// PAIR: two CTAs of a cluster work as one (tcgen05.mma.cta_group::2, M = 256): each loads the A tile
// of its own 128 output pixels and HALF of every weight tile (BN/2 rows), one lane of the leader
// issues MMAs that read both CTAs' shared memory, each CTA drains its own accumulator rows.  The
// streamed kernel is bound by the L2->SM path (one A tile and one weight tile per 128 x BN x 64
// block); halving the weight bytes per CTA is the point.  Barrier protocol as in conv3x3_pair.cu.
// BROW: the B operand is a plain row-major [K, N] matrix (linalg.matmul's right-hand side as it lies in
// memory): 64 x 64 boxes of it land by TMA as MN-major 128-byte-swizzled tiles -- k rows of 128 bytes,
// 8-row groups 1024 bytes apart, one box per 64 columns 8192 bytes apart -- and the instruction
// descriptor marks B as MN-major, so nothing is repacked; rows and columns past the matrix read as zero.  On CTA pairs each
// CTA brings half of the columns: 32 KB instead of 48 per 128 x 256 x 64 products.
template <int BN, bool RESIDENT, bool DUAL, bool PAIR, bool BROW>
__global__ void __launch_bounds__(kThreads, 1)
tconv_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out,
             const __grid_constant__ CUtensorMap tm_out2, const __grid_constant__ CUtensorMap tm_b,
             const __grid_constant__ CUtensorMap tm_b2, const __grid_constant__ CUtensorMap tm_res, const TcParams p) {
  static_assert(!PAIR || !RESIDENT, "the pair kernel streams its weights");
  static_assert(!BROW || (!RESIDENT && !DUAL), "a row-major B is streamed");
  constexpr int WTILE = (PAIR ? BN / 2 : BN) * 128;   // this CTA's part of a weight tile
  constexpr int ACC_W = DUAL ? 2 * BN : BN;   // columns of one accumulator buffer
  constexpr int ACC_COLS = 2 * ACC_W;         // two accumulator buffers
  const int taps_x = p.taps + (DUAL ? 1 : 0); // taps per channel block in the pipeline

  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ __align__(16) float4 s_cols[epi::kWarps][32];   // scale / shift of the slab each epilogue warp works on
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const int KB = p.taps * p.CB;
  const int stage_bytes = RESIDENT ? kABytes : kABytes + WTILE;
  const uint32_t sRing = base;
  const uint32_t sW = sRing + (uint32_t)p.stages * stage_bytes;       // resident weights
  const uint32_t sStage = sW + (RESIDENT ? (uint32_t)(KB + (DUAL ? p.CB : 0)) * WTILE : 0u);   // resident: main tiles, then the branch's
  const uint32_t bars = sStage + (uint32_t)(epi::kWarps * p.epi_bufs) * epi::kBufBytes;
  const uint32_t full = bars, empty = bars + 8 * kMaxStages;
  const uint32_t acc_full = empty + 8 * kMaxStages, acc_empty = acc_full + 16;
  const uint32_t w_full = acc_empty + 16;
  const uint32_t res_full = w_full + 8;
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

  const int warp = ptx::warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;   // 0 = leader
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kMaxStages; ++i) {
      ptx::mbar_init(full + 8 * i, 1);   // pair: only the leader's are used, for both CTAs' bytes
      ptx::mbar_init(empty + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(acc_full + 8 * i, 1);
      ptx::mbar_init(acc_empty + 8 * i, PAIR ? 2 * epi::kWarps : epi::kWarps);   // one arrival per epilogue warp (of both CTAs)
    }
    ptx::mbar_init(w_full, 1);
    for (int i = 0; i < epi::kWarps * epi::kMaxBufs; ++i) ptx::mbar_init(res_full + 8 * i, 1);
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_in);
    ptx::prefetch_tensormap(&tm_out);
    if (DUAL) ptx::prefetch_tensormap(&tm_out2);
    if (BROW || PAIR) ptx::prefetch_tensormap(&tm_b);
    if (PAIR && DUAL) ptx::prefetch_tensormap(&tm_b2);
    if (p.residual) ptx::prefetch_tensormap(&tm_res);
  }
  if (warp == 1) {
    if (PAIR) {
      ptx::tmem_alloc_pair(tmem_slot, ACC_COLS);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_slot, ACC_COLS);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR) ptx::cluster_sync_all();   // both CTAs' barriers exist before anyone arrives remotely
  ptx::tc_fence_after();
  const uint32_t tmem_base = (uint32_t)ptx::warp_uniform(*reinterpret_cast<volatile int*>(smem_raw + (tmem_slot - raw)));
  volatile int* abort_flag = &s_abort;

  // Resident weights pin a CTA to one Kout tile (blockIdx.y); otherwise the CTA strides over
  // (pixel tile, Kout tile) pairs with the Kout tiles of a pixel tile adjacent.
  // Pair: a work item is two consecutive pixel tiles (one per CTA) times one Kout tile; a tile past
  // the end reads zeros and stores nothing.
  const int m_units = PAIR ? (p.m_items + 1) / 2 : p.m_items;
  const int total_items = RESIDENT ? m_units : m_units * p.n_tiles;
  constexpr bool CAN_SPLIT = BROW && !PAIR;
  const int S = CAN_SPLIT ? p.splits : 1, krank = CAN_SPLIT && S > 1 ? (int)ptx::cluster_ctarank() : 0;
  const int cb_lo = CAN_SPLIT ? p.CB * krank / S : 0, cb_hi = CAN_SPLIT ? p.CB * (krank + 1) / S : p.CB;
  const int per_worker = PAIR ? 2 : S;
  const int worker = (int)blockIdx.x / per_worker, workers = (int)gridDim.x / per_worker;
  // The last round of a matmul on pairs, when at most half of the pairs would have an item: every item is cut in two by
  // columns and the halves run side by side (4096^3, 256 items on 74 pairs: 138 -> 128 us of kernel time when it
  // was made; with whole-warp copies the kernel takes 102).
  const int full_rounds = PAIR && BROW && p.tail_start >= 0 ? p.tail_start / workers : 0x7fffffff;
  auto item_of = [&](int i, int& n0, int& oy0, int& ox0, int& n_tile) {
    int w = worker + i * workers;
    if (PAIR && BROW && i >= full_rounds) {
      if (i > full_rounds) return false;
      w = p.tail_start + (worker >> 1);
    }
    if (w >= total_items) return false;
    int m_item;
    if (RESIDENT) {
      m_item = w;
      n_tile = (int)blockIdx.y;
    } else {
      m_item = (int)epi::div_by((uint32_t)w, p.div_nt);
      n_tile = w - m_item * p.n_tiles;
    }
    if (PAIR) m_item = 2 * m_item + (int)rank;
    const int t2 = (int)epi::div_by((uint32_t)m_item, p.div_tx);
    const int tx = m_item - t2 * p.tiles_x;
    const int t3 = (int)epi::div_by((uint32_t)t2, p.div_ty);
    const int ty = t2 - t3 * p.tiles_y;
    n0 = t3 * p.tn;
    oy0 = ty * p.th;
    ox0 = tx * p.tw;
    return true;
  };

  auto halved = [&](int i) { return PAIR && BROW && i >= full_rounds; };
  auto first_col = [&](int i, int n_tile) { return n_tile * BN + (halved(i) ? (worker & 1) * (BN / 2) : 0); };
  // Packed weights are the plan's own and nobody writes them once they are made, so their copies start before the previous
  // kernel of the stream has finished: everything the ring holds.  At small batches, where a kernel leaves most SMs idle,
  // that hides the whole weight fetch behind the previous layer.
  const uint32_t full_lead = PAIR ? ptx::map_to_cta(full, 0) : full;
  // the bytes of a stage, of both CTAs, are counted on the leader's barrier
  auto expect_stage = [&](uint32_t st, uint32_t issue, bool half = false) {
    if (!PAIR) ptx::mbar_arrive_expect_tx(full + 8 * st, (uint32_t)stage_bytes, issue);
    else if (rank == 0) ptx::mbar_arrive_expect_tx(full + 8 * st, 2u * (uint32_t)(half ? kABytes + WTILE / 2 : stage_bytes), issue);
  };
  auto load_weights = [&](int n_tile, int cb, int tap, uint32_t st, uint32_t issue) {
    const uint32_t dst = sRing + st * stage_bytes + kABytes;
    const bool second = DUAL && tap == p.taps;
    if (PAIR) {   // the weights are packed for N tile BN/2; this CTA takes tile 2 * n_tile + rank
      const int wt = 2 * n_tile + (int)rank;
      if (second) ptx::tma_load_2d_pair(dst, &tm_b2, 0, (wt * p.CB + cb) * (BN / 2), full_lead + 8 * st, issue);
      else ptx::tma_load_2d_pair(dst, &tm_b, 0, (wt * KB + tap * p.CB + cb) * (BN / 2), full_lead + 8 * st, issue);
    } else {
      ptx::bulk_g2s(dst, second ? p.wpack2 + ((size_t)n_tile * p.CB + cb) * WTILE : p.wpack + ((size_t)n_tile * KB + (size_t)tap * p.CB + cb) * WTILE,
                    WTILE, full + 8 * st, issue);
    }
  };
  uint32_t early = 0;   // ring stages whose weights are on their way
  auto load_resident = [&]() {
    const uint8_t* src = p.wpack + (size_t)blockIdx.y * KB * WTILE;
    ptx::mbar_arrive_expect_tx(w_full, (uint32_t)(KB + (DUAL ? p.CB : 0)) * WTILE);
    for (int i = 0; i < KB; ++i) ptx::bulk_g2s(sW + (uint32_t)i * WTILE, src + (size_t)i * WTILE, WTILE, w_full);
    if (DUAL) {
      const uint8_t* src2 = p.wpack2 + (size_t)blockIdx.y * p.CB * WTILE;
      for (int i = 0; i < p.CB; ++i) ptx::bulk_g2s(sW + (uint32_t)(KB + i) * WTILE, src2 + (size_t)i * WTILE, WTILE, w_full);
    }
  };
  if (warp == 0 && !BROW && p.w_ready) {
    if (RESIDENT) {
      if (lane == 0) load_resident();
      __syncwarp();
    } else {
      const uint32_t issue = ptx::elect_one();
      for (int i = 0; early < (uint32_t)p.stages; ++i) {
        int n0, oy0, ox0, n_tile;
        if (!item_of(i, n0, oy0, ox0, n_tile)) break;
        for (int cb = 0; cb < p.CB && early < (uint32_t)p.stages; ++cb)
          for (int tap = 0; tap < taps_x && early < (uint32_t)p.stages; ++tap, ++early) {
            expect_stage(early, issue);
            load_weights(n_tile, cb, tap, early, issue);
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
      if (RESIDENT && !p.w_ready && lane == 0) load_resident();
      __syncwarp();
      const uint32_t issue = ptx::elect_one();
      uint32_t cnt = 0, st = 0, ring = 1;   // stages begun; the next one and the parity of its round
      uint32_t seen = 1;                    // nothing has used the ring yet
      bool okw = true;
      for (int i = 0; okw; ++i) {
        int n0, oy0, ox0, n_tile;
        if (!item_of(i, n0, oy0, ox0, n_tile)) break;
        const int xb = p.stride * ox0 - p.pad + p.in_off, yb = p.stride * oy0 - p.pad + p.in_off;
        const int centre_r = DUAL ? (p.taps / 2) / p.S : 0, centre_s = DUAL ? p.taps / 2 - centre_r * p.S : 0;
        // channel block outermost, taps innermost: the same accumulation order as the shifted-view
        // 3x3 kernel, so both kernels give bit-identical sums
        for (int cb = cb_lo; cb < cb_hi && okw; ++cb) {
          int r = 0, s = 0;
          for (int tap = 0; tap < taps_x; ++tap, ++cnt) {
            if (DUAL && tap == p.taps) { r = centre_r; s = centre_s; }   // the extra tap re-reads the centre tap's pixels
            const bool begun = cnt < early;   // this stage's first use: weights already issued
            if (!ptx::warp_all(seen)) {
              if (!ptx::warp_wait(empty + 8 * st, ring, abort_flag)) { okw = false; break; }
            }
            if (!begun) expect_stage(st, issue, halved(i));
            const uint32_t dst = sRing + st * stage_bytes;
            if (PAIR) ptx::tma_load_4d_pair(dst, &tm_in, cb * 64, xb + s, yb + r, n0, full_lead + 8 * st, issue);
            else ptx::tma_load_4d(dst, &tm_in, cb * 64, xb + s, yb + r, n0, full + 8 * st, issue);
            if (BROW) {
#pragma unroll
              for (int j = 0; j < WTILE / 8192; ++j) {
                if (PAIR) {
                  const int mine = halved(i) ? BN / 4 : BN / 2;   // columns of this CTA
                  if (j * 64 < mine)
                    ptx::tma_load_2d_pair(dst + kABytes + (uint32_t)j * 8192u, &tm_b, first_col(i, n_tile) + (int)rank * mine + j * 64, cb * 64,
                                          full_lead + 8 * st, issue);
                } else {
                  ptx::tma_load_2d(dst + kABytes + (uint32_t)j * 8192u, &tm_b, n_tile * BN + j * 64, cb * 64, full + 8 * st, issue);
                }
              }
            } else if (!RESIDENT && !begun) {
              load_weights(n_tile, cb, tap, st, issue);
            }
            if (++s == p.S) { s = 0; ++r; }
            const bool wrap = st + 1 == (uint32_t)p.stages;
            st = wrap ? 0u : st + 1;
            ring ^= wrap ? 1u : 0u;
            seen = ptx::mbar_peek(empty + 8 * st, ring);
          }
        }
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    }
  } else if (warp == 1) {
    if (!PAIR || rank == 0)
    // ------------------------------------------------------------------ MMA issuer ------
    {
      const uint32_t issue = ptx::elect_one();
      const uint32_t idesc = ptx::umma_idesc(PAIR ? 256 : 128, BN, p.bf16 ? 1 : 0) | (BROW ? (1u << 16) : 0u);   // bit 16: B is MN-major
      bool okw = true;
      if (RESIDENT) okw = ptx::warp_wait(w_full, 0, abort_flag);
      uint32_t st = 0, ring = 0, acc_cnt = 0;   // stage, parity of the ring's round
      uint32_t seen = okw ? ptx::mbar_peek(full, 0) : 0u;
      for (int i = 0; okw; ++i) {
        int n0, oy0, ox0, n_tile;
        if (!item_of(i, n0, oy0, ox0, n_tile)) break;
        const uint32_t ab = acc_cnt & 1u;
        if (!ptx::warp_wait(acc_empty + 8 * ab, ((acc_cnt >> 1) & 1u) ^ 1u, abort_flag)) { okw = false; break; }
        ptx::tc_fence_after();
        const uint32_t d = tmem_base + ab * ACC_W;
        const uint32_t id = halved(i) ? idesc - ((uint32_t)(BN / 2 / 8) << 17) : idesc;   // N field
        for (int cb = cb_lo; cb < cb_hi && okw; ++cb)
          for (int tap = 0; tap < taps_x; ++tap) {   // producer order: cb outer, tap inner
            const bool second = DUAL && tap == p.taps;
            if (!ptx::warp_all(seen) && !ptx::warp_wait(full + 8 * st, ring, abort_flag)) { okw = false; break; }
            ptx::tc_fence_after();
            const bool wrap = st + 1 == (uint32_t)p.stages;
            const uint32_t st_next = wrap ? 0u : st + 1, ring_next = ring ^ (wrap ? 1u : 0u);
            seen = ptx::mbar_peek(full + 8 * st_next, ring_next);
            const uint32_t a_addr = sRing + st * stage_bytes;
            const uint32_t a_lo = ptx::smem_desc_k128_lo(a_addr);
            // MN-major B: leading-dimension offset 8192 bytes (next 64 columns), one k step of 16 = two 8-row groups
            const uint32_t b_lo = BROW ? ((((a_addr + kABytes) & 0x3FFFFu) >> 4) | ((8192u >> 4) << 16))
                                       : ptx::smem_desc_k128_lo(
                RESIDENT ? sW + (uint32_t)(second ? KB + cb : tap * p.CB + cb) * WTILE : a_addr + kABytes);
            constexpr uint32_t kBStep = BROW ? (2048u >> 4) : 2u;
            const uint32_t first = second ? (uint32_t)cb : (uint32_t)((cb - cb_lo) | tap);
#pragma unroll
            for (uint32_t k4 = 0; k4 < 4; ++k4) {
              const uint64_t da = ptx::desc_from_halves(a_lo + k4 * 2, ptx::kSmemDescK128Hi);
              const uint64_t db = ptx::desc_from_halves(b_lo + k4 * kBStep, ptx::kSmemDescK128Hi);
              if (PAIR) ptx::umma_f16_pair(second ? d + BN : d, da, db, id, first | k4, issue);
              else ptx::umma_f16(second ? d + BN : d, da, db, id, first | k4, issue);
            }
            if (PAIR) ptx::tc_commit_pair(empty + 8 * st, issue);
            else ptx::tc_commit(empty + 8 * st, issue);
            st = st_next;
            ring = ring_next;
          }
        if (!okw) break;
        if (PAIR) ptx::tc_commit_pair(acc_full + 8 * ab, issue);
        else ptx::tc_commit(acc_full + 8 * ab, issue);
        ++acc_cnt;
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitMma);
    }
  } else {
    // ------------------------------------------------------------------ epilogue --------
    // Eight independent warps (epilogue.cuh).  Slabs of an item are numbered output-major, then by column; warp group
    // `half` takes every second slab of the running count, so both groups drain one accumulator together when it has
    // several slabs and alternate between the accumulators when it has one.
    const int ew = warp - 2, quad = warp & 3, half = ew >> 2;
    const uint32_t sw = (uint32_t)(lane & 7);
    const int nb = p.epi_bufs;
    const uint32_t my_stage = sStage + (uint32_t)(ew * nb) * epi::kBufBytes;
    const uint32_t my_res = res_full + (uint32_t)(ew * epi::kMaxBufs) * 8u;
    const uint32_t tab = ptx::smem_u32(&s_cols[ew][0]);
    const int slab_cols = p.out_f32 ? 32 : 64;      // 128-byte rows either way
    // slabs of an output and of an item, as powers of two
    const int slabs_log = (BN == 64 ? 0 : (BN == 128 ? 1 : 2)) + (p.out_f32 ? 1 : 0);
    const int spi_log = slabs_log + (DUAL ? 1 : 0);
    const int spi = 1 << spi_log, slabs = 1 << slabs_log;
    const int mode = epi::mode_of(p.bf16 != 0, p.residual != 0, p.relu != 0, p.act), mode2 = epi::mode_of(p.bf16 != 0, false, false, 0);
    // the 32 pixels of this warp's rows form a box inside the tile
    const int qx = (quad * 32) % p.tw, qy = (quad * 32 / p.tw) % p.th, qn = quad * 32 / (p.tw * p.th);
    const bool has_res = p.residual != 0;
    // where a slab lies; the item is looked up only when it changes
    struct Pos { int i, n0, oy0, ox0, n_tile; bool ok; };
    auto seek = [&](Pos& q, int i) {
      if (q.i != i) {
        q.i = i;
        q.ok = item_of(i, q.n0, q.oy0, q.ox0, q.n_tile);
      }
      return q.ok;
    };
    auto live_at = [&](const Pos& q, int ncol) {
      return ncol < p.Kout && q.ox0 + qx < p.OW && q.oy0 + qy < p.OH && q.n0 + qn < p.NB;
    };
    Pos cur{-1, 0, 0, 0, 0, false}, ahead{-1, 0, 0, 0, 0, false};
    uint32_t phase = 0, inflight = 0;   // per staging buffer: parity of its next residual, one on its way
    int ahead_j = half, ahead_b = 0;
    // residual rows of the next slab in line -> its staging buffer
    auto fetch_res = [&]() {
      const int i = ahead_j >> spi_log, sl = ahead_j & (spi - 1);
      if (seek(ahead, i)) {
        const int ncol = first_col(i, ahead.n_tile) + sl * slab_cols;
        if (live_at(ahead, ncol)) {
          inflight |= 1u << ahead_b;
          if (lane == 0) {
            ptx::mbar_arrive_expect_tx(my_res + 8 * ahead_b, epi::kBufBytes);
            ptx::tma_load_4d(my_stage + (uint32_t)ahead_b * epi::kBufBytes, &tm_res, ncol, ahead.ox0 + qx + p.out_off,
                             ahead.oy0 + qy + p.out_off, ahead.n0 + qn, my_res + 8 * ahead_b);
          }
        }
      }
      ahead_j += 2;
      if (++ahead_b == nb) ahead_b = 0;
    };
    auto cols_of = [&](int i, int rem, Pos& q) {
      if (!seek(q, i)) return epi::ColParams{1.0f, 1.0f, 0.0f, 0.0f};
      const int oi = DUAL ? rem >> slabs_log : 0, sl = DUAL ? rem & (slabs - 1) : rem;
      return epi::fetch_cols(oi ? p.scale2 : p.scale, oi ? p.shift2 : p.shift, first_col(i, q.n_tile) + sl * slab_cols, p.Kout, lane);
    };
    Pos colpos{-1, 0, 0, 0, 0, false};
    int j = half, b = 0;   // running slab count of this warp (+= 2), staging buffer
    epi::ColParams cols = cols_of(j >> spi_log, j & (spi - 1), colpos);
    if (has_res)
      for (int k = 0; k + 1 < nb; ++k) fetch_res();
    bool okw = true;
    for (int i = 0; okw; ++i) {
      if (!seek(cur, i)) break;
      const uint32_t ab = (uint32_t)i & 1u;
      okw = ptx::mbar_wait_abortable(acc_full + 8 * ab, ((uint32_t)i >> 1) & 1u, abort_flag);
      okw = __all_sync(0xffffffffu, okw);
      if (!okw) break;
      ptx::tc_fence_after();
      if (CAN_SPLIT && S > 1) {   // partial sums into the ring, which nothing reads or fills any more: the tile's MMAs are complete
        const int row = quad * 32 + lane;
#pragma unroll
        for (int c = 0; c < BN / 64; ++c) {
          const int col = half * (BN / 2) + c * 32;
          uint32_t acc[32];
          ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)col, acc);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 8; ++e)
            epi::sts128(sRing + (uint32_t)row * (BN * 4) + (((uint32_t)(col / 4 + e) ^ sw) << 4), acc[4 * e], acc[4 * e + 1], acc[4 * e + 2], acc[4 * e + 3]);
        }
        break;
      }
      auto hand_back = [&]() {   // this warp has read its part of the accumulator
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (!PAIR || rank == 0) ptx::mbar_arrive(acc_empty + 8 * ab);
          else ptx::mbar_arrive_remote_cta(ptx::map_to_cta(acc_empty, 0) + 8 * ab);
        }
      };
      const int end_j = (i + 1) << spi_log;
      if (j >= end_j) hand_back();   // no slab of this item is this warp's
      for (; j < end_j; j += 2) {
        const int rem = j & (spi - 1);
        const int oi = DUAL ? rem >> slabs_log : 0, sl = DUAL ? rem & (slabs - 1) : rem;
        const int ncol = first_col(i, cur.n_tile) + sl * slab_cols;
        const bool live = live_at(cur, ncol) && !(halved(i) && sl * slab_cols >= BN / 2);
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + ab * ACC_W + (uint32_t)(oi * BN + sl * slab_cols);
        uint32_t acc[64];
        if (p.out_f32) epi::load_slab_f32(taddr, acc);
        else epi::load_slab(taddr, acc);
        epi::put_cols(tab, cols, lane);
        if (has_res) {
          // the buffer the next residual goes to was stored from one slab ago
          if (lane == 0) ptx::bulk_wait_read<0>();
          __syncwarp();
          fetch_res();
        } else {
          if (lane == 0) {
            if (nb == 1) ptx::bulk_wait_read<0>();
            else ptx::bulk_wait_read<1>();
          }
        }
        ptx::tmem_ld_wait();
        __syncwarp();
        if (j + 2 >= end_j) hand_back();
        cols = cols_of((j + 2) >> spi_log, (j + 2) & (spi - 1), colpos);
        if (live) {
          const uint32_t buf = my_stage + (uint32_t)b * epi::kBufBytes;
          if (has_res) {
            okw = ptx::mbar_wait_abortable(my_res + 8 * b, (phase >> b) & 1u, abort_flag);
            okw = __all_sync(0xffffffffu, okw);
            if (!okw) break;
            phase ^= 1u << b;
            inflight &= ~(1u << b);
          }
          if (p.out_f32) {
            if (p.relu) epi::slab32_f32<true>(acc, tab, buf, lane);
            else epi::slab32_f32<false>(acc, tab, buf, lane);
          } else {
            epi::slab64_by_mode<DUAL ? 1 : 3>(oi ? mode2 : mode, acc, tab, buf, lane);
          }
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_4d((DUAL && oi) ? &tm_out2 : &tm_out, ncol, cur.ox0 + qx + p.out_off, cur.oy0 + qy + p.out_off, cur.n0 + qn, buf);
            ptx::bulk_commit();
          }
        }
        __syncwarp();
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
  if (PAIR) ptx::cluster_sync_all();   // the peer's shared memory and barriers stay valid until both are done
  if (CAN_SPLIT && S > 1) {
    // every CTA finishes its share of the rows from all partial sums, in rank order: the result does not depend on timing
    ptx::cluster_sync_all();
    int n0, oy0, ox0, n_tile;
    item_of(0, n0, oy0, ox0, n_tile);
    const int rows = 128 / S;
    for (int idx = threadIdx.x; idx < rows * (BN / 4); idx += kThreads) {
      const int r = krank * rows + idx / (BN / 4), c4 = idx % (BN / 4), n = n_tile * BN + c4 * 4;
      if (n >= p.Kout || ox0 + r >= p.OW || s_abort) continue;
      const uint32_t at = sRing + (uint32_t)r * (BN * 4) + (((uint32_t)c4 ^ (uint32_t)(r & 7)) << 4);
      float4 part[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < S) part[q] = ptx::ld_cluster_f4(ptx::map_to_cta(at, (uint32_t)q));
      float v[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < S) { v[0] += part[q].x; v[1] += part[q].y; v[2] += part[q].z; v[3] += part[q].w; }
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = fmaf(v[e], p.scale ? __ldg(p.scale + n + e) : 1.0f, p.shift ? __ldg(p.shift + n + e) : 0.0f);
      const size_t o = (size_t)(ox0 + r) * p.Kout + n;
      if (p.out_f32) {
        if (p.relu)
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = !(v[e] <= 0.0f) ? v[e] : 0.0f;
        *reinterpret_cast<float4*>(static_cast<float*>(p.out) + o) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        *reinterpret_cast<uint2*>(static_cast<unsigned short*>(p.out) + o) =
            make_uint2(epi::pack16(v[0], v[1], p.bf16 != 0, p.relu != 0), epi::pack16(v[2], v[3], p.bf16 != 0, p.relu != 0));
      }
    }
    __syncwarp();
    ptx::cluster_sync_all();   // the peers' reads of this CTA's partial sums are over
  }
  if (warp == 1) {
    __syncwarp();
    if (PAIR) ptx::tmem_dealloc_pair(tmem_base, ACC_COLS);
    else ptx::tmem_dealloc(tmem_base, ACC_COLS);
  }
}

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

// 4-D map over an activation [NB][rows][pitch][C] (C innermost), box (box_c, bx, by, bn) with
// traversal strides (1, sx, sy, 1); 128-byte swizzle; out-of-range elements read as zero.
bool make_map4(CUtensorMap* m, const void* ptr, CUtensorMapDataType dt, int esz, int C, long long pitch,
               long long rows, long long NB, int box_c, int bx, int by, int bn, int sx, int sy) {
  auto enc = get_encode();
  if (!enc) return false;
  cuuint64_t gdim[4] = {(cuuint64_t)C, (cuuint64_t)pitch, (cuuint64_t)rows, (cuuint64_t)NB};
  cuuint64_t gstr[3] = {(cuuint64_t)C * esz, (cuuint64_t)pitch * C * esz, (cuuint64_t)rows * pitch * C * esz};
  cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bn};
  cuuint32_t estr[4] = {1, (cuuint32_t)sx, (cuuint32_t)sy, 1};
  return enc(m, dt, 4, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

constexpr int kSplitBlocks = 4;   // matmul: fewest blocks of 64 of a CTA that shares a tile's depth
constexpr size_t kSmemLimit = 222 * 1024;   // dynamic part: the kernel also holds 4 KB of static shared memory (scale / shift of the slabs in work)

// 2-D map over a row-major [K, N] 16-bit matrix, box 64 columns x 64 rows, 128-byte swizzle, zero fill.
bool make_map_b(CUtensorMap* m, const void* ptr, CUtensorMapDataType dt, long long K, long long N) {
  auto enc = get_encode();
  if (!enc) return false;
  cuuint64_t gdim[2] = {(cuuint64_t)N, (cuuint64_t)K};
  cuuint64_t gstr[1] = {(cuuint64_t)N * 2};
  cuuint32_t box[2] = {64, 64};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, dt, 2, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2-D map over packed weights: `tiles` tiles of `rows` x 64 values that already lie in the order shared memory wants.
bool make_map_w(CUtensorMap* m, const void* ptr, CUtensorMapDataType dt, int rows, long long tiles) {
  auto enc = get_encode();
  if (!enc) return false;
  cuuint64_t gdim[2] = {64, (cuuint64_t)(tiles * rows)};
  cuuint64_t gstr[1] = {128};
  cuuint32_t box[2] = {64, (cuuint32_t)rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, dt, 2, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool RESIDENT, bool DUAL = false, bool PAIR = false, bool BROW = false>
cudaError_t launch_cfg(const TconvArgs& a, TcParams p, cudaStream_t stream) {
  const size_t wtile = (size_t)(PAIR ? BN / 2 : BN) * 128;
  const int KB = p.taps * p.CB;
  const size_t stage = RESIDENT ? kABytes : kABytes + wtile;
  const size_t wres = RESIDENT ? (size_t)(KB + (DUAL ? p.CB : 0)) * wtile : 0;
  // a long reduction (1024 and more) is better served by five stages than by a second staging buffer: one epilogue for many blocks
  p.epi_bufs = epi::pick_bufs(p.residual != 0, kSmemLimit - 1024 - kBarBytes, wres + (PAIR && BROW && KB >= 16 ? 5 : 3) * stage, wres + 2 * stage);
  const size_t fixed = 1024 + (size_t)(epi::kWarps * p.epi_bufs) * epi::kBufBytes + kBarBytes;
  if (fixed + wres + 2 * stage > kSmemLimit) return cudaErrorInvalidConfiguration;
  size_t st = (kSmemLimit - fixed - wres) / stage;
  if (st > kMaxStages) st = kMaxStages;
  p.stages = (int)st;
  const size_t smem = fixed + wres + st * stage;

  const Layout il = a.in_l, ol = a.out_l;
  const auto dt = p.bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm_in, tm_out;
  if (!make_map4(&tm_in, a.in, dt, 2, a.C, il.pitch, il.img_rows, a.N, 64, p.tw * p.stride, p.th * p.stride, p.tn,
                 p.stride, p.stride))
    return cudaErrorInvalidValue;
  const bool f32 = p.out_f32 != 0;
  // an epilogue warp stores its own 32 pixels: a box of the tile (all three extents are powers of two)
  const int qw = p.tw < 32 ? p.tw : 32, qh = p.th < 32 / qw ? p.th : 32 / qw, qn = 32 / (qw * qh);
  if (!make_map4(&tm_out, a.out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : dt, f32 ? 4 : 2, a.Kout, ol.pitch, ol.img_rows,
                 a.N, f32 ? 32 : 64, qw, qh, qn, 1, 1))
    return cudaErrorInvalidValue;
  CUtensorMap tm_out2 = tm_out;
  if (DUAL && !make_map4(&tm_out2, a.out2, dt, 2, a.Kout, ol.pitch, ol.img_rows, a.N, 64, qw, qh, qn, 1, 1))
    return cudaErrorInvalidValue;
  CUtensorMap tm_res = tm_out;
  if (p.residual && !make_map4(&tm_res, a.residual, dt, 2, a.Kout, ol.pitch, ol.img_rows, a.N, 64, qw, qh, qn, 1, 1))
    return cudaErrorInvalidValue;
  CUtensorMap tm_b = tm_out, tm_b2 = tm_out;
  if (PAIR && !BROW && (!make_map_w(&tm_b, p.wpack, dt, BN / 2, (long long)p.n_tiles * 2 * KB) ||
                        (DUAL && !make_map_w(&tm_b2, p.wpack2, dt, BN / 2, (long long)p.n_tiles * 2 * p.CB))))
    return cudaErrorInvalidValue;
  if (BROW && !make_map_b(&tm_b, a.b_rowmajor, dt, a.b_rows, a.Kout)) return cudaErrorInvalidValue;
  auto kern = tconv_kernel<BN, RESIDENT, DUAL, PAIR, BROW>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int sms = a.sm_count > 0 ? a.sm_count : 148;
  dim3 grid;
  if (RESIDENT) {
    int gx = sms / p.n_tiles;
    if (gx < 1) gx = 1;
    if (gx > p.m_items) gx = p.m_items;
    grid = dim3(gx, p.n_tiles);
  } else if (PAIR) {
    const long long items = (long long)((p.m_items + 1) / 2) * p.n_tiles;
    static const int fit = max_clusters(kern, 2, kThreads, kSmemLimit, sms);   // the same on every device this library runs on
    const long long pairs = fit;
    if (BROW && items > pairs) {
      const long long tail = items % pairs;   // halves only while both of every item fit in the one round
      if (tail > 0 && 2 * tail <= pairs) p.tail_start = (int)(items - tail);
    }
    grid = dim3(2 * (unsigned)(items < pairs ? items : pairs), 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, tm_in, tm_out, tm_out2, tm_b, tm_b2, tm_res, p);
  } else {
    const long long items = (long long)p.m_items * p.n_tiles;
    if (BROW) {
      // Fewer tiles than SMs: clusters split the depth of a tile, as far as all of them run at once and each CTA keeps
      // kSplitBlocks blocks of 64.
      static const ClusterFit fit = cluster_fit(kern, kThreads, kSmemLimit, sms);
      for (int s = 2; s <= 8; s *= 2) {
        if (items > fit.of[s] || p.CB < kSplitBlocks * s || st * stage < (size_t)BN * 512) break;
        p.splits = s;
      }
      if (p.splits > 1) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(items * p.splits));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)p.splits;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, kern, tm_in, tm_out, tm_out2, tm_b, tm_b2, tm_res, p);
      }
    }
    grid = dim3((unsigned)(items < sms ? items : sms), 1);
  }
  return launch_pdl(kern, grid, dim3(kThreads), smem, stream, tm_in, tm_out, tm_out2, tm_b, tm_b2, tm_res, p);
}

}  // namespace

bool tconv_supported(int C, int Kout, DType out_dt, long long ldo) {
  // channels are read in blocks of 64 (a last block that reaches past C is zero-filled by the copy engine and
  // meets zero weights); pixel and output row pitches must be 16-byte aligned for the tensor maps
  return C % 8 == 0 && C >= 8 && ldo == Kout && (Kout * (out_dt == kF32 ? 4 : 2)) % 16 == 0;
}

// M-tile shape: tw covers the output row in as few pieces as possible.
void tconv_tile(int N, int OH, int OW, int* tw, int* th, int* tn) {
  int w = 128;
  if (OW <= 8) w = 8;
  else if (OW <= 16) w = 16;
  else if (OW <= 32) w = 32;
  else if (OW <= 64) w = 64;
  else if (OW < 112) w = 128;
  else {
    // pick the divisor-friendly width among 32/64/128 with the least ragged waste
    int best = 128, waste = (OW + 127) / 128 * 128 - OW;
    for (int c : {64, 32}) {
      const int ws = (OW + c - 1) / c * c - OW;
      if (ws < waste) { best = c; waste = ws; }
    }
    w = best;
  }
  int h = 128 / w;
  if (h > OH) {
    int hh = 1;
    while (hh * 2 <= h && hh < OH) hh *= 2;   // smallest power of two >= OH, capped at 128/w
    h = hh;
  }
  *tw = w; *th = h; *tn = 128 / (w * h);
  (void)N;
}

// A pointwise convolution between dense tensors is a matrix of N * H * W rows (a fully connected layer's tile would hold
// sixteen of its one-pixel images).
void pointwise_as_matrix(TconvArgs* t) {
  TconvArgs& a = *t;
  if (a.R == 1 && a.S == 1 && a.stride == 1 && a.pad == 0 && !a.wpack2 && a.in_l.off == 0 && a.in_l.pitch == a.W && a.in_l.img_rows == a.H &&
      a.out_l.off == 0 && a.out_l.pitch == a.W && a.out_l.img_rows == a.H && (long long)a.N * a.H * a.W < (1LL << 30)) {
    const int rows = a.N * a.H * a.W;
    a.N = 1;
    a.H = a.OH = 1;
    a.W = a.OW = rows;
    a.in_l = a.out_l = Layout{1, rows, 0};
  }
}

cudaError_t launch_tconv(const TconvArgs& args, cudaStream_t stream) {
  TconvArgs a = args;
  pointwise_as_matrix(&a);
  const bool brow = a.b_rowmajor != nullptr;
  if (brow) {   // plain GEMM with a row-major B: K and N multiples of 8 (16-byte row pitches), nothing else
    if (a.ab == kF32 || a.C % 8 != 0 || a.Kout % 8 != 0 || a.R != 1 || a.S != 1 || a.stride != 1 || a.pad != 0 || a.wpack2 ||
        a.resident || a.b_rows != a.C || (reinterpret_cast<uintptr_t>(a.b_rowmajor) & 15))
      return cudaErrorInvalidValue;
  } else if (a.ab == kF32 || !tconv_supported(a.C, a.Kout, a.out_dtype, a.Kout)) {
    return cudaErrorInvalidValue;
  }
  if ((reinterpret_cast<uintptr_t>(a.in) & 15) || (reinterpret_cast<uintptr_t>(a.out) & 15) ||
      (reinterpret_cast<uintptr_t>(a.residual) & 31) || (!brow && (reinterpret_cast<uintptr_t>(a.wpack) & 15)))
    return cudaErrorMisalignedAddress;
  TcParams p;
  p.wpack = static_cast<const uint8_t*>(a.wpack);
  p.scale = a.scale; p.shift = a.shift; p.residual = a.residual != nullptr;
  p.epi_bufs = 1;
  p.wpack2 = static_cast<const uint8_t*>(a.wpack2); p.scale2 = a.scale2; p.shift2 = a.shift2;
  p.error_flag = a.error_flag;
  p.Kout = a.Kout; p.CB = (a.C + 63) / 64; p.taps = a.R * a.S; p.S = a.S; p.stride = a.stride; p.pad = a.pad;
  p.in_off = a.in_l.off; p.out_off = a.out_l.off;
  p.OH = a.OH; p.OW = a.OW; p.NB = a.N;
  p.out_pitch = a.out_l.pitch; p.out_rows = a.out_l.img_rows;
  tconv_tile(a.N, a.OH, a.OW, &p.tw, &p.th, &p.tn);
  // a single row (a matrix) takes whole tiles: in pieces of 32 or 64, which leave less of the last one empty, most of EVERY
  // tile would lie outside (fp16 matmul 3000x2000x1504: 51.2 -> 34.8 us)
  if (a.N == 1 && a.OH == 1 && a.stride == 1) { p.tw = 128; p.th = p.tn = 1; }
  if (p.tw * a.stride > 256 || p.th * a.stride > 256) return cudaErrorInvalidConfiguration;
  p.tiles_x = (a.OW + p.tw - 1) / p.tw;
  p.tiles_y = (a.OH + p.th - 1) / p.th;
  p.tiles_n = (a.N + p.tn - 1) / p.tn;
  p.n_tiles = (a.Kout + a.bn - 1) / a.bn;
  const long long mi = (long long)p.tiles_x * p.tiles_y * p.tiles_n;
  if (mi <= 0 || mi * p.n_tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
  p.m_items = (int)mi;
  p.div_tx = epi::fast_div((uint32_t)p.tiles_x); p.div_ty = epi::fast_div((uint32_t)p.tiles_y);
  p.div_nt = epi::fast_div((uint32_t)p.n_tiles);
  p.relu = a.relu; p.bf16 = a.ab == kBF16; p.out_f32 = a.out_dtype == kF32;
  p.act = a.act;
  p.w_ready = a.weights_ready;
  p.tail_start = -1;
  p.splits = 1;
  p.out = a.out;
  p.stages = 0;
  if (p.residual && p.out_f32) return cudaErrorInvalidValue;
  if (brow) {
    if (a.pair && a.bn == 256) return launch_cfg<256, false, false, true, true>(a, p, stream);   // CTA pairs: 256 x 256 tiles
    if (!a.pair && a.bn == 64) return launch_cfg<64, false, false, false, true>(a, p, stream);
    if (!a.pair && a.bn == 128) return launch_cfg<128, false, false, false, true>(a, p, stream);
    return cudaErrorInvalidConfiguration;
  }
  if (a.pair) {     // CTA pairs: a.wpack (and a.wpack2) packed for N tile bn / 2, streamed weights, 16-bit output
    if (a.resident || p.out_f32 || (a.bn != 128 && a.bn != 256) || a.Kout % a.bn != 0) return cudaErrorInvalidValue;
    if (a.wpack2) {
      if (!a.out2 || a.bn != 128 || a.R != a.S || a.R % 2 == 0 || a.pad != a.R / 2 ||
          (reinterpret_cast<uintptr_t>(a.wpack2) & 15) || (reinterpret_cast<uintptr_t>(a.out2) & 15))
        return cudaErrorInvalidValue;
      return launch_cfg<128, false, true, true>(a, p, stream);
    }
    return a.bn == 128 ? launch_cfg<128, false, false, true>(a, p, stream) : launch_cfg<256, false, false, true>(a, p, stream);
  }
  if (a.wpack2) {   // fused 1x1 stride-s branch on the centre tap: odd square filter, pad = R/2, N tile 128 streamed
    if (!a.out2 || a.bn != 128 || p.out_f32 || a.R != a.S || a.R % 2 == 0 || a.pad != a.R / 2 ||
        a.Kout % 128 != 0 || (reinterpret_cast<uintptr_t>(a.wpack2) & 15) || (reinterpret_cast<uintptr_t>(a.out2) & 15))
      return cudaErrorInvalidValue;
    return a.resident ? launch_cfg<128, true, true>(a, p, stream) : launch_cfg<128, false, true>(a, p, stream);
  }
#define NNCV_TC(BN_, RES_) \
  if (a.bn == BN_ && (a.resident != 0) == RES_) return launch_cfg<BN_, RES_>(a, p, stream);
  NNCV_TC(64, true)
  NNCV_TC(64, false)
  NNCV_TC(128, true)
  NNCV_TC(128, false)
  NNCV_TC(256, false)
#undef NNCV_TC
  return cudaErrorInvalidConfiguration;
}

// N tile of a matmul with a row-major B: the least rounds x (blocks x time + epilogue), in us as measured with every SM at
// work: a block of 64 of a 128 x 64 tile 0.28, 128 x 128 0.32, 256 x 256 on a CTA pair 0.42; a pair's launch 2, an exchange of
// partial sums 3.  (Before, the widest tile that still filled the SMs: 2048^3 took two rounds of 128 x 128, 38.7 us,
// where one of 64 pairs takes 28.3; 2048x1024x1024 two of 128 x 64, 22.4, where one of 128 x 128 takes 16.4.)
static int matmul_pick(int M, int N, int K, int sms) {
  static const double block[3] = {0.28, 0.32, 0.42}, epilogue[3] = {0.6, 0.9, 2.0};
  const long long mi = ((long long)M + 127) / 128;
  const int CB = (K + 63) / 64;
  int best_bn = 64;
  double best = 1e30;
  for (int i = 0; i < 3; ++i) {
    const int bn = 64 << i;
    if (bn > 64 && N <= bn / 2) break;
    const bool pair = bn == 256;
    const long long items = (pair ? (mi + 1) / 2 : mi) * ((N + bn - 1) / bn), slots = pair ? sms / 2 : sms;
    int s = 1;
    while (!pair && s < 8 && items * 2 * s <= slots * 15 / 16 && CB >= kSplitBlocks * 2 * s) s *= 2;
    double rounds = (double)((items + slots - 1) / slots);
    if (pair && items > slots && items % slots != 0 && 2 * (items % slots) <= slots) rounds -= 0.3;   // a last round of halves
    const double t = rounds * ((CB + s - 1) / s * block[i] + epilogue[i]) + (pair ? 2.0 : s > 1 ? 3.0 : 0.0);
    if (t < best) { best = t; best_bn = bn; }
  }
  return best_bn;
}

bool matmul_direct(const void* A, const void* B, void* C, int M, int N, int K, DType ab, DType c, const float* bias, int relu, int sms,
                   int* error_flag, TconvArgs* out) {
  if (N % 8 != 0 || N < 64 || K < 64 || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15))
    return false;
  // 64 x 64 boxes of the row-major [K, N] matrix are MN-major operand tiles
  TconvArgs& a = *out;
  a.in = A; a.b_rowmajor = B; a.b_rows = K; a.shift = bias; a.out = C;
  a.N = 1; a.H = 1; a.W = M; a.OH = 1; a.OW = M; a.C = K; a.Kout = N;
  a.in_l = Layout{1, M, 0}; a.out_l = Layout{1, M, 0};
  a.bn = matmul_pick(M, N, K, sms); a.resident = 0; a.ab = ab; a.out_dtype = c; a.relu = relu;
  // 256 x 256 tiles on CTA pairs read each column of B from L2 half as often: 4096^3 fp16 148 -> 138 us of kernel time when
  // they were made, 8192x4096x512 38.8 -> 38.1, and 2048^3, with less than a round of pairs, no slower than 128 x 256 on single CTAs
  a.pair = a.bn == 256;
  a.sm_count = sms; a.error_flag = error_flag;
  return true;
}

// N tile and residency: keep all weights of one Kout tile in shared memory when they fit beside
// four A stages; otherwise stream them with the widest tile the grid can still fill.
void tconv_pick(long long m_items, int C, int Kout, int taps, int* bn, int* resident) {
  const size_t budget = kSmemLimit - (1024 + (size_t)epi::kWarps * epi::kBufBytes + kBarBytes) - 4 * (size_t)kABytes;
  const size_t kb = (size_t)taps * ((C + 63) / 64);
  for (int b : {128, 64}) {
    if (Kout >= b && kb * b * 128 <= budget) {
      *bn = b; *resident = 1;
      return;
    }
  }
  *resident = 0;
  int b = Kout >= 256 ? 256 : (Kout > 64 ? 128 : 64);
  while (b > 64 && m_items * ((Kout + b - 1) / b) < 148) b >>= 1;
  *bn = b;
}

}  // namespace nncv_b200
