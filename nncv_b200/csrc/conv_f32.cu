// fp32 convolutions on the tensor cores: implicit GEMM over THREE bf16 PLANES per operand.
//
// Every fp32 value x is kept as x = x1 + x2 + x3, three bf16 numbers, each the nearest to what the ones before leave; with
// 8 significand bits each and signed remainders the sum is exact (from 2^-110 on; below, the third falls short of bf16's smallest
// number and x is kept to an absolute 2^-134).  A product is then six bf16 products with fp32
// accumulation,
//     a*b ~= a1*b1 + (a1*b2 + a2*b1) + a2*b2 + (a1*b3 + a3*b1),
// and what is dropped (a2*b3, a3*b2, a3*b3) is below 2^-26 of the product: less than the rounding of ONE fp32 multiply.
// (Two tf32 parts, the other way to do this, keep 22 of the 24 bits, take as much tensor time -- three products at half
// the rate -- and 8 bytes an element instead of 6.)
// tcgen05.mma cuts its products and sums instead of rounding them, an error of one sign that the layers of a network add
// up: with normal operands every step of 16 channels takes 0.2 * 2^-24 off the sum it leaves.  So the large products a1*b1
// stay in TMEM for ONE step only: the epilogue warps add each step, rounded, to a sum in registers.  (With the four steps of a
// block of 64 channels in one accumulator the logits of ResNet-18 and ResNet-50 were 5.6e-7 and 1.2e-6 off the result in 64 bits,
// nearly all of it this bias; the CUDA-core kernel's are 2.2e-7 to 3.3e-7 and 3.5e-7 off, now these 1.4e-7 to 1.9e-7 and 1.9e-7.
// Networks on the device 3 to 4 % slower for it: ResNet-18 8x224 429 -> 446 us, ResNet-50 4x224 725 -> 755; with the care for
// infinities 452 and 769.)  The small products,
// 2^-8 of the large ones, share an accumulator for up to kSmallBlocks blocks.
//
// Activations between the layers of an fp32 network are stored as planes, [3][N][H][W][C] bf16: the epilogue splits each
// result once, and the tile loads are plain TMA copies of all three planes (nncv's fp32 graph: tests/Nets/Res18.mlir:118-629).
// The 7x7 stride-2 stem reads row pairs through a tensor map with overlapping strides, as stem.cu does: it becomes a
// convolution with four taps of 64 "channels".
//
// Two kernels.  conv_f32_kernel: one CTA computes 128 pixels x 64 or 128 output channels.  What bounds it: the port of shared memory, 128
// bytes a clock for what the MMAs of a block of 64 channels read (1152 or 1536 clocks) and about twice that for what is copied in (72 or
// 96 KB); 1430 and 1900 clocks a block were measured.  HALO, for filters of stride 1: one box of pixels serves a whole column of the filter
// (42 KB a block), and the filter's planes lie together, so that a1 multiplies b2 and b3 in one MMA of 128 columns (896 clocks): 1220.
// Two warps issue the MMAs of 64-column tiles, one the large products: an MMA takes its warp about 29 clocks, a wait or a commit about 80.
// us before and now: 56x56x64 of eight images 24.5 23.0, of 32 77 70, 28x28x128 of eight 24 21; 64 x 32 tiles 512 -> 512 on 7x7 by one CTA a
// tile 38.9 28.6.  128 columns leave room for one pair of accumulators, and what the tensor core does while that pair is handed over decides:
// one warp issues, ten of the twenty small steps between the two halves of the large products (512 -> 512 on 7x7 of 64 images by two
// warps 99 us, by one with twelve steps and eight 92, with ten and ten 90).
// Without HALO the first planes, which both issuing warps read, have a ring of their own: in one ring the warp of the large products has to
// wait for the other planes too, or a slot's barrier could be two uses ahead of it.  Slots for first and other planes, us: 64 columns,
// 64 -> 128 on 56x56 at stride 2 of eight images, one ring 16.7, 2 + 5 17.1, 3 + 4 16.35, 4 + 3 16.8; 128 columns, 128 -> 128 on 28x28 of
// 32, one ring 57.5, 1 + 4 72.6, 2 + 3 56.8, 3 + 2 65.8.  With few pixels a
// cluster of up to eight CTAs splits the reduction of a tile; each leaves its partial sums in shared memory and finishes
// its share of the rows from all of them, in rank order, so that the result does not depend on timing.  (The CUDA-core
// kernel needed a second pass over partial sums in global memory for that, and ran at a fifth of the fp32 rate.)
// Roles: warp 0 TMA producer, one plane of both operands per ring slot (HALO: boxes, and blocks of the filter); warps 1 and 18 MMA
// issuers (128 columns: warp 1); warps 2-17 epilogue (with eight of them, twice the columns each, ResNet-18 8x224 took 421 us and ResNet-50 4x224 802, where
// these took 395 and 704 with one sum a column; sixteen in two sets, a pair of accumulators each, saved nothing in the blocks and cost 1 us a tile).
// conv_f32_small_kernel, for one to four images: 64 pixels x 32 output channels, below.  conv_f32_choose takes one by a model of both.
//
// ResNet-18 fp32 against the CUDA-core kernel, from device memory: 1x256 470 -> 177 us, 8x224 1626 -> 401 us.
// Every wait is bounded and abortable; a timed-out wait sets the device status word.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <mutex>

#include "epilogue.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace nncv_b200 {

namespace {

constexpr int kEpiWarps = 16, kEpiThreads = 32 * kEpiWarps;
constexpr int kLargeWarp = 2 + kEpiWarps, kThreads = 32 * (kLargeWarp + 1);
constexpr int kABytes = 128 * 128;
constexpr int kBBytes = 64 * 128;           // packed weights: tiles of 64 output channels x 64 input channels
constexpr int kTileBytes = 128 * 64 * 4;    // partial sums of 64 of the tile's columns, fp32
constexpr int kSmallBlocks = 4;             // blocks of 64 channels whose small products share an accumulator
constexpr int kHaloB = 8, kBoxes = 2;       // halo tiles: blocks of weights (three planes) and boxes that rings can hold
constexpr float kCut = 3.0f / (1 << 28);    // what a step of the tensor core cuts off its sum, on average (0.19 * 2^-24)
template <int BN>
struct Ring {   // a slot holds one plane of a block: 128 pixels and BN output channels x 64 channels
  static constexpr int kSlots = BN == 64 ? 7 : 5;
  static constexpr int kFirst = BN == 64 ? 3 : 2;   // of them for first planes
  static constexpr int kSlot = kABytes + BN / 64 * kBBytes;
  static constexpr size_t kSmem = 1024 + (size_t)kSlots * kSlot + kTileBytes + 256;
};

struct F32Params {
  const uint8_t* wpack;       // [Kout tile][plane][k block] 64 x 64 bf16 tiles, swizzled
  const float* scale;
  const float* shift;
  const void* residual;       // planes (res_f32: fp32) of the output's shape, or null
  void* out;                  // planes, or fp32 with row pitch ldo
  long long res_plane, out_plane;  // elements from one plane to the next
  long long ldo;
  int* error_flag;
  int out_f32, res_f32, relu;
  int Kout, CB, taps, S, stride, pad_x, pad_y;
  int OH, OW, NB;
  // row r of a tile is pixel (r / mp / rows_img, r / mp % rows_img, r % mp) of its tn x th x tw, or none
  int tw, th, tn, mp, rows_img;
  int tiles_x, tiles_y, n_tiles, items;
  epi::FastDiv div_tx, div_ty, div_nt, div_mp, div_ri;
  // halo tiles: rows of the filter, bytes of a plane's box, blocks of weights that fit
  int R, a_plane, b_stages;
  int splits;                 // CTAs of a cluster that share a tile's reduction (a power of two up to 8)
};

// Infinities and NaN stay in the first plane; a finite value too large to be rounded to bf16 is cut to the largest one.
__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
  constexpr float kMaxBf16 = 3.38953139e38f;   // 2^128 - 2^120
  const bool finite = fabsf(x) <= FLT_MAX;
  a = __float2bfloat16_rn(finite ? fminf(fmaxf(x, -kMaxBf16), kMaxBf16) : x);
  const float r = finite ? x - __bfloat162float(a) : 0.0f;
  b = __float2bfloat16_rn(r);
  c = __float2bfloat16_rn(r - __bfloat162float(b));
}
// four values -> 8 bytes of each plane.  Where all four are finite and round to bf16 without overflow (nearly always) two are
// converted at a time and nothing is clamped: 7 instructions a value where split3 takes about 20, and the same planes.
__device__ __forceinline__ void split2(float x, float y, uint32_t (&o)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    o[q] = *reinterpret_cast<const uint32_t*>(&h);
    x -= __uint_as_float(o[q] << 16);
    y -= __uint_as_float(o[q] & 0xffff0000u);
  }
}
__device__ __forceinline__ void split4(const float4& v, uint2 (&o)[3]) {
  constexpr uint32_t kMaxBits = 0x7f7f0000u;   // the largest bf16
  const uint32_t top = max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu),
                           max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
  if (top <= kMaxBits) {
    uint32_t a[3], b[3];
    split2(v.x, v.y, a);
    split2(v.z, v.w, b);
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = make_uint2(a[q], b[q]);
    return;
  }
  const float x[4] = {v.x, v.y, v.z, v.w};
  __nv_bfloat16 s[3][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) split3(x[e], s[0][e], s[1][e], s[2][e]);
#pragma unroll
  for (int q = 0; q < 3; ++q) o[q] = *reinterpret_cast<const uint2*>(s[q]);
}
__device__ __forceinline__ float4 join4(const uint2 (&w)[3]) {
  float4 v;
  float* f = reinterpret_cast<float*>(&v);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float p[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const uint32_t u = (e & 2) ? w[q].y : w[q].x;
      p[q] = __uint_as_float((e & 1) ? (u & 0xffff0000u) : (u << 16));
    }
    f[e] = p[0] + (p[1] + p[2]);
  }
  return v;
}

template <int kBN, bool HALO>   // output channels of a tile: 64 or 128
__global__ void __launch_bounds__(kThreads, 1)
conv_f32_kernel(const __grid_constant__ CUtensorMap tm_in, const F32Params p) {
  static_assert(!HALO || kBN == 64, "halo tiles are 64 channels wide");
  constexpr int kSlots = HALO ? kHaloB : Ring<kBN>::kSlots, kSlot = HALO ? 3 * kBBytes : Ring<kBN>::kSlot, kNT = kBN / 64;
  // Accumulators: pairs for two steps of the large products, and two for the small ones.  A pair is handed over as one: the
  // epilogue's time is the latency of a hand-over, about 400 clocks, and four a block of 64 channels took longer than the copies.
  constexpr uint32_t kPairs = kBN == 64 ? 2 : 1, kAcc = kPairs + 2;
  constexpr uint32_t kTmemCols = 512, kSmallCols = kPairs * 2 * kBN;
  constexpr int kCols = kBN / 4;            // columns of a thread's row
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ __align__(8) unsigned long long s_bars[2 * kSlots + 2 * kAcc + 2 + 2 * kBoxes];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  // the ring; with halo tiles the boxes of pixels, then a ring of weights alone
  const uint32_t sBox = (raw + 1023u) & ~1023u;
  const int slots = HALO ? p.b_stages : kSlots;
  const uint32_t sRing = sBox + (HALO ? (uint32_t)(kBoxes * 3 * p.a_plane) : 0u);
  const uint32_t sTile = sRing + slots * kSlot;
  const uint32_t full = ptx::smem_u32(s_bars), empty = full + 8 * kSlots;
  const uint32_t d_full = empty + 8 * kSlots, d_empty = d_full + 8 * kAcc;   // pairs first
  const uint32_t part_ready = d_empty + 8 * kAcc, part_done = part_ready + 8;
  const uint32_t a_full = part_done + 8, a_empty = a_full + 8 * kBoxes;
  // the slots for first planes, and for the others (halo tiles: one ring of blocks of weights)
  constexpr uint32_t kFirst = HALO ? 0u : (uint32_t)Ring<kBN>::kFirst;
  constexpr bool kOneIssuer = !HALO && kBN == 128;
  __shared__ uint32_t s_tmem;
  const int warp = ptx::warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int S = p.splits;
  const uint32_t rank = S > 1 ? ptx::cluster_ctarank() : 0u;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kSlots; ++i) {
      ptx::mbar_init(full + 8 * i, 1);
      ptx::mbar_init(empty + 8 * i, !kOneIssuer && (HALO || i < (int)kFirst) ? 2 : 1);   // the issuing warps that read it
    }
    for (uint32_t i = 0; i < kAcc; ++i) {
      ptx::mbar_init(d_full + 8 * i, 1);
      ptx::mbar_init(d_empty + 8 * i, kEpiWarps);
    }
    ptx::mbar_init(part_ready, S);
    ptx::mbar_init(part_done, S);
    for (int i = 0; i < kBoxes; ++i) {
      ptx::mbar_init(a_full + 8 * i, 1);
      ptx::mbar_init(a_empty + 8 * i, 2);
    }
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_in);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&s_tmem), kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (S > 1) ptx::cluster_sync_all();   // every CTA's barriers exist before anyone arrives remotely
  ptx::tc_fence_after();
  const uint32_t tmem_base = (uint32_t)ptx::warp_uniform((int)*reinterpret_cast<volatile uint32_t*>(&s_tmem));
  volatile int* abort_flag = &s_abort;

  const int cluster_id = (int)blockIdx.x / S, clusters = (int)gridDim.x / S;
  const int kb_all = p.taps * p.CB;
  const int kb0 = kb_all * (int)rank / S, kb1 = kb_all * ((int)rank + 1) / S;   // this CTA's part of the reduction
  auto item_of = [&](int i, int& n0, int& oy0, int& ox0, int& n_tile) {
    const int w = cluster_id + i * clusters;
    if (w >= p.items) return false;
    const int m = (int)epi::div_by((uint32_t)w, p.div_nt);
    n_tile = w - m * p.n_tiles;
    const int t2 = (int)epi::div_by((uint32_t)m, p.div_tx);
    ox0 = (m - t2 * p.tiles_x) * p.tw;
    const int t3 = (int)epi::div_by((uint32_t)t2, p.div_ty);
    oy0 = (t2 - t3 * p.tiles_y) * p.th;
    n0 = t3 * p.tn;
    return true;
  };
  // block kb of the reduction: channel block outermost, then the taps
  const int packed_tiles = (p.Kout + 63) / 64;
  auto load_weights = [&](int n_tile, int plane, int cb, int tap, uint32_t slot, uint32_t issue) {
#pragma unroll
    for (int q = 0; q < kNT; ++q) {
      // the second half of the last, ragged tile has no weights: its columns are never stored, any tile will do
      const int t = min(n_tile * kNT + q, packed_tiles - 1);
      ptx::bulk_g2s(sRing + slot * kSlot + kABytes + q * kBBytes,
                    p.wpack + (((size_t)t * 3 + plane) * kb_all + (size_t)tap * p.CB + cb) * kBBytes, kBBytes, full + 8 * slot, issue);
    }
  };
  // halo tiles: blocks go channel block outermost, then filter column c, then filter row r
  auto block_of = [&](int kb, int& cb, int& c, int& r) {
    cb = kb / p.taps;
    c = (kb - cb * p.taps) / p.R;
    r = kb - cb * p.taps - c * p.R;
  };
  auto next_block = [&](int& cb, int& c, int& r) {
    if (++r == p.R) {
      r = 0;
      if (++c == p.S) { c = 0; ++cb; }
    }
  };
  auto load_block = [&](int n_tile, int cb, int tap, uint32_t slot, uint32_t issue) {
#pragma unroll
    for (int pl = 0; pl < 3; ++pl)
      ptx::bulk_g2s(sRing + slot * kSlot + pl * kBBytes, p.wpack + (((size_t)n_tile * 3 + pl) * kb_all + (size_t)tap * p.CB + cb) * kBBytes, kBBytes,
                    full + 8 * slot, issue);
  };
  // the slots of a ring in turn
  struct Turn {
    uint32_t slot, first, end, ring = 0;
    __device__ __forceinline__ void next() {
      if (++slot == end) { slot = first; ring ^= 1u; }
    }
  };
  const Turn firsts{0, 0, HALO ? (uint32_t)slots : kFirst}, others{kFirst, kFirst, (uint32_t)kSlots};
  // the packed weights never change: their first copies do not wait for the previous kernel
  uint32_t early = 0;
  if (warp == 0) {
    const uint32_t issue = ptx::elect_one();
    int n0, oy0, ox0, n_tile;
    if (HALO && item_of(0, n0, oy0, ox0, n_tile)) {
      int cb, c, r;
      block_of(kb0, cb, c, r);
      for (int kb = kb0; kb < kb1 && early < (uint32_t)slots; ++kb, ++early) {
        ptx::mbar_arrive_expect_tx(full + 8 * early, kSlot, issue);
        load_block(n_tile, cb, r * p.S + c, early, issue);
        next_block(cb, c, r);
      }
    } else if (!HALO && item_of(0, n0, oy0, ox0, n_tile)) {
      int cb = kb0 / p.taps, tap = kb0 - cb * p.taps;
      Turn t1 = firsts, t2 = others;
      for (int kb = kb0; kb < kb1; ++kb) {
        int pl = 0;
        for (; pl < 3; ++pl, ++early) {
          Turn& t = pl == 0 ? t1 : t2;
          if (t.ring != 0) break;   // round once
          ptx::mbar_arrive_expect_tx(full + 8 * t.slot, kSlot, issue);
          load_weights(n_tile, pl, cb, tap, t.slot, issue);
          t.next();
        }
        if (pl < 3) break;
        if (++tap == p.taps) { tap = 0; ++cb; }
      }
    }
  }
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer ----
    if constexpr (HALO) {
      const uint32_t issue = ptx::elect_one();
      uint32_t slot = 0, ring = 0, cnt = 0, seen = 1, as = 0, a_ring = 0;
      bool okw = true;
      for (int i = 0; okw; ++i) {
        int n0, oy0, ox0, n_tile;
        if (!item_of(i, n0, oy0, ox0, n_tile)) break;
        int cb, c, r;
        block_of(kb0, cb, c, r);
        for (int kb = kb0; kb < kb1 && okw; ++kb, ++cnt) {
          if (kb == kb0 || r == 0) {   // the pixels under a column of the filter
            if (!ptx::warp_wait(a_empty + 8 * as, a_ring ^ 1u, abort_flag)) { okw = false; break; }
            ptx::mbar_arrive_expect_tx(a_full + 8 * as, 3u * (uint32_t)p.a_plane, issue);
            for (int pl = 0; pl < 3; ++pl)
              ptx::tma_load_5d(sBox + (as * 3 + pl) * (uint32_t)p.a_plane, &tm_in, cb * 64, ox0 - p.pad_x + c, oy0 - p.pad_y, n0, pl, a_full + 8 * as, issue);
            if (++as == (uint32_t)kBoxes) { as = 0; a_ring ^= 1u; }
          }
          if (cnt >= early) {
            if (!ptx::warp_all(seen) && !ptx::warp_wait(empty + 8 * slot, ring ^ 1u, abort_flag)) { okw = false; break; }
            ptx::mbar_arrive_expect_tx(full + 8 * slot, kSlot, issue);
            load_block(n_tile, cb, r * p.S + c, slot, issue);
          }
          if (++slot == (uint32_t)slots) { slot = 0; ring ^= 1u; }
          seen = ptx::mbar_peek(empty + 8 * slot, ring ^ 1u);
          next_block(cb, c, r);
        }
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    } else {
      const uint32_t issue = ptx::elect_one();
      Turn t1 = firsts, t2 = others;
      uint32_t cnt = 0, seen = 1;
      bool okw = true;
      for (int i = 0; okw; ++i) {
        int n0, oy0, ox0, n_tile;
        if (!item_of(i, n0, oy0, ox0, n_tile)) break;
        const int xb = p.stride * ox0 - p.pad_x, yb = p.stride * oy0 - p.pad_y;
        int cb = kb0 / p.taps, tap = kb0 - cb * p.taps;
        int r = tap / p.S, s = tap - r * p.S;
        for (int kb = kb0; kb < kb1 && okw; ++kb) {
#pragma unroll
          for (int pl = 0; pl < 3; ++pl, ++cnt) {
            const bool begun = cnt < early;
            Turn& t = pl == 0 ? t1 : t2;
            if (!ptx::warp_all(seen) && !ptx::warp_wait(empty + 8 * t.slot, t.ring ^ 1u, abort_flag)) { okw = false; break; }
            if (!begun) ptx::mbar_arrive_expect_tx(full + 8 * t.slot, kSlot, issue);
            const uint32_t dst = sRing + t.slot * kSlot;
            ptx::tma_load_5d(dst, &tm_in, cb * 64, xb + s, yb + r, n0, pl, full + 8 * t.slot, issue);
            if (!begun) load_weights(n_tile, pl, cb, tap, t.slot, issue);
            t.next();
            const Turn& n = pl == 2 ? t1 : t2;
            seen = ptx::mbar_peek(empty + 8 * n.slot, n.ring ^ 1u);
          }
          if (++s == p.S) { s = 0; ++r; }
          if (++tap == p.taps) { tap = r = s = 0; ++cb; }
        }
      }
      if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
    }
  } else if (warp == 1 || warp == kLargeWarp) {
    // ------------------------------------------------------------------ MMA issuers -----
    // One warp for the large products, one for the small ones: an MMA takes its warp about 29 clocks and a wait or a commit about 80,
    // so a lone warp needed longer for the 20 or 24 MMAs of a block, with their hand-overs, than the tensor core.  MMAs of 128 columns
    // take twice as long, and a lone warp orders them.
    const bool large_warp = warp == kLargeWarp;
    const uint32_t issue = ptx::elect_one();
    const uint32_t idesc = ptx::umma_idesc(128, kBN, 1), idesc2 = HALO ? ptx::umma_idesc(128, 128, 1) : idesc;
    Turn t1 = firsts, t2 = others;   // halo tiles: blocks of weights, none
    uint32_t as = 0, a_ring = 0;     // halo tiles: the box in use
    uint32_t uses = 0, pair_uses = 0;   // of small accumulators and of pairs, as far as this warp fills them
    bool okw = true;
    uint32_t seen = ptx::mbar_peek(full, 0);
    // the slot t is full; `then` is the one that this warp needs after it
    auto arrive = [&](Turn& t, const Turn& then, uint32_t& now) {
      if (!ptx::warp_all(seen) && !ptx::warp_wait(full + 8 * t.slot, t.ring, abort_flag)) return false;
      ptx::tc_fence_after();
      now = t.slot;
      t.next();
      seen = ptx::mbar_peek(full + 8 * then.slot, then.ring);
      return true;
    };
    // step k4 (16 channels) of operands whose descriptors start at a and b
    auto mma = [&](uint32_t d, uint32_t a, uint32_t b, uint32_t k4, uint32_t id, uint32_t accumulate) {
      ptx::umma_f16(d, ptx::desc_from_halves(a + k4 * 2, ptx::kSmemDescK128Hi), ptx::desc_from_halves(b + k4 * 2, ptx::kSmemDescK128Hi), id, accumulate, issue);
    };
    // a product of two planes of the block: four steps of 16 channels
    auto product = [&](uint32_t d, uint32_t a, uint32_t b, uint32_t id, uint32_t fresh) {
#pragma unroll
      for (uint32_t k4 = 0; k4 < 4; ++k4) mma(d, a, b, k4, id, k4 == 0 ? (fresh ^ 1u) : 1u);
    };
    // two steps of the large products, each into an accumulator of its own, handed over as a pair
    auto two_large = [&](uint32_t a, uint32_t b, uint32_t k4) {
      const uint32_t pair = pair_uses % kPairs;
      if (!ptx::warp_wait(d_empty + 8 * pair, ((pair_uses / kPairs) & 1u) ^ 1u, abort_flag)) return false;
      ptx::tc_fence_after();
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j) mma(tmem_base + (2 * pair + j) * kBN, a, b, k4 + j, idesc, 0u);
      ptx::tc_commit(d_full + 8 * pair, issue);
      ++pair_uses;
      return true;
    };
    for (int i = 0; okw && !(kOneIssuer && large_warp); ++i) {
      int n0, oy0, ox0, n_tile;
      if (!item_of(i, n0, oy0, ox0, n_tile)) break;
      int r = HALO ? kb0 % p.R : 0;   // rows of the filter divide the taps
      for (int kb = kb0; kb < kb1; ++kb) {
        const bool group_first = (kb - kb0) % kSmallBlocks == 0, group_last = (kb - kb0) % kSmallBlocks == kSmallBlocks - 1 || kb + 1 == kb1;
        const uint32_t acc = kPairs + (uses & 1u), ds = tmem_base + kSmallCols + (uses & 1u) * (HALO ? 2 : 1) * kBN;
        auto small_ready = [&]() {
          if (!group_first) return true;
          if (!ptx::warp_wait(d_empty + 8 * acc, ((uses >> 1) & 1u) ^ 1u, abort_flag)) return false;
          ptx::tc_fence_after();
          return true;
        };
        const uint32_t fresh = group_first ? 1u : 0u;
        uint32_t now[3];
        if constexpr (HALO) {
          if ((kb == kb0 || r == 0) && !ptx::warp_wait(a_full + 8 * as, a_ring, abort_flag)) { okw = false; break; }
          if (!arrive(t1, t1, now[0])) { okw = false; break; }
          // filter row r reads the box from its row r on: mp pixels, a multiple of eight rows of 128 bytes
          const uint32_t b = ptx::smem_desc_k128_lo(sRing + now[0] * kSlot), bp = kBBytes >> 4, ap = (uint32_t)p.a_plane >> 4;
          const uint32_t a = ptx::smem_desc_k128_lo(sBox + as * 3 * (uint32_t)p.a_plane + (uint32_t)(r * p.mp) * 128u);
          if (large_warp) {
            if (!two_large(a, b, 0) || !two_large(a, b, 2)) { okw = false; break; }
          } else {
            if (!small_ready()) { okw = false; break; }
            // two accumulators side by side: a1 b2 | a1 b3, a2 b1 | a2 b2, a3 b1
            product(ds, a, b + bp, idesc2, fresh);
            product(ds, a + ap, b, idesc2, 0u);
            product(ds, a + 2 * ap, b, idesc, 0u);
          }
          ptx::tc_commit(empty + 8 * now[0], issue);
          if (++r == p.R) r = 0;
          if (r == 0 || kb + 1 == kb1) {
            ptx::tc_commit(a_empty + 8 * as, issue);
            if (++as == (uint32_t)kBoxes) { as = 0; a_ring ^= 1u; }
          }
        } else {
          auto at = [&](uint32_t sl) { return ptx::smem_desc_k128_lo(sRing + sl * kSlot); };
          constexpr uint32_t kB = kABytes >> 4;
          if (!arrive(t1, large_warp ? t1 : t2, now[0])) { okw = false; break; }
          const uint32_t first = at(now[0]);
          if (large_warp) {
            if (!two_large(first, first + kB, 0) || !two_large(first, first + kB, 2)) { okw = false; break; }
            ptx::tc_commit(empty + 8 * now[0], issue);
          } else {
            if (kOneIssuer && !two_large(first, first + kB, 0)) { okw = false; break; }
            if (!arrive(t2, t2, now[1]) || !small_ready()) { okw = false; break; }
            product(ds, first, at(now[1]) + kB, idesc, fresh);
            product(ds, at(now[1]), first + kB, idesc, 0u);
            const uint32_t second = at(now[1]);
#pragma unroll
            for (uint32_t k4 = 0; k4 < 4; ++k4) {
              // half of the twenty small steps later, when the epilogue has had the time to empty the accumulators
              if (kOneIssuer && k4 == 2 && !two_large(first, first + kB, 2)) { okw = false; break; }
              mma(ds, second, second + kB, k4, idesc, 1u);
            }
            if (!okw) break;
            if (!arrive(t2, t1, now[2])) { okw = false; break; }
            product(ds, first, at(now[2]) + kB, idesc, 0u);
            product(ds, at(now[2]), first + kB, idesc, 0u);
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) ptx::tc_commit(empty + 8 * now[pl], issue);
          }
        }
        if (!large_warp && group_last) {
          ptx::tc_commit(d_full + 8 * acc, issue);
          ++uses;
        }
      }
    }
    if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitMma);
  } else {
    // ------------------------------------------------------------------ epilogue --------
    const int quad = warp & 3, part = (warp - 2) >> 2;   // rows, and a quarter of the tile's columns
    const int row = quad * 32 + lane;
    const int et = (int)threadIdx.x - 64;
    const int rows_each = 128 / S, row_lo = (int)rank * rows_each;
    const int g = et & 15;             // four columns of the tile
    constexpr int kRows = 128 * 16 / kEpiThreads;   // rows a thread finishes
    uint32_t large = 0, small = 0;     // running counts of uses of the accumulators
    bool okw = true;
    for (int i = 0; okw; ++i) {
      int n0, oy0, ox0, n_tile;
      if (!item_of(i, n0, oy0, ox0, n_tile)) break;
      const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * kCols);
      // 64 columns: the large products in two sums, of steps 0 and 1 and of steps 2 and 3 of the blocks, half as many roundings one after
      // another: clusters of fewer CTAs have longer sums, and with one sum the logits of ResNet-18 were 1.0 % further off on average than
      // before these tiles, with two 0.1 % (ResNet-50 0.2 % and 1.4 % nearer), for 0.3 % of the time (ResNet-18 8x224 399 -> 401 us).
      constexpr bool kTwo = kBN == 64;
      float sum[kCols], other[kTwo ? kCols : 1];
#pragma unroll
      for (int e = 0; e < kCols; ++e) sum[e] = other[kTwo ? e : 0] = 0.0f;
      auto hand_back = [&](uint32_t acc) {
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(d_empty + 8 * acc);
      };
      // adds a pair's columns (this thread's row) to the sums `into`
      auto take_pair = [&](uint32_t pair, uint32_t turn, float* into) {
        if (!ptx::warp_wait(d_full + 8 * pair, turn & 1u, abort_flag)) return false;
        ptx::tc_fence_after();
#pragma unroll
        for (int h = 0; h < kCols / 16; ++h) {
          uint32_t v[2][16];
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j) ptx::tmem_ld_32x16(lane_base + (2 * pair + j) * kBN + h * 16, v[j]);
          ptx::tmem_ld_wait();
          if (h == kCols / 16 - 1) hand_back(pair);
#pragma unroll
          for (int e = 0; e < 16; ++e) into[h * 16 + e] += __uint_as_float(v[0][e]) + __uint_as_float(v[1][e]);
        }
        return true;
      };
      // adds small products; kCut of the sum is given back with the last of them, whose low bits decide how it rounds.  An
      // infinite or NaN operand makes the large products what they have to be; its small products (inf * 0, inf - inf) say nothing.
      auto take_small = [&](bool last) {
        const uint32_t acc = kPairs + (small & 1u);
        if (!ptx::warp_wait(d_full + 8 * acc, (small >> 1) & 1u, abort_flag)) return false;
        ptx::tc_fence_after();
#pragma unroll
        for (int h = 0; h < kCols / 16; ++h) {
          uint32_t v[16], w[HALO ? 16 : 1];
          ptx::tmem_ld_32x16(lane_base + kSmallCols + (small & 1u) * (HALO ? 2 * kBN : kBN) + h * 16, v);
          if constexpr (HALO) ptx::tmem_ld_32x16(lane_base + kSmallCols + (small & 1u) * 2 * kBN + kBN + h * 16, w);
          ptx::tmem_ld_wait();
          if (h == kCols / 16 - 1) hand_back(acc);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float rest = HALO ? __uint_as_float(v[e]) + __uint_as_float(w[HALO ? e : 0]) : __uint_as_float(v[e]);
            rest = fabsf(rest) <= FLT_MAX ? rest : 0.0f;
            float& s = sum[h * 16 + e];
            if (!last) { s += rest; continue; }
            if (kTwo) s += other[kTwo ? h * 16 + e : 0];
            s = fabsf(s) <= FLT_MAX ? s + fmaf(s, kCut, rest) : s;
          }
        }
        ++small;
        return true;
      };
      for (int kb = kb0; kb < kb1 && okw; ++kb) {
        okw = take_pair(large % kPairs, large / kPairs, sum);
        ++large;
        okw = okw && take_pair(large % kPairs, large / kPairs, kTwo ? other : sum);
        ++large;
        if (okw && ((kb - kb0) % kSmallBlocks == kSmallBlocks - 1 || kb + 1 == kb1)) okw = take_small(kb + 1 == kb1);
      }
      // the pixels this thread finishes: row r of the tile -> its index in the output, -1 outside
      int pix[kRows];
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        const int rr = (et >> 4) + k * (kEpiThreads / 16), r = row_lo + rr;
        const int t1 = (int)epi::div_by((uint32_t)r, p.div_mp), tj = r - t1 * p.mp;
        const int t2 = (int)epi::div_by((uint32_t)t1, p.div_ri), ti = t1 - t2 * p.rows_img;
        const int img = n0 + t2, oy = oy0 + ti, ox = ox0 + tj;
        const bool in_tile = !HALO || (tj < p.tw && ti < p.th && t2 < p.tn);
        pix[k] = in_tile && rr < rows_each && img < p.NB && oy < p.OH && ox < p.OW ? (img * p.OH + oy) * p.OW + ox : -1;
      }
      // 64 columns at a time
#pragma unroll
      for (int pass = 0; pass < kNT; ++pass) {
        const uint32_t turn = (uint32_t)(i * kNT + pass);   // uses of the shared tile
        const int n = n_tile * kBN + pass * 64 + 4 * g;
        // residual planes, requested before the sums are in the shared tile
        uint2 res[kRows][3];
        if (p.residual && !p.res_f32 && n < p.Kout) {
#pragma unroll
          for (int k = 0; k < kRows; ++k)
            if (pix[k] >= 0) {
#pragma unroll
              for (int q = 0; q < 3; ++q)
                res[k][q] = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p.residual) + q * p.res_plane + (long long)pix[k] * p.Kout + n));
            }
        }
        // the previous item's partial sums have been read by everybody
        if (okw && turn > 0 && S > 1) okw = ptx::warp_wait_cluster(part_done, (turn - 1) & 1u, abort_flag);
        if (!ptx::named_bar_and(1, kEpiThreads, okw)) { okw = false; break; }
        if (kNT == 1 || part >> 1 == pass) {
          constexpr int kChunks = kCols / 4;   // 16 bytes each; sixteen chunks a row, those of a row's parts one after another
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            epi::sts128(sTile + (uint32_t)row * 256u + (((uint32_t)((kNT == 1 ? part : part & 1) * kChunks + c) ^ (uint32_t)(row & 7)) << 4),
                        __float_as_uint(sum[4 * c]), __float_as_uint(sum[4 * c + 1]), __float_as_uint(sum[4 * c + 2]), __float_as_uint(sum[4 * c + 3]));
        }
        ptx::named_bar_sync(2, kEpiThreads);
        if (S > 1) {
          if (et < S) ptx::mbar_arrive_remote(ptx::map_to_cta(part_ready, (uint32_t)et));
          okw = ptx::warp_wait_cluster(part_ready, turn & 1u, abort_flag);
          if (!ptx::named_bar_and(1, kEpiThreads, okw)) { okw = false; break; }
        }
        if (n < p.Kout) {
          float4 sc = make_float4(1.f, 1.f, 1.f, 1.f), sh = make_float4(0.f, 0.f, 0.f, 0.f);
          float* scp = reinterpret_cast<float*>(&sc);
          float* shp = reinterpret_cast<float*>(&sh);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (p.scale) scp[e] = __ldg(p.scale + n + e);
            if (p.shift) shp[e] = __ldg(p.shift + n + e);
          }
#pragma unroll
          for (int k = 0; k < kRows; ++k) {
            if (pix[k] < 0) continue;
            const int r = row_lo + (et >> 4) + k * (kEpiThreads / 16);
            const uint32_t at = sTile + (uint32_t)r * 256u + (((uint32_t)g ^ (uint32_t)(r & 7)) << 4);
            float4 v;
            if (S == 1) {
              const uint4 w = epi::lds128(at);
              v = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
            } else {
              v = ptx::ld_cluster_f4(ptx::map_to_cta(at, 0));
              for (int q = 1; q < S; ++q) {
                const float4 w = ptx::ld_cluster_f4(ptx::map_to_cta(at, (uint32_t)q));
                v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
              }
            }
            v.x = fmaf(v.x, sc.x, sh.x); v.y = fmaf(v.y, sc.y, sh.y); v.z = fmaf(v.z, sc.z, sh.z); v.w = fmaf(v.w, sc.w, sh.w);
            if (p.residual) {
              float4 f;
              if (p.res_f32) {
                f = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p.residual) + (long long)pix[k] * p.ldo + n));
              } else {
                f = join4(res[k]);
              }
              v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
            }
            if (p.relu) {
              v.x = !(v.x <= 0.0f) ? v.x : 0.0f; v.y = !(v.y <= 0.0f) ? v.y : 0.0f;
              v.z = !(v.z <= 0.0f) ? v.z : 0.0f; v.w = !(v.w <= 0.0f) ? v.w : 0.0f;
            }
            if (p.out_f32) {
              *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (long long)pix[k] * p.ldo + n) = v;
            } else {
              uint2 o[3];
              split4(v, o);
#pragma unroll
              for (int q = 0; q < 3; ++q)
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + q * p.out_plane + (long long)pix[k] * p.Kout + n) = o[q];
            }
          }
        }
        if (S > 1) {
          ptx::named_bar_sync(2, kEpiThreads);
          if (et < S) ptx::mbar_arrive_remote(ptx::map_to_cta(part_done, (uint32_t)et));
        }
      }
    }
    if (!okw && et == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitEpilogue);
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (S > 1) ptx::cluster_sync_all();   // the peers' reads of this CTA's partial sums are over
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------ small batches ----------
// The same convolution on 64 x 32 tiles, one a CTA, for few pixels.  At one image what bounds a layer is its chain, and most of
// that of the kernel above is not tensor work: after 2 to 9 blocks, whose MMAs read 6 KB each (48 clocks), a CTA of a cluster waits
// for its peers' word, for 32 KB of their partial sums and until all may leave.  Here a block takes 16 MMAs, two products side by
// side where they share an operand, of 24 to 32 clocks each; four warps copy, whole blocks are handed over, and the partial sums,
// a quarter as many, are SENT: every CTA stores the rows that a peer finishes into that peer's shared memory and arrives on its
// barrier, so that nobody reads from a CTA that could leave, and nobody waits for more than its own rows.  One image, us, wide tiles
// and these: 14x14x256 -> 256 3x3 13.4 11.0 (128 CTAs; the tensor pipe 12 % busy), 7x7x512 -> 512 16.1 14.1, 56x56x256 -> 64 pointwise
// 11.0 8.0; ResNet-18 224 -> 187.
// The sums are formed as above: each step of 16 channels of the large products rounded to registers, small products in groups; but
// with fewer CTAs to a tile a sum has more terms one after another, so a block's four steps are added first, and even and odd
// blocks apart (one chain: 9.5e-8 instead of 7.1e-8 off the result in 64 bits for 64 channels 3x3, where the kernel above split).
constexpr int kSM = 64, kSN = 32;                       // tile
constexpr int kSABytes = kSM * 128, kSBBytes = kSN * 128;
constexpr int kSB = 3 * kSABytes, kSStage = kSB + 3 * kSBBytes;   // the pixels' planes, then the filter's, one below the other
constexpr int kSStages = 6;                             // 216 KB: six blocks of 64 channels
constexpr size_t kSSmem = 1024 + (size_t)kSStages * kSStage;
constexpr int kSCopyWarps = 4, kSLargeWarp = 1 + kSCopyWarps + 4, kSThreads = (kSLargeWarp + 1) * 32;

// Loads that stay where they stand (the compiler moves plain ones down to their use, behind the waits they should overlap).
__device__ __forceinline__ uint2 load_now(const __nv_bfloat16* q) {
  uint2 r;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(q));
  return r;
}
__device__ __forceinline__ float4 load_now(const float* q) {
  float4 r;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(q));
  return r;
}
__device__ __forceinline__ float4 load_single(const float* q) {   // four values that need not lie on a 16-byte boundary
  float4 r;
  asm volatile("ld.global.f32 %0, [%4];\n ld.global.f32 %1, [%4 + 4];\n ld.global.f32 %2, [%4 + 8];\n ld.global.f32 %3, [%4 + 12];"
               : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(q));
  return r;
}

__global__ void __launch_bounds__(kSThreads, 1) conv_f32_small_kernel(const __grid_constant__ CUtensorMap tm_in, const F32Params p) {
  constexpr uint32_t kQuad = 4 * kSN, kSmallCols = 2 * kQuad;   // two sets of the four large steps' accumulators, two pairs of small ones
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(16) float s_recv[kSM * kSN];             // [part][row of this CTA's][column]
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) unsigned long long s_bars[2 * kSStages + 9];
  const uint32_t ring = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t full = ptx::smem_u32(s_bars), empty = full + 8 * kSStages, d_full = empty + 8 * kSStages, d_empty = d_full + 16;
  const uint32_t s_full = d_empty + 16, s_empty = s_full + 16, recv = s_empty + 16;
  const int warp = ptx::warp_uniform((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int S = p.splits;
  const uint32_t rank = S > 1 ? ptx::cluster_ctarank() : 0u;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kSStages; ++i) {
      ptx::mbar_init(full + 8 * i, 1);
      ptx::mbar_init(empty + 8 * i, 2);   // both issuing warps
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(d_full + 8 * i, 1);
      ptx::mbar_init(d_empty + 8 * i, 4);
      ptx::mbar_init(s_full + 8 * i, 1);
      ptx::mbar_init(s_empty + 8 * i, 4);
    }
    ptx::mbar_init(recv, S > 4 ? S : 4);   // one arrival of each warp that sends rows here
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&tm_in);
  }
  if (warp == 0) {
    ptx::tmem_alloc(ptx::smem_u32(&s_tmem), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (S > 1) ptx::cluster_sync_all();   // every CTA's barriers exist before anyone sends
  ptx::tc_fence_after();
  const uint32_t tmem = (uint32_t)ptx::warp_uniform((int)*reinterpret_cast<volatile uint32_t*>(&s_tmem));
  volatile int* abort_flag = &s_abort;

  const int w = (int)blockIdx.x / S;
  const int m_item = (int)epi::div_by((uint32_t)w, p.div_nt), n_tile = w - m_item * p.n_tiles;
  const int t2 = (int)epi::div_by((uint32_t)m_item, p.div_tx), t3 = (int)epi::div_by((uint32_t)t2, p.div_ty);
  const int ox0 = (m_item - t2 * p.tiles_x) * p.tw, oy0 = (t2 - t3 * p.tiles_y) * p.th, n0 = t3 * p.tn;
  const int kb_all = p.taps * p.CB, kb0 = kb_all * (int)rank / S, blocks = kb_all * ((int)rank + 1) / S - kb0;   // this CTA's part

  if (warp == 0 || warp == kSLargeWarp) {
    // ------------------------------------------------------------------ MMAs: large products, small ones ----
    const bool large_warp = warp == kSLargeWarp;
    const uint32_t issue = ptx::elect_one();
    const uint32_t idesc = ptx::umma_idesc(kSM, kSN, 1), idesc2 = ptx::umma_idesc(kSM, 2 * kSN, 1);
    const uint32_t ring_lo = ptx::smem_desc_k128_lo(ring);
    // pixels' plane pa times the filter's plane pb (and the next one, idesc2)
    auto mma = [&](uint32_t d, uint32_t at, uint32_t pa, uint32_t pb, uint32_t k4, uint32_t id, uint32_t accumulate) {
      ptx::umma_f16(d, ptx::desc_from_halves(at + ((pa * kSABytes) >> 4) + k4 * 2, ptx::kSmemDescK128Hi),
                    ptx::desc_from_halves(at + ((kSB + pb * kSBBytes) >> 4) + k4 * 2, ptx::kSmemDescK128Hi), id, accumulate, issue);
    };
    uint32_t st = 0, par = 0;
    bool okw = true;
    for (int i = 0; i < blocks; ++i) {
      const uint32_t q = (uint32_t)i & 1u, group = (uint32_t)i / kSmallBlocks, sb = group & 1u;
      const bool first = i % kSmallBlocks == 0, last = i % kSmallBlocks == kSmallBlocks - 1 || i + 1 == blocks;
      if (!ptx::warp_spin(full + 8 * st, par, abort_flag)) { okw = false; break; }
      const uint32_t at = ring_lo + st * (uint32_t)(kSStage >> 4), ds = tmem + kSmallCols + sb * 2 * kSN;
      if (large_warp) {
        if (i >= 2 && !ptx::warp_spin(d_empty + 8 * q, (((uint32_t)i >> 1) & 1u) ^ 1u, abort_flag)) { okw = false; break; }
        ptx::tc_fence_after();
#pragma unroll
        for (uint32_t k4 = 0; k4 < 4; ++k4) mma(tmem + q * kQuad + k4 * kSN, at, 0, 0, k4, idesc, 0u);
        ptx::tc_commit(d_full + 8 * q, issue);
      } else {
        if (first && group >= 2 && !ptx::warp_spin(s_empty + 8 * sb, ((group >> 1) & 1u) ^ 1u, abort_flag)) { okw = false; break; }
        ptx::tc_fence_after();
        // the small products in two accumulators side by side: a1 b2 | a1 b3, a2 b1 | a2 b2, a3 b1
#pragma unroll
        for (uint32_t k4 = 0; k4 < 4; ++k4) mma(ds, at, 0, 1, k4, idesc2, first && k4 == 0 ? 0u : 1u);
#pragma unroll
        for (uint32_t k4 = 0; k4 < 4; ++k4) mma(ds, at, 1, 0, k4, idesc2, 1u);
#pragma unroll
        for (uint32_t k4 = 0; k4 < 4; ++k4) mma(ds, at, 2, 0, k4, idesc, 1u);
        if (last) ptx::tc_commit(s_full + 8 * sb, issue);
      }
      ptx::tc_commit(empty + 8 * st, issue);
      if (++st == kSStages) { st = 0; par ^= 1u; }
    }
    if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitMma);
    ptx::grid_dependency_wait();
  } else if (warp <= kSCopyWarps) {
    // ------------------------------------------------------------------ copies: block i by warp 1 + i % 4 ----
    const uint32_t issue = ptx::elect_one();
    const int me = warp - 1;
    auto where = [&](int i, int& cb, int& tap) {
      cb = (kb0 + i) / p.taps;
      tap = kb0 + i - cb * p.taps;
    };
    auto load_weights = [&](int cb, int tap, uint32_t st) {
#pragma unroll
      for (int pl = 0; pl < 3; ++pl)   // packed as tiles of 64 output channels: half of one
        ptx::bulk_g2s(ring + st * kSStage + kSB + pl * kSBBytes,
                      p.wpack + (((size_t)(n_tile >> 1) * 3 + pl) * kb_all + (size_t)tap * p.CB + cb) * kBBytes + (n_tile & 1) * kSBBytes, kSBBytes, full + 8 * st, issue);
    };
    // the packed weights never change: their first copies do not wait for the previous kernel
    for (int i = me; i < kSStages && i < blocks; i += kSCopyWarps) {
      int cb, tap;
      where(i, cb, tap);
      ptx::mbar_arrive_expect_tx(full + 8 * i, kSStage, issue);
      load_weights(cb, tap, (uint32_t)i);
    }
    const int xb = p.stride * ox0 - p.pad_x, yb = p.stride * oy0 - p.pad_y;
    int cb, tap;
    where(me, cb, tap);
    int r = tap / p.S, s = tap - r * p.S;
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();
    bool okw = true;
    for (int i = me; i < blocks; i += kSCopyWarps) {
      const uint32_t turn = (uint32_t)i / kSStages, st = (uint32_t)i - turn * kSStages;
      if (turn > 0) {
        if (!ptx::warp_spin(empty + 8 * st, (turn & 1u) ^ 1u, abort_flag)) { okw = false; break; }
        ptx::mbar_arrive_expect_tx(full + 8 * st, kSStage, issue);
      }
#pragma unroll
      for (int pl = 0; pl < 3; ++pl)
        ptx::tma_load_5d(ring + st * kSStage + pl * kSABytes, &tm_in, cb * 64, xb + s, yb + r, n0, pl, full + 8 * st, issue);
      if (turn > 0) load_weights(cb, tap, st);
      where(i + kSCopyWarps, cb, tap);
      r = tap / p.S;
      s = tap - r * p.S;
    }
    if (!okw && lane == 0 && p.error_flag) atomicCAS(p.error_flag, 0, (int)kErrWaitProducer);
  } else {
    // ------------------------------------------------------------------ epilogue --------
    ptx::grid_dependency_wait();
    // rows 16 quad .. 16 quad + 15 of the tile lie in the first sixteen lanes of the warp's quadrant
    const int quad = warp & 3, et = (int)threadIdx.x - (1 + kSCopyWarps) * 32;
    const int rows_each = kSM / S, n = n_tile * kSN + 4 * (et & 7);
    const bool live = n < p.Kout;
    // the rows this thread finishes, four columns each: (et >> 3) + 16 k of this CTA's
    long long pix[4];
    uint2 res[4][3];
    float4 res32[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int rr = (et >> 3) + 16 * k, r = (int)rank * rows_each + rr;
      const int t1 = (int)epi::div_by((uint32_t)r, p.div_mp), tj = r - t1 * p.mp;
      const int tt = (int)epi::div_by((uint32_t)t1, p.div_ri), ti = t1 - tt * p.rows_img;
      const int img = n0 + tt, oy = oy0 + ti, ox = ox0 + tj;
      pix[k] = live && rr < rows_each && img < p.NB && oy < p.OH && ox < p.OW ? ((long long)img * p.OH + oy) * p.OW + ox : -1;
      if (p.residual && pix[k] >= 0) {
        if (p.res_f32) {
          res32[k] = load_now(static_cast<const float*>(p.residual) + pix[k] * p.ldo + n);
        } else {
#pragma unroll
          for (int q = 0; q < 3; ++q) res[k][q] = load_now(static_cast<const __nv_bfloat16*>(p.residual) + q * p.res_plane + pix[k] * p.Kout + n);
        }
      }
    }
    const float4 sc = p.scale && live ? load_single(p.scale + n) : make_float4(1.f, 1.f, 1.f, 1.f);
    const float4 sh = p.shift && live ? load_single(p.shift + n) : make_float4(0.f, 0.f, 0.f, 0.f);
    // large products of even and of odd blocks, small products: three sums, added at the end
    float sum[16], odd[16], rest[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) sum[e] = odd[e] = rest[e] = 0.0f;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
    auto hand_back = [&](uint32_t bar) {
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar);
    };
    bool okw = true;
    for (int i = 0; i < blocks; ++i) {
      const uint32_t q = (uint32_t)i & 1u;
      if (!ptx::warp_spin(d_full + 8 * q, ((uint32_t)i >> 1) & 1u, abort_flag)) { okw = false; break; }
      ptx::tc_fence_after();
      uint32_t v[4][16];
#pragma unroll
      for (uint32_t k4 = 0; k4 < 4; ++k4) ptx::tmem_ld_16x32_f(lane_base + q * kQuad + k4 * kSN, v[k4]);
      ptx::tmem_ld_wait();
      hand_back(d_empty + 8 * q);
      float t[16];
#pragma unroll
      for (int e = 0; e < 16; ++e)
        t[e] = (__uint_as_float(v[0][e]) + __uint_as_float(v[1][e])) + (__uint_as_float(v[2][e]) + __uint_as_float(v[3][e]));
      if (q) {
#pragma unroll
        for (int e = 0; e < 16; ++e) odd[e] += t[e];
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) sum[e] += t[e];
      }
      if (i % kSmallBlocks == kSmallBlocks - 1 || i + 1 == blocks) {
        const uint32_t group = (uint32_t)i / kSmallBlocks, sb = group & 1u;
        if (!ptx::warp_spin(s_full + 8 * sb, (group >> 1) & 1u, abort_flag)) { okw = false; break; }
        ptx::tc_fence_after();
        ptx::tmem_ld_16x32_f(lane_base + kSmallCols + sb * 2 * kSN, v[0]);
        ptx::tmem_ld_16x32_f(lane_base + kSmallCols + sb * 2 * kSN + kSN, v[1]);
        ptx::tmem_ld_wait();
        hand_back(s_empty + 8 * sb);
#pragma unroll
        for (int e = 0; e < 16; ++e) rest[e] += __uint_as_float(v[0][e]) + __uint_as_float(v[1][e]);
      }
    }
    if (okw) {
      // what the steps lost on average is given back with the small products; an infinite or NaN sum stays as it is (see take_small)
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float s = sum[e] + odd[e], t = s + fmaf(s, kCut, rest[e]);
        sum[e] = fabsf(s) <= FLT_MAX ? t : s;
      }
      // rows to the CTA that finishes them (a lone CTA is no cluster: it keeps them by plain stores)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = quad * 16 + h * 8 + (lane >> 2), to = r / rows_each, rr = r - to * rows_each;
        float* const own = s_recv + ((int)rank * rows_each + rr) * kSN + 2 * (lane & 3);
        const uint32_t dst = S > 1 ? ptx::map_to_cta(ptx::smem_u32(own), (uint32_t)to) : 0u;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (S > 1) ptx::st_cluster_f2(dst + (uint32_t)g * 32u, sum[4 * g + 2 * h], sum[4 * g + 2 * h + 1]);
          else *reinterpret_cast<float2*>(own + 8 * g) = make_float2(sum[4 * g + 2 * h], sum[4 * g + 2 * h + 1]);
        }
      }
      __syncwarp();
      if (S == 1) {
        if (lane == 0) ptx::mbar_arrive(recv);
      } else if (lane < (S == 8 ? 2 : 1)) {   // a warp's sixteen rows are one CTA's, of eight CTAs two's
        ptx::mbar_arrive_remote(ptx::map_to_cta(recv, (uint32_t)(quad * 16 / rows_each + lane)));
      }
      okw = S > 1 ? ptx::warp_spin_cluster(recv, 0, abort_flag) : ptx::warp_spin(recv, 0, abort_flag);
    }
    if (okw) {
      float4 v[4];
      const float* mine = s_recv + (et >> 3) * kSN + 4 * (et & 7);
      auto add = [&](float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
      if (S == 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = *reinterpret_cast<const float4*>(mine + 16 * k * kSN);
      } else {   // parts in rank order
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int rr = (et >> 3) + 16 * k;
          v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (rr >= rows_each) continue;
          v[k] = *reinterpret_cast<const float4*>(mine + 16 * k * kSN);
          for (int q = 1; q < S; ++q) add(v[k], *reinterpret_cast<const float4*>(mine + (16 * k + q * rows_each) * kSN));
        }
        v[2] = v[3] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k].x = fmaf(v[k].x, sc.x, sh.x); v[k].y = fmaf(v[k].y, sc.y, sh.y);
        v[k].z = fmaf(v[k].z, sc.z, sh.z); v[k].w = fmaf(v[k].w, sc.w, sh.w);
      }
      if (p.residual) {
        if (p.res_f32) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (pix[k] >= 0) add(v[k], res32[k]);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (pix[k] >= 0) add(v[k], join4(res[k]));
        }
      }
      if (p.relu) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[k].x = !(v[k].x <= 0.0f) ? v[k].x : 0.0f; v[k].y = !(v[k].y <= 0.0f) ? v[k].y : 0.0f;
          v[k].z = !(v[k].z <= 0.0f) ? v[k].z : 0.0f; v[k].w = !(v[k].w <= 0.0f) ? v[k].w : 0.0f;
        }
      }
      if (p.out_f32) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (pix[k] >= 0) *reinterpret_cast<float4*>(static_cast<float*>(p.out) + pix[k] * p.ldo + n) = v[k];
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (pix[k] >= 0) {
            uint2 o[3];
            split4(v[k], o);
#pragma unroll
            for (int q = 0; q < 3; ++q)
              *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + q * p.out_plane + pix[k] * p.Kout + n) = o[q];
          }
      }
    } else if (lane == 0 && p.error_flag) {
      atomicCAS(p.error_flag, 0, (int)kErrWaitEpilogue);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  // Everything that was sent to this CTA has arrived, unless a wait gave up: then it stays until the others have left or given up too.
  if (S > 1 && s_abort) ptx::cluster_sync_all();
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------ weights and layouts ----
// Filter value w(n, t, c), t = tap, c = channel of a block, as three planes of swizzled 64 x 64 tiles.  STEM: the four
// "taps" are pairs of input rows, the 64 "channels" the 2 rows x 8 pixels x 4 channels of a window (see nchw_to_planes).
template <typename SrcT, bool STEM>
__global__ void pack_planes_kernel(const SrcT* __restrict__ src, long long sn, long long sc, long long stap, int Kout, int C, int CB, int taps,
                                   int n_tiles, uint8_t* __restrict__ dst) {
  const int kb_all = taps * CB;
  const long long total = (long long)n_tiles * kb_all * 64 * 64;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i & 63), row = (int)(i >> 6) & 63;
    const long long tile = i >> 12;
    const int kb = (int)(tile % kb_all), nt = (int)(tile / kb_all);
    const int n = nt * 64 + row, tap = kb / CB, c = (kb - tap * CB) * 64 + k;
    float v = 0.0f;
    if (STEM) {
      // element k of a window: 16-byte chunks alternate between the rows of the pair, two pixels of four channels each
      const int chunk = k >> 3, px = 2 * (chunk >> 1) + ((k & 7) >> 2), ch = k & 3;
      const int r = 2 * tap + (chunk & 1) - 1, s = px - 1;
      if (n < Kout && ch < 3 && r >= 0 && r < 7 && s >= 0) v = (float)src[n * sn + ch * sc + (long long)(r * 7 + s) * stap];
    } else if (n < Kout && c < C) {
      v = (float)src[n * sn + c * sc + tap * stap];
    }
    __nv_bfloat16 q[3];
    split3(v, q[0], q[1], q[2]);
    const uint32_t off = (uint32_t)row * 128u + ((((uint32_t)k >> 3) ^ ((uint32_t)row & 7u)) << 4) + ((uint32_t)k & 7u) * 2u;
#pragma unroll
    for (int pl = 0; pl < 3; ++pl)
      *reinterpret_cast<__nv_bfloat16*>(dst + ((size_t)(nt * 3 + pl) * kb_all + kb) * kBBytes + off) = q[pl];
  }
}

// fp32 tensor -> planes, four elements a thread.
__global__ void split_planes_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n4, long long plane) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    uint2 o[3];
    split4(__ldg(reinterpret_cast<const float4*>(src) + i), o);
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * plane + 4 * i) = o[q];
  }
}

// Stem input: NCHW images of three channels -> planes [3][N][row pair][pixel pair][row of the pair][2 pixels x 4 channels],
// four zero pixels in front of a row and at least four behind (the buffer is zeroed once; only pixels are written).  A
// stride-2 window of 8 pixels of both rows is then 128 contiguous bytes, 32 bytes from one output pixel's to the next.
template <typename SrcT>
__global__ void nchw_to_planes_kernel(const SrcT* __restrict__ src, __nv_bfloat16* __restrict__ dst, int N, int H, int W, int pair_elems,
                                      long long plane) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const long long total = (long long)N * H * W;
  const int H2 = (H + 1) / 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % W);
    const long long t = i / W;
    const int y = (int)(t % H);
    const long long n = t / H;
    const SrcT* s = src + (size_t)n * 3 * H * W + (size_t)y * W + x;
    float4 v = make_float4((float)s[0], (float)s[(size_t)H * W], (float)s[2 * (size_t)H * W], 0.0f);
    uint2 o[3];
    split4(v, o);
    const int px = x + 4;
    const long long at = ((long long)n * H2 + (y >> 1)) * pair_elems + (px >> 1) * 16 + (y & 1) * 8 + (px & 1) * 4;
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * plane + at) = o[q];
  }
}

// Max-pool over a -inf padded map, planes out (the maximum of fp32 values; NaN propagates).  The input is planes, or plain fp32 where
// the convolution before it has no other reader: that map is then 4 bytes an element instead of 6, its epilogue splits nothing, and of
// the nine values under a window only the largest is split.  K: the window's size, 0 for any.
// ResNet-18 8x224: the stem 38 -> 36 us, the pool 21 -> 14.5 (nine loads of planes, joined one after another); 256x256 10.5 -> 5.
template <bool F32IN, int K>
__global__ void maxpool_planes_kernel(const void* __restrict__ src, __nv_bfloat16* __restrict__ dst, int N, int H, int W, int C, int OH,
                                      int OW, int k_any, int stride, int pad, long long in_plane, long long out_plane) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const int k = K ? K : k_any, cv = C / 4;
  const unsigned total = (unsigned)N * OH * OW * cv;
  auto load = [&](long long at) {
    if constexpr (F32IN) {
      return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(src) + at));
    } else {
      uint2 w[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) w[q] = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(src) + q * in_plane + at));
      return join4(w);
    }
  };
  auto up = [](float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
  };
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    unsigned t = i / (unsigned)cv;
    const int c = (int)(i - t * cv) * 4;
    const unsigned t2 = t / (unsigned)OW;
    const int ox = (int)(t - t2 * OW);
    const int n = (int)(t2 / (unsigned)OH), oy = (int)(t2 - (unsigned)n * OH);
    const float4 none = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    float4 m = none;
    const int y0 = oy * stride - pad, x0 = ox * stride - pad;
    if constexpr (K != 0) {   // all loads of a window in flight
      float4 v[K * K];
#pragma unroll
      for (int r = 0; r < K; ++r)
#pragma unroll
        for (int s = 0; s < K; ++s)
          v[r * K + s] = (unsigned)(y0 + r) < (unsigned)H && (unsigned)(x0 + s) < (unsigned)W
                             ? load((((long long)n * H + y0 + r) * W + x0 + s) * C + c) : none;
#pragma unroll
      for (int e = 0; e < K * K; ++e) m = make_float4(up(m.x, v[e].x), up(m.y, v[e].y), up(m.z, v[e].z), up(m.w, v[e].w));
    } else {
      for (int r = 0; r < k; ++r)
        for (int s = 0; s < k; ++s)
          if ((unsigned)(y0 + r) < (unsigned)H && (unsigned)(x0 + s) < (unsigned)W) {
            const float4 v = load((((long long)n * H + y0 + r) * W + x0 + s) * C + c);
            m = make_float4(up(m.x, v.x), up(m.y, v.y), up(m.z, v.z), up(m.w, v.w));
          }
    }
    uint2 o[3];
    split4(m, o);
    const long long at = (((long long)n * OH + oy) * OW + ox) * C + c;
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * out_plane + at) = o[q];
  }
}

// Global average pool, planes in and out: eight adjacent lanes share one (image, four channels) and add their sums by shuffles.
__global__ void avgpool_planes_kernel(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, int N, int HW, int C,
                                      long long in_plane, long long out_plane) {
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  const int cv = C / 4;
  const long long total = (long long)N * cv * 8;
  for (long long i0 = blockIdx.x * (long long)blockDim.x; i0 < total; i0 += (long long)gridDim.x * blockDim.x) {
    const long long i = i0 + threadIdx.x;
    const bool live = i < total;
    const int slice = (int)(i & 7);
    const long long g = live ? i >> 3 : 0;
    const int c = (int)(g % cv) * 4;
    const long long n = g / cv;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live)
      for (int px = slice; px < HW; px += 8) {
        uint2 w[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) w[q] = __ldg(reinterpret_cast<const uint2*>(src + q * in_plane + (n * HW + px) * C + c));
        const float4 v = join4(w);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, d);
      s.y += __shfl_xor_sync(0xffffffffu, s.y, d);
      s.z += __shfl_xor_sync(0xffffffffu, s.z, d);
      s.w += __shfl_xor_sync(0xffffffffu, s.w, d);
    }
    if (live && slice == 0) {
      const float inv = (float)HW;
      uint2 o[3];
      split4(make_float4(s.x / inv, s.y / inv, s.z / inv, s.w / inv), o);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * out_plane + n * C + c) = o[q];
    }
  }
}

PFN_cuTensorMapEncodeTiled_v12000 f32_get_encode() {
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

int grid_of(long long total, int threads) {
  const long long b = (total + threads - 1) / threads, cap = 148LL * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

size_t packed_planes_bytes(int Kout, int C, int taps) { return (size_t)((Kout + 63) / 64) * 3 * taps * ((C + 63) / 64) * kBBytes; }

cudaError_t launch_pack_planes(const void* src, DType src_dt, long long sn, long long sc, long long stap, int Kout, int C, int taps, bool stem,
                               void* dst, cudaStream_t stream) {
  const int CB = stem ? 1 : (C + 63) / 64, nt = (Kout + 63) / 64, tp = stem ? 4 : taps;
  const int grid = grid_of((long long)nt * tp * CB * 4096, 256);
  uint8_t* d = static_cast<uint8_t*>(dst);
#define NNCV_PK(T_) \
  if (stem) pack_planes_kernel<T_, true><<<grid, 256, 0, stream>>>(static_cast<const T_*>(src), sn, sc, stap, Kout, C, CB, tp, nt, d); \
  else pack_planes_kernel<T_, false><<<grid, 256, 0, stream>>>(static_cast<const T_*>(src), sn, sc, stap, Kout, C, CB, tp, nt, d)
  if (src_dt == kF32) { NNCV_PK(float); }
  else if (src_dt == kF16) { NNCV_PK(__half); }
  else { NNCV_PK(__nv_bfloat16); }
#undef NNCV_PK
  return cudaGetLastError();
}

cudaError_t launch_split_planes(const float* src, void* dst, long long n, cudaStream_t stream) {
  if (n % 4 != 0) return cudaErrorInvalidValue;
  return launch_pdl(split_planes_kernel, dim3(grid_of(n / 4, 256)), dim3(256), 0, stream, src, static_cast<__nv_bfloat16*>(dst), n / 4, n);
}

int stem_planes_pair_elems(int W) { return ((W + 8 + 1) & ~1) * 8; }   // pixels of a padded row, even, x 2 rows x 4 channels
long long stem_planes_elems(int N, int H, int W) { return (long long)N * ((H + 1) / 2) * stem_planes_pair_elems(W); }

cudaError_t launch_nchw_to_planes(const void* src, DType src_dt, void* dst, int N, int H, int W, cudaStream_t stream) {
  const dim3 grid(grid_of((long long)N * H * W, 256));
  const int pe = stem_planes_pair_elems(W);
  const long long plane = stem_planes_elems(N, H, W);
  __nv_bfloat16* d = static_cast<__nv_bfloat16*>(dst);
  if (src_dt == kF32) return launch_pdl(nchw_to_planes_kernel<float>, grid, dim3(256), 0, stream, static_cast<const float*>(src), d, N, H, W, pe, plane);
  if (src_dt == kF16) return launch_pdl(nchw_to_planes_kernel<__half>, grid, dim3(256), 0, stream, static_cast<const __half*>(src), d, N, H, W, pe, plane);
  return launch_pdl(nchw_to_planes_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(src), d, N, H, W, pe, plane);
}

cudaError_t launch_maxpool_planes(const void* src, int src_f32, void* dst, int N, int H, int W, int C, int k, int stride, int pad,
                                  cudaStream_t stream) {
  const int OH = (H + 2 * pad - k) / stride + 1, OW = (W + 2 * pad - k) / stride + 1;
  const long long total = (long long)N * OH * OW * (C / 4);
  if (C % 4 != 0 || total >= (1LL << 31) - (1LL << 21)) return cudaErrorInvalidValue;
  auto go = [&](auto kernel) {
    return launch_pdl(kernel, dim3(grid_of(total, 256)), dim3(256), 0, stream, src, static_cast<__nv_bfloat16*>(dst), N, H, W, C, OH, OW, k, stride,
                      pad, (long long)N * H * W * C, (long long)N * OH * OW * C);
  };
  if (src_f32) return k == 3 ? go(maxpool_planes_kernel<true, 3>) : go(maxpool_planes_kernel<true, 0>);
  return go(maxpool_planes_kernel<false, 0>);
}

cudaError_t launch_avgpool_planes(const void* src, void* dst, int N, int HW, int C, cudaStream_t stream) {
  if (C % 4 != 0) return cudaErrorInvalidValue;
  return launch_pdl(avgpool_planes_kernel, dim3(grid_of((long long)N * (C / 4) * 8, 256)), dim3(256), 0, stream,
                    static_cast<const __nv_bfloat16*>(src), static_cast<__nv_bfloat16*>(dst), N, HW, C, (long long)N * HW * C, (long long)N * C);
}

bool conv_f32_supported(int C, int Kout, int tw_stride) { return C % 8 == 0 && Kout % 4 == 0 && tw_stride <= 256; }

// A pointwise convolution is a matrix of N * H * W rows: no tile straddles an image's border (a 7 x 7 map fills 49 of the 64 slots of
// its half tile).
static bool as_matrix(ConvF32Args* a) {
  if (a->stem || a->R != 1 || a->S != 1 || a->stride != 1 || a->pad != 0 || (long long)a->N * a->H * a->W >= (1LL << 30)) return false;
  a->W = a->OW = a->N * a->H * a->W;
  a->N = a->H = a->OH = 1;
  return true;
}
// The pixels of a tile: tn images x th rows x tw columns.  Row r of the tile is column r % mp of row r / mp, rows_img rows an image.
// Halo tiles (filters of stride 1 and more than one row): one box brings the pixels of a block of 64 channels under a whole column of the
// filter, and filter row r reads it from its row r on.  mp is a multiple of 8, so that every view is whole groups of eight rows of 128
// bytes, as the operand's layout has them.  (One box for all taps, 180 pixels for 128 with eight rows 1280 bytes apart, was no faster:
// 57.2 us and 57.3 for 512 -> 512 on 7x7 by one CTA a tile.)  The tile of the fewest, then of the least to copy.
struct F32Tile {
  int tw = 0, th = 0, tn = 1, mp = 0, rows_img = 0;
  int box_h = 0, box_n = 1;
  long long tiles = 0;
  int plane() const { return mp * box_h * box_n * 128; }
};
static long long tiles_of(const F32Tile& t, const ConvF32Args& a) {
  return (long long)((a.OW + t.tw - 1) / t.tw) * ((a.OH + t.th - 1) / t.th) * ((a.N + t.tn - 1) / t.tn);
}
constexpr size_t kHaloSmem = 226 * 1024, kHaloFixed = 1024 + kTileBytes, kHaloBlock = 3 * kBBytes;   // all; neither boxes nor weights; a block of weights
static bool halo_fits(const F32Tile& t) {   // two boxes and three blocks of weights
  return t.box_h <= 256 && kHaloFixed + 2 * 3 * (size_t)t.plane() + 3 * kHaloBlock <= kHaloSmem;
}
static bool halo_tile(const ConvF32Args& a, F32Tile* best) {
  constexpr int rows = 128;
  const int R = a.stem ? 4 : a.R;
  if (!a.stem && (a.stride != 1 || R == 1)) return false;
  bool found = false;
  auto offer = [&](F32Tile t) {
    t.tiles = tiles_of(t, a);
    if (!halo_fits(t) || (found && (t.tiles > best->tiles || (t.tiles == best->tiles && t.plane() >= best->plane())))) return;
    *best = t;
    found = true;
  };
  for (int mp : {8, 16, 32, 64, 128, (a.OW + 7) & ~7}) {
    if (mp > rows || mp >= a.OW + 8) continue;
    F32Tile t;
    t.mp = mp;
    t.tw = mp < a.OW ? mp : a.OW;
    t.th = a.OH < rows / mp ? a.OH : rows / mp;
    t.rows_img = 256;
    t.box_h = t.th + R - 1;
    offer(t);
    // whole images one below the other: the row above an image is zero and serves the one before as the row below
    const int images = (rows / mp + 1) / (a.OH + 1);
    if (!a.stem && R == 3 && a.pad == 1 && images > 1) {
      t.th = a.OH;
      t.rows_img = t.box_h = a.OH + 1;
      t.tn = images;
      t.box_n = images + 1;
      offer(t);
    }
  }
  return found;
}
static F32Tile f32_tile(const ConvF32Args& a, bool matrix, int bn) {
  F32Tile t;
  if (bn == kSN) {
    conv_small_tile(a.N, a.OH, a.OW, &t.tw, &t.th, &t.tn);
  } else if (matrix) {
    t.tw = 128;
    t.th = 1;
  } else {
    tconv_tile(a.N, a.OH, a.OW, &t.tw, &t.th, &t.tn);
  }
  t.mp = t.tw;
  t.rows_img = t.th;
  t.tiles = tiles_of(t, a);
  return t;
}
// Clusters of s CTAs with tiles of bn columns that run at once.  Fewer fit the GPU than its SMs would hold (they do not cross GPC
// borders), so the runtime is asked.
static int clusters_that_fit(int bn, int s, int sms) {
  static const ClusterFit small = cluster_fit(conv_f32_small_kernel, kSThreads, kSSmem, sms);
  static const ClusterFit wide = cluster_fit(conv_f32_kernel<64, false>, kThreads, Ring<64>::kSmem, sms);
  static const ClusterFit wider = cluster_fit(conv_f32_kernel<128, false>, kThreads, Ring<128>::kSmem, sms);
  return bn == kSN ? small.of[s] : bn == 64 ? wide.of[s] : wider.of[s];
}

// Tile width and the CTAs of a cluster that share a tile's reduction: the pair with the least rounds x time, in clocks.  A block of 64
// channels, as measured by one CTA a tile: 560 on 64 x 32 tiles, on 128 x 64 tiles 1220 with halo tiles and 1450 without (which fill
// better on narrow maps), on 128 x 128 tiles 1920; without boxes the copies of all SMs together allow 1565 and 2087.  A tile's beginning
// and end 9000, 5560 and 11100 (the widest is finished in two passes), a launch of wide tiles 6700 more, a split 2700 or 2000: fitted to
// 190 layers of 1 to 32 images (ResNet-18's and ResNet-50's, and random ones), each at every tile and split, before the first planes had a
// ring and 128 columns one issuing warp; of 250 such layers of 1 to 64 images since, the choice takes 0.2 % more than the fastest.  On
// either side of the lines, us: 14x14x256 -> 256 3x3 of one image 64 x 32 10.4, wide 11.4; 7x7x512 -> 512 of one 12.6 and 15.1; 28x28x128
// of eight 128 x 64 22.0, 128 x 128 23.9, 64 x 32 39.8.  Clusters of sixteen were slower at batch 1 than clusters of eight (21 us against
// 15 for 256 channels on 16 x 16 pixels).
void conv_f32_choose(ConvF32Args* args) {
  if (args->chosen) return;
  args->chosen = 1;
  ConvF32Args a = *args;
  const bool matrix = as_matrix(&a);
  const int kb_all = (a.stem ? 4 : a.R * a.S) * (a.stem ? 1 : (a.C + 63) / 64), stride = a.stem ? 1 : a.stride, sms = a.sm_count > 0 ? a.sm_count : 148;
  double best = 1e30;
  F32Tile box;
  const bool boxes = args->halo >= 0 && halo_tile(a, &box);
  for (int forced = 2; forced >= 0 && best == 1e30; --forced)   // what was asked for, the tile alone, neither
    for (int b : {64, 128, kSN}) {
      if ((b == 128 && a.Kout <= 64) || (forced >= 1 && a.bn != 0 && b != a.bn)) continue;
      for (int halo = 0; halo < (b == 64 && boxes ? 2 : 1); ++halo) {
        if (!halo && b == 64 && boxes && a.halo > 0) continue;
        const F32Tile t = halo ? box : f32_tile(a, matrix, b);
        if (b == kSN && (t.tw > t.th ? t.tw : t.th) * stride > 256) continue;
        const long long tiles = t.tiles * ((a.Kout + b - 1) / b);
        for (int s = 1; s <= 8 && s <= kb_all; s *= 2) {
          if (forced == 2 && a.splits != 0 && s != a.splits) continue;
          const int slots = clusters_that_fit(b, s, sms), blocks = (kb_all + s - 1) / s;
          const double rounds = (double)((tiles + slots - 1) / slots), load = (double)(std::min<long long>(tiles, slots) * s) / sms;
          const double block = b == kSN ? 560.0 : halo ? 1220.0 : b == 64 ? std::max(1450.0, 1565.0 * load) : std::max(1920.0, 2087.0 * load);
          const double cost = b == kSN ? rounds * (blocks * block + 9000.0 + (s > 1 ? 2700.0 : 0.0))
                                       : rounds * (blocks * block + (b == 64 ? 5560.0 : 11100.0)) + 6700.0 + (s > 1 ? 2000.0 : 0.0);
          if (cost < best) { best = cost; args->bn = b; args->splits = s; args->halo = halo ? 1 : -1; }
        }
      }
    }
}

template <typename Kern>
static cudaError_t launch_f32(Kern kern, int threads, size_t smem, int ctas, const CUtensorMap& tm, const F32Params& p, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.splits > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, tm, p);
}

cudaError_t launch_conv_f32(const ConvF32Args& args, cudaStream_t stream) {
  ConvF32Args a = args;
  const bool stem = a.stem != 0;
  const bool matrix = as_matrix(&a);
  F32Params p{};
  p.wpack = static_cast<const uint8_t*>(a.wpack);
  p.scale = a.scale; p.shift = a.shift;
  p.residual = a.residual; p.res_f32 = a.res_f32;
  p.out = a.out; p.out_f32 = a.out_f32; p.relu = a.relu; p.error_flag = a.error_flag;
  p.Kout = a.Kout; p.OH = a.OH; p.OW = a.OW; p.NB = a.N;
  p.CB = stem ? 1 : (a.C + 63) / 64;
  p.taps = stem ? 4 : a.R * a.S;
  p.S = stem ? 1 : a.S;
  p.stride = stem ? 1 : a.stride;
  p.pad_x = stem ? 0 : a.pad;
  p.pad_y = stem ? 2 : a.pad;
  p.ldo = a.ldo;
  const long long pixels = (long long)a.N * a.OH * a.OW;
  if (pixels > 0x7fffffffLL) return cudaErrorInvalidValue;
  p.res_plane = p.out_plane = pixels * a.Kout;
  const F32Tile wide = f32_tile(a, matrix, 64);
  if (!conv_f32_supported(stem ? 64 : a.C, a.Kout, (wide.tw > wide.th ? wide.tw : wide.th) * p.stride)) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(a.in) & 15) || (reinterpret_cast<uintptr_t>(a.out) & 15) || (reinterpret_cast<uintptr_t>(a.residual) & (a.res_f32 ? 15 : 7)) ||
      ((a.out_f32 || a.res_f32) && a.ldo % 4 != 0))
    return cudaErrorMisalignedAddress;
  conv_f32_choose(&a);
  const int bn = a.bn, sms = a.sm_count > 0 ? a.sm_count : 148;
  F32Tile t = f32_tile(a, matrix, bn);
  if (a.halo > 0 && !halo_tile(a, &t)) return cudaErrorInvalidValue;
  p.splits = a.splits;
  p.tw = t.tw; p.th = t.th; p.tn = t.tn; p.mp = t.mp; p.rows_img = t.rows_img;
  p.tiles_x = (a.OW + t.tw - 1) / t.tw; p.tiles_y = (a.OH + t.th - 1) / t.th;
  p.n_tiles = (a.Kout + bn - 1) / bn;
  const long long items = t.tiles * p.n_tiles;
  if (items <= 0 || items * a.splits > 0x7fffffffLL) return cudaErrorInvalidValue;
  p.items = (int)items;
  p.div_tx = epi::fast_div((uint32_t)p.tiles_x); p.div_ty = epi::fast_div((uint32_t)p.tiles_y); p.div_nt = epi::fast_div((uint32_t)p.n_tiles);
  p.div_mp = epi::fast_div((uint32_t)t.mp); p.div_ri = epi::fast_div((uint32_t)t.rows_img);
  size_t smem = bn == kSN ? kSSmem : bn == 64 ? Ring<64>::kSmem : Ring<128>::kSmem;
  if (a.halo > 0) {
    // two boxes, weights in the rest
    p.R = stem ? 4 : a.R;
    p.a_plane = t.plane();
    p.b_stages = (int)std::min((kHaloSmem - kHaloFixed - 3 * (size_t)p.a_plane * kBoxes) / kHaloBlock, (size_t)kHaloB);
    smem = kHaloFixed + 3 * (size_t)p.a_plane * kBoxes + kHaloBlock * p.b_stages;
  }

  auto enc = f32_get_encode();
  if (!enc) return cudaErrorNotSupported;
  // [3][N][H][W][C] planes; the stem's [3][N][row pairs][windows][64] has windows that overlap
  cuuint64_t gdim[5], gstr[4];
  if (stem) {
    const cuuint64_t H2 = (cuuint64_t)(a.H + 1) / 2, pair = (cuuint64_t)stem_planes_pair_elems(a.W) * 2;
    gdim[0] = 64; gdim[1] = (cuuint64_t)a.OW; gdim[2] = H2; gdim[3] = (cuuint64_t)a.N; gdim[4] = 3;
    gstr[0] = 32; gstr[1] = pair; gstr[2] = H2 * pair; gstr[3] = (cuuint64_t)a.N * H2 * pair;
  } else {
    const cuuint64_t px = (cuuint64_t)a.C * 2;
    gdim[0] = (cuuint64_t)a.C; gdim[1] = (cuuint64_t)a.W; gdim[2] = (cuuint64_t)a.H; gdim[3] = (cuuint64_t)a.N; gdim[4] = 3;
    gstr[0] = px; gstr[1] = px * a.W; gstr[2] = px * a.W * a.H; gstr[3] = px * a.W * a.H * a.N;
  }
  cuuint32_t box[5] = {64, (cuuint32_t)(t.tw * p.stride), (cuuint32_t)(t.th * p.stride), (cuuint32_t)t.tn, 1};
  if (a.halo > 0) { box[1] = (cuuint32_t)t.mp; box[2] = (cuuint32_t)t.box_h; box[3] = (cuuint32_t)t.box_n; }
  cuuint32_t estr[5] = {1, (cuuint32_t)p.stride, (cuuint32_t)p.stride, 1, 1};
  CUtensorMap tm;
  if (enc(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(a.in), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  if (bn == kSN) {
    return launch_f32(conv_f32_small_kernel, kSThreads, smem, p.items * p.splits, tm, p, stream);
  }
  const int slots = clusters_that_fit(bn, p.splits, sms), ctas = (p.items < slots ? p.items : slots) * p.splits;
  if (a.halo > 0) return launch_f32(conv_f32_kernel<64, true>, kThreads, smem, ctas, tm, p, stream);
  return bn == 64 ? launch_f32(conv_f32_kernel<64, false>, kThreads, smem, ctas, tm, p, stream)
                  : launch_f32(conv_f32_kernel<128, false>, kThreads, smem, ctas, tm, p, stream);
}

}  // namespace nncv_b200
