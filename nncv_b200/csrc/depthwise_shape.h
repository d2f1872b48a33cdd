// Tile, outputs of a thread and block of the depthwise kernel (depthwise.cu) for a layer.  Host code without CUDA.
#pragma once

#include <algorithm>
#include <cstddef>

namespace nncv_b200 {
namespace dw {

// Threads of a block at most, and blocks of that size an SM (by registers; the kernel's launch bounds).  es: bytes of an element,
// px: output columns of a thread.
constexpr int max_threads(int es) { return es == 4 ? 256 : 128; }
constexpr int ctas(int es, int ks, int px) { return es == 4 ? (ks == 3 ? 3 : 2) : px == 2 ? (ks == 3 ? 4 : 3) : (ks == 3 ? 6 : 4); }
constexpr int kMaxStages = 3;
// Shared memory of an SM, and what a block takes of it besides its own: 1 KB of the system's and the kernel's static variables.
constexpr size_t kSmSmem = 228 * 1024, kBlockSmem = 1024 + 128;

// cbv: 16-byte channel vectors of a block's chunk, tw: columns of a tile, px x kp: outputs of a thread.
struct Shape { int cbv, tw, px, kp, threads, stages, per_sm; size_t smem; };

// 16-bit types: two columns x eight rows a thread at stride 1 (two x four at stride 2, where a patch has twice the rows) read and
// convert each input value for two columns at once; one column x eight rows leaves none of an odd, narrow map's threads idle and
// needs fewer registers.  fp32, whose rows are twice as long and need no conversion: four rows of one column.  A tile is any split of
// columns and whole 16-byte channel vectors that a block's threads cover.
//
// The least modelled cost counts, in instructions of a thread times threads, of the busiest SM:
//   - multiply-adds and shared-memory reads of its tiles, and six warps' worth of latency for each (shared by the blocks beside one
//     another);
//   - halo columns, and rows of a patch shorter than 256 (and more so 128) bytes;
//   - a round of filter loads, 300 + 4 R^2, for every `threads` channels of the chunk: a block may have more threads than strips so
//     that one round does (12x4x88, 5x5 stride 2 fp16: 32 threads 6.7 us, 128 4.5);
//   - 1100 for the barrier and the wait of each tile.
// The weights are fitted to 504 layers of one to 256 images (random ones, and a mobile network's), fp16, bf16 and fp32, every tile
// timed: the choice takes 4.3 % (16 bits) and 4.8 % (fp32) more than the best tile.  A rule without the loads' and the barrier's share
// took 8.8 % more in 16 bits, one that weighed idle threads alone 13 % more in fp32, and for one layer in ten they were slower than 256
// threads of one column x eight rows throughout.
// Batch 256 fp16, us, one column, two columns: 240 channels 5x5 on 14x14 37.6 34.3, 576 on 7x7 24.3 28.7, 88 3x3 on 28x28 27.2 25.3, 16
// 3x3 stride 2 112 -> 56 32.6 43.6, 72 3x3 stride 2 56 -> 28 41.9 29.9.
inline Shape choose(int N, int C, int OH, int OW, int R, int stride, int es, int sms) {
  const int V = 16 / es, cv = C / V;
  const size_t wvec = (size_t)(R * R + (es == 2 ? 1 : 2)) * V * sizeof(float);   // filter and shift (scale) of a channel vector
  Shape best{};
  double least = 1e30;
  for (int px = es == 2 ? 2 : 1; px >= 1; --px) {
    const int kp = es == 4 || (px == 2 && stride == 2) ? 4 : 8, th = es == 4 ? 8 : kp, ih = (th - 1) * stride + R;
    const int most = max_threads(es), slots = most * px / 2;   // 16-byte vectors of a tile
    const int by_regs = most * ctas(es, R, px), tiles_y = (OH + th - 1) / th;
    const double loads = (double)((kp - 1) * stride + R) * ((px - 1) * stride + R);
    const double work = ((2.0 * R * R + 1.0) * kp * px + 2.0 * loads) * (px == 2 ? 1.1 : 1.0);
    for (int v = std::min(32, cv); v >= 2; --v) {        // ties go to the wider chunk (longer contiguous runs in memory)
      const int widest = slots / v / px * px, fewest = (OW + widest - 1) / widest, chunks = (cv + v - 1) / v;
      const double rows = (v < 16 ? 0.64 + 0.0225 * v : 1.0) * (v < 8 ? 0.44 + 0.07 * v : 1.0);
      for (int tiles = fewest, last = 0; tiles <= fewest + 2; ++tiles) {
        const int t = ((OW + tiles - 1) / tiles + px - 1) / px * px, iw = (t - 1) * stride + R;
        if (iw > 256 || t == last) continue;
        last = t;
        const size_t stage = ((size_t)iw * ih * v * 16 + 127) & ~(size_t)127;
        if (2 * stage + v * wvec > 200 * 1024) continue;
        const long long all = (long long)N * tiles_y * ((OW + t - 1) / t);
        const double turns = (double)((all * chunks + sms - 1) / sms);   // tiles of the busiest SM
        const int strips = (t * v * 2 / px + 31) & ~31;
        for (int q = 0; q < 3; ++q) {
          const int threads = q == 0 ? strips : q * most / 2;
          if (q > 0 && threads <= strips) continue;
          const auto fit = [&](int stages) {
            return std::min(std::min(by_regs / threads, 16), (int)(kSmSmem / (stages * stage + v * wvec + kBlockSmem)));
          };
          const int per_sm = fit(2);
          if (per_sm < 1) continue;
          const long long gx = std::max(1LL, std::min((long long)sms * per_sm / chunks, all));
          const int rounds = (V * v + threads - 1) / threads;
          const double cost = work * (strips + 6.0 * 32.0 / std::min((double)per_sm, turns)) * turns / (rows * (0.15 + 0.85 * t * stride / iw)) +
                              128.0 * (rounds * (300.0 + 4.0 * R * R) + 1100.0 * (double)((all + gx - 1) / gx));
          if (cost < least * (1.0 - 1e-9)) {
            least = cost;
            // a third stage where it costs no block of an SM (fp32, of a large patch, 56x56x72 at stride 2: 83 us with it, 79 without)
            const int stages = fit(3) == per_sm && (es == 2 || per_sm > 1) ? kMaxStages : 2;
            best = Shape{v, t, px, kp, threads, stages, per_sm, stages * stage + v * wvec};
          }
        }
      }
    }
  }
  return best;
}

// The same, kept for the layers that a thread asks for in turn: choosing takes longer than a launch.  Four places for the layers of
// one hash value, so that a network's few dozen do not push one another out.
inline Shape shape_of(int N, int C, int OH, int OW, int R, int stride, int es, int sms) {
  struct Kept { int key[8]; Shape shape; };
  struct Row { Kept way[4]; unsigned next; };
  thread_local Row table[32] = {};
  const int key[8] = {N, C, OH, OW, R, stride, es, sms};
  unsigned h = 2166136261u;
  for (int k : key) h = (h ^ (unsigned)k) * 16777619u;
  Row& row = table[(h >> 16) % 32u];
  for (const Kept& k : row.way)
    if (std::equal(key, key + 8, k.key)) return k.shape;
  Kept& k = row.way[row.next++ % 4u];
  k.shape = choose(N, C, OH, OW, R, stride, es, sms);
  std::copy(key, key + 8, k.key);
  return k.shape;
}

}  // namespace dw
}  // namespace nncv_b200
