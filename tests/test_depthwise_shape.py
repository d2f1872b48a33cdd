"""The choice of tile and block of the depthwise kernel (csrc/depthwise_shape.h), on the CPU."""
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nncv_b200", "csrc")
SMS = 148

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "depthwise_shape.h"
using namespace nncv_b200;
struct In { int v[7]; };
int main() {
  std::vector<In> all;
  In i;
  while (scanf("%d %d %d %d %d %d %d", i.v, i.v + 1, i.v + 2, i.v + 3, i.v + 4, i.v + 5, i.v + 6) == 7) all.push_back(i);
  std::vector<dw::Shape> out(all.size());
  for (size_t k = 0; k < all.size(); ++k) {
    const int* a = all[k].v;
    out[k] = dw::choose(a[0], a[1], a[2], a[3], a[4], a[5], a[6], 148);
  }
  // what is kept is what was chosen, in any order and in several threads
  std::vector<int> wrong(4, 0);
  std::vector<std::thread> threads;
  for (int t = 0; t < 4; ++t)
    threads.emplace_back([&, t] {
      unsigned r = t + 1;
      for (size_t k = 0; k < 4 * all.size(); ++k) {
        r = r * 1664525u + 1013904223u;
        const size_t j = (r >> 8) % all.size();
        const int* a = all[j].v;
        for (int twice = 0; twice < 2; ++twice) {
          const dw::Shape s = dw::shape_of(a[0], a[1], a[2], a[3], a[4], a[5], a[6], 148);
          const dw::Shape& c = out[j];
          wrong[t] += s.cbv != c.cbv || s.tw != c.tw || s.px != c.px || s.kp != c.kp || s.threads != c.threads || s.stages != c.stages ||
                      s.per_sm != c.per_sm || s.smem != c.smem;
        }
      }
    });
  for (auto& t : threads) t.join();
  printf("%d\n", wrong[0] + wrong[1] + wrong[2] + wrong[3]);
  for (const dw::Shape& s : out) printf("%d %d %d %d %d %d %d %zu\n", s.cbv, s.tw, s.px, s.kp, s.threads, s.stages, s.per_sm, s.smem);
}
"""


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", "t.cpp", "-o", "t"], cwd=d, check=True)

    def run(layers):
        """layers: (n, c, h, w, k, stride, bytes of an element) with pad k // 2 -> the choices, as dicts."""
        text = "".join(f"{n} {c} {(h - 1) // s + 1} {(w - 1) // s + 1} {k} {s} {es}\n" for n, c, h, w, k, s, es in layers)
        lines = subprocess.run([str(d / "t")], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
        assert int(lines[0]) == 0, "a kept choice differs from the chosen one"
        names = ("cbv", "tw", "px", "kp", "threads", "stages", "per_sm", "smem")
        return [dict(zip(names, map(int, line.split()))) for line in lines[1:]]

    return run


def _layers(count):
    rng = random.Random(5)
    out = []
    for _ in range(count):
        es = rng.choice((2, 4))
        c = (16 // es) * rng.choice((2, 3, 5, 7, 11, 16, 30, 33, 71, 128))
        out.append((rng.choice((1, 2, 9, 64, 256)), c, rng.randint(1, 130), rng.choice((1, 2, 3, 4, 5, 7, 14, 27, 56, 112, 300)), rng.choice((3, 5)),
                    rng.choice((1, 2)), es))
    return out


def test_every_choice_can_be_launched(choose):
    layers = _layers(600)
    for (n, c, h, w, k, stride, es), d in zip(layers, choose(layers)):
        most, regs = (256, {3: 3, 5: 2}[k]) if es == 4 else (128, {(3, 2): 4, (5, 2): 3, (3, 1): 6, (5, 1): 4}[(k, d["px"])])
        th = 8 if es == 4 else d["kp"]
        assert 2 <= d["cbv"] <= min(32, c * es // 16) and d["tw"] >= 1 and d["tw"] % d["px"] == 0
        assert (d["px"], d["kp"]) in {(1, 4)} if es == 4 else (d["px"], d["kp"]) in {(1, 8), (2, 8 if stride == 1 else 4)}
        # every strip of the tile has a thread
        assert d["threads"] % 32 == 0 and d["tw"] * (th // d["kp"]) * d["cbv"] * (4 // es) // d["px"] <= d["threads"] <= most
        iw, ih = (d["tw"] - 1) * stride + k, (th - 1) * stride + k
        stage = (iw * ih * d["cbv"] * 16 + 127) // 128 * 128
        assert iw <= 256 and 2 <= d["stages"] <= 3
        assert d["smem"] == d["stages"] * stage + (k * k + (1 if es == 2 else 2)) * d["cbv"] * (16 // es) * 4 <= 227 * 1024
        # the blocks an SM that the grid is made for fit it: 228 KB, 1 KB and the kernel's own variables a block
        two = d["smem"] - (d["stages"] - 2) * stage
        assert d["per_sm"] == min(regs * most // d["threads"], 16, 228 * 1024 // (two + 1024 + 128)) >= 1
        assert d["per_sm"] * (d["smem"] + 1024) <= 228 * 1024


@pytest.mark.parametrize("layer", [(54, 592, 17, 5, 3, 2, 4), (27, 144, 37, 4, 5, 2, 4), (8, 384, 19, 79, 3, 2, 4)])
def test_fp32_blocks_share_an_sm(choose, layer):
    """With the SM counted smaller than it is these layers ran one block an SM and took up to a quarter longer."""
    assert choose([layer])[0]["per_sm"] >= 2


@pytest.mark.parametrize("layer", [(9, 40, 19, 5, 5, 1, 2), (5, 40, 30, 6, 5, 2, 2), (4, 40, 13, 3, 5, 2, 2), (43, 24, 7, 6, 5, 1, 2), (7, 40, 40, 10, 5, 1, 2)])
def test_one_round_fetches_the_filter(choose, layer):
    """Layers of one tile a block are bound by latency; in two rounds of loads they took up to a quarter longer."""
    d = choose([layer])[0]
    assert d["cbv"] * 8 <= d["threads"]
