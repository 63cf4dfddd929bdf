"""The device words of a resident run (epi_b200/csrc/epi_run_words.h), on the
host: the header is compiled into a small model of the run's blocks, and every
interleaving of their reads, writes and barrier arrivals is walked."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "epi_b200" / "csrc"


def build(tmp_path, source):
    src, exe = tmp_path / "model.cpp", tmp_path / "model"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(CSRC), "-o", str(exe), str(src)],
                   check=True)
    return exe


# A block of k_resident: [rebuild: barrier, block 0 clears the word, barrier],
# commit (may raise the word), barrier, read the word. Exits 0 when in every
# interleaving all blocks decide alike and as the steps raised.
FLAGS = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
#include "epi_run_words.h"
struct OneWord {  // every step raises and reads the same word
  int32_t *gate, *words;
  int32_t* raised_by(int32_t) const { return gate; }
  int32_t* read_by(int32_t) const { return gate; }
  void hand_on(int32_t) const {}
};
enum { COMMIT, READ, REBUILD, CLEAR, REBUILT, OUT };
struct Block { int at, step, arrived; };
struct World { int32_t w[3]; int count; std::vector<Block> b; };
template <typename F> bool walk(int nb, int ns, unsigned raises, int first) {
  auto raised = [&](int b, int k) { return raises >> (k * nb + b) & 1; };
  auto expect = [&](int k) {  // does step k begin with a rebuild?
    if (k == 0) return first;
    int v = 0;
    for (int b = 0; b < nb; ++b) v |= raised(b, k - 1);
    return v;
  };
  World w0{{first, 0, 0}, 0, std::vector<Block>(nb, Block{first ? REBUILD : COMMIT, 0, 0})};
  for (auto& b : w0.b) b.arrived = 0;
  std::set<std::vector<int>> seen;
  std::vector<World> todo{w0};
  while (!todo.empty()) {
    World w = todo.back();
    todo.pop_back();
    std::vector<int> key{w.w[0], w.w[1], w.w[2], w.count};
    for (auto& b : w.b) key.insert(key.end(), {b.at, b.step, b.arrived});
    if (!seen.insert(key).second) continue;
    bool over = true;
    for (int k = 0; k < nb; ++k) {
      if (w.b[k].at == OUT) continue;
      over = false;
      World v = w;
      Block& b = v.b[k];
      const F f{v.w, v.w + 1};
      // arrived: barriers this block has arrived at; it waits until all have
      auto arrive = [&] { ++b.arrived; ++v.count; };
      if (v.count < b.arrived * nb) continue;  // waiting
      switch (b.at) {
        case REBUILD: arrive(); b.at = CLEAR; break;
        case CLEAR: if (k == 0) *f.read_by(b.step) = 0; arrive(); b.at = REBUILT; break;
        case REBUILT: b.at = COMMIT; break;
        case COMMIT: if (raised(k, b.step)) *f.raised_by(b.step) = 1; arrive(); b.at = READ; break;
        case READ: {
          if (b.step + 1 == ns) { if (k == 0 && *f.read_by(ns)) f.hand_on(ns); b.at = OUT; break; }
          const int got = *f.read_by(b.step + 1);
          ++b.step;
          if (got != expect(b.step)) return false;
          b.at = got ? REBUILD : COMMIT;
        }
      }
      todo.push_back(v);
    }
    if (over && (w.w[0] != expect(ns) || w.w[1] || w.w[2])) return false;
  }
  return true;
}
template <typename F> bool all(int nb, int ns) {
  for (unsigned r = 0; r < 1u << (nb * ns); ++r)
    for (int first = 0; first < 2; ++first)
      if (!walk<F>(nb, ns, r, first)) return false;
  return true;
}
int main() {
  if (all<OneWord>(2, 3)) { puts("the model misses a word read and raised at once"); return 2; }
  return all<epi::RunFlags>(2, 4) && all<epi::RunFlags>(2, 5) && all<epi::RunFlags>(3, 3) ? 0 : 1;
}
"""


def test_blocks_agree_on_rebuilds_in_every_interleaving(tmp_path):
    subprocess.run([str(build(tmp_path, FLAGS))], check=True, timeout=300)


# Runs on a stream: some launches are refused, the others add their arrivals to
# their own word and clear the next one. Exits 0 when every run finds zero.
RUNS = r"""
#include <cstdio>
#include "epi_run_words.h"
int main() {
  for (unsigned refused = 0; refused < 1u << 12; ++refused) {
    epi::RunCount runs;
    unsigned word[2] = {0, 0};
    for (int k = 0; k < 12; ++k) {
      const int own = runs.own(), next = runs.next();
      if (own == next || word[own] != 0) return 1;
      if (refused >> k & 1) continue;
      ++runs.launched;
      word[next] = 0;
      word[own] += 148 * (1 + k);
    }
  }
  return 0;
}
"""


def test_a_refused_launch_leaves_the_next_run_a_zero_barrier_word(tmp_path):
    subprocess.run([str(build(tmp_path, RUNS))], check=True, timeout=60)
