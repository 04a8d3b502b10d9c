"""How the two warps that share a query tile's rows exchange maxima and sums (csrc/attn_pair.h), run on the host as two coroutines
under many orders of their steps.  Every value read must be the one that the partner wrote for that step, and no warp may be left
waiting in a barrier."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgengraph_b200", "csrc")
PROGRAM = r"""
#include <ucontext.h>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "attn_pair.h"

constexpr int kTiles = 3, kBlocks = 3;
std::mt19937 rng;
ucontext_t main_ctx, ctx[2];
char stack[2][1 << 16];
bool done[2], blocked[2];
// what the two warps share
int arrived, generation, delivered[2];
bool ored, result, aborted;
float word[2];
// the problem: blocks per tile, a maximum and a sum for each block and half, one wait that runs out (or none)
int blocks[kTiles], expiring_warp, expiring_wait;
float maxima[2][kTiles][kBlocks], sums[2][kTiles][kBlocks];
struct Stored { int tile; float m, l; };
std::vector<Stored> stored[2];
int waits[2];

void yield(int id) { swapcontext(&ctx[id], &main_ctx); }

struct Pair {
  int id;
  bool vote(bool x) const {
    yield(id);
    ored = (arrived == 0 ? false : ored) || x;
    if (++arrived == 2) {
      arrived = 0;
      result = ored;
      ++generation;
      blocked[id ^ 1] = false;
      return result;
    }
    const int mine = generation;
    blocked[id] = true;
    while (generation == mine) yield(id);
    return result;
  }
  void put(float x) const { yield(id); word[id] = x; }
  float get() const { yield(id); return word[id ^ 1]; }
};

// a bounded wait: runs out where the problem says so, and once the other warp has given up
template <class Ready>
bool wait(int id, Ready ready) {
  if (id == expiring_warp && waits[id]++ == expiring_wait) {
    aborted = true;
    return false;
  }
  for (;;) {
    yield(id);
    if (ready()) return true;
    if (aborted) return false;
  }
}

void warp(int id) {
  const Pair w{id};
  int g = 0;
  for (int t = 0; t < kTiles; ++t) {
    if (!wait(id, [] { return true; })) return b200::pair_leave(w);   // the next tile
    float m = -1e30f, l = 0.f;
    for (int n = 0; n < blocks[t]; ++n, ++g) {
      // S of block g is computed after P V of block g - 2
      const bool ok = wait(id, [&] { return g < 2 || (delivered[0] >= g - 1 && delivered[1] >= g - 1); });
      float m_blk = maxima[id][t][n];
      const b200::PairStep step = b200::pair_block(w, ok, n == 0 || m_blk - m > 8.f, m_blk);
      if (step == b200::PairStep::kLeave) return;
      if (step == b200::PairStep::kMoved && (n == 0 || m_blk - m > 8.f)) {
        if (n > 0 && !wait(id, [&] { return delivered[0] >= g && delivered[1] >= g; })) return b200::pair_leave(w);
        m = m_blk;
      }
      l += sums[id][t][n];
      yield(id);
      ++delivered[id];   // P
    }
    if (!b200::pair_total(w, [&] { return wait(id, [&] { return delivered[0] >= g && delivered[1] >= g; }); }, l)) return;
    stored[id].push_back({t, m, l});
  }
  b200::pair_finish(w);
}
void entry(int id) {
  warp(id);
  done[id] = true;
  swapcontext(&ctx[id], &main_ctx);
}

// 0 done, 1 a warp waits in the barrier for good, 2 a wrong value
int run_one(unsigned seed, bool failures) {
  rng.seed(seed);
  arrived = generation = 0;
  ored = result = aborted = false;
  expiring_warp = failures ? (int)(rng() % 2) : -1;
  expiring_wait = (int)(rng() % 16);
  for (int t = 0; t < kTiles; ++t) {
    blocks[t] = 1 + rng() % kBlocks;
    for (int h = 0; h < 2; ++h)
      for (int n = 0; n < kBlocks; ++n) maxima[h][t][n] = (float)(rng() % 40), sums[h][t][n] = (float)(1000 + rng() % 1000);
  }
  for (int id = 0; id < 2; ++id) {
    done[id] = blocked[id] = false;
    delivered[id] = waits[id] = 0;
    stored[id].clear();
    getcontext(&ctx[id]);
    ctx[id].uc_stack.ss_sp = stack[id];
    ctx[id].uc_stack.ss_size = sizeof stack[id];
    ctx[id].uc_link = nullptr;
    makecontext(&ctx[id], (void (*)())entry, 1, id);
  }
  // orders from even to very uneven: one warp may stand still for a long time
  const int uneven = (int)(rng() % 4);
  int turn = 0, last = 0;
  for (int steps = 0; !done[0] || !done[1]; ++steps) {
    if (uneven == 0 || rng() % (1u << (2 * uneven)) == 0) turn = (int)(rng() % 2);
    int id = turn;
    if (done[id] || blocked[id]) id ^= 1;
    if (done[id] || blocked[id]) return 1;
    if (steps - last > 64) id = done[id ^ 1] || blocked[id ^ 1] ? id : id ^ 1, last = steps;   // a poll needs the other's progress
    swapcontext(&main_ctx, &ctx[id]);
  }
  for (int id = 0; id < 2; ++id) {
    if (!failures && (int)stored[id].size() != kTiles) return 2;
    for (const Stored& s : stored[id]) {
      float m = -1e30f, l[2] = {0.f, 0.f};
      for (int n = 0; n < blocks[s.tile]; ++n) {
        const float a = maxima[0][s.tile][n], b = maxima[1][s.tile][n];
        if (n == 0 || fmaxf(a, b) - m > 8.f) m = fmaxf(a, b);
        for (int h = 0; h < 2; ++h) l[h] += sums[h][s.tile][n];
      }
      if (s.m != m || s.l != l[0] + l[1]) return 2;
    }
  }
  return 0;
}

int main(int argc, char** argv) {
  const bool failures = atoi(argv[1]) != 0;
  int bad[3] = {};
  for (unsigned seed = 0; seed < 100000; ++seed) ++bad[run_one(seed, failures)];
  printf("%d %d\n", bad[1], bad[2]);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
  d = tmp_path_factory.mktemp("pair")
  (d / "pair.cpp").write_text(PROGRAM)
  subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I", CSRC, "-o", str(d / "pair"), str(d / "pair.cpp")], check=True)
  return str(d / "pair")


def test_every_value_read_belongs_to_its_step(program):
  waiting, wrong = map(int, subprocess.run([program, "0"], check=True, capture_output=True, text=True, timeout=300).stdout.split())
  assert (waiting, wrong) == (0, 0)


def test_a_wait_that_runs_out_ends_both_warps(program):
  waiting, wrong = map(int, subprocess.run([program, "1"], check=True, capture_output=True, text=True, timeout=300).stdout.split())
  assert (waiting, wrong) == (0, 0)
