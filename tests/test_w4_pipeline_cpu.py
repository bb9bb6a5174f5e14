"""The barriers of the 4-bit GEMM as a host model: its roles as actors that move one at a time in a random order, with the slot numbering of
``w4_steps.h``, the header the kernel includes.

A weight operand carries the (tile, K step, row quarter) it was made of; the product checks all four when it completes.  Two planted mistakes show that
the model sees what it is for: slots that follow the running step, and epilogue warps that leave one by one."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "batchgen_b200", "ops", "csrc")

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <random>
#include <vector>
#include "w4_steps.h"
using namespace bg::mx;

struct Bar {                                 // an mbarrier: phases complete after `count` arrivals, waits test a parity
  int count = 1, pending = 1, phase = 0;
  void init(int c) { count = pending = c; phase = 0; }
  void arrive() { if (--pending == 0) { pending = count; ++phase; } }
  bool passes(unsigned parity) const { return (unsigned)((phase & 1) ^ 1) == parity; }
};

constexpr int kX = 6, kQ = 4, kWarps = 4 * kGroups;
enum Wait { kBlocked, kPass, kLeave };

struct Run {
  std::mt19937 rng;
  int KB, tiles;
  bool by_step, one_by_one, abort_flag = false;
  long wrong = 0;
  Bar x_full[kX], x_empty[kX], q_full[kQ], q_empty[kQ], w_full[kGroups], w_empty[kGroups], t_full[2], t_empty[2];
  int slot[kGroups][4];                      // tile * KB + step that a quarter of the rows holds
  struct Actor { std::function<bool()> move; bool done = false, looked = false; };
  std::vector<Actor> a;
  std::vector<std::function<void()>> inflight;             // products and commits, in order
  size_t completed = 0;
  int at_bar = 0, bar_gen = 0;               // the named barrier of the four epilogue warps

  int slot_of(int tile, int kb) const { return by_step ? (tile * KB + kb) % kGroups : step_group(kb); }
  unsigned use_of(int tile, int kb) const { return by_step ? (tile * KB + kb) / kGroups : slot_use(KB, tile, kb); }
  // as mbar_wait: the barrier first; a look at the abort flag only after a look at an incomplete barrier
  Wait wait(int me, const Bar& b, unsigned parity) {
    if (a[me].looked && abort_flag) return kLeave;
    a[me].looked = false;
    if (b.passes(parity)) return kPass;
    a[me].looked = true;
    return kBlocked;
  }

  // 0: every actor ended; 1: stuck
  int go(bool raise_abort, bool silu) {
    for (auto& b : x_full) b.init(1);
    for (auto& b : x_empty) b.init(1);
    for (auto& b : q_full) b.init(1);
    for (auto& b : q_empty) b.init(kWarps);
    for (int g = 0; g < kGroups; ++g) { w_full[g].init(4); w_empty[g].init(1); }
    for (int b = 0; b < 2; ++b) { t_full[b].init(1); t_empty[b].init(4); }
    const int total = tiles * KB, stages = (KB + kGroups - 1) / kGroups;
    a.resize(2 + kWarps + 1 + 4 + 1);
    int n = 0;
    { const int me = n++; int it = 0;                      // token tiles
      a[me].move = [=, this]() mutable {
        const Wait w = wait(me, x_empty[it % kX], ((it / kX) & 1) ^ 1);
        if (w == kBlocked) return false;
        if (w == kPass) { x_full[it % kX].arrive(); ++it; }
        if (w == kLeave || it == total) a[me].done = true;
        return true; }; }
    { const int me = n++; int it = 0;                      // packed weights
      a[me].move = [=, this]() mutable {
        const Wait w = wait(me, q_empty[it % kQ], ((it / kQ) & 1) ^ 1);
        if (w == kBlocked) return false;
        if (w == kPass) { q_full[it % kQ].arrive(); ++it; }
        if (w == kLeave || it == tiles * stages) a[me].done = true;
        return true; }; }
    for (int v = 0; v < kWarps; ++v) {                     // expansion warps
      const int me = n++, g = v / 4, quad = v % 4; int tile = 0, kb = g, stage = 0; bool have = false;
      a[me].move = [=, this]() mutable {
        if (!have) {
          const Wait w = wait(me, q_full[stage % kQ], (stage / kQ) & 1);
          if (w == kBlocked) return false;
          if (w == kLeave) { a[me].done = true; return true; }
          q_empty[stage % kQ].arrive(); ++stage;
          if (kb < KB) { have = true; return true; }
        } else {
          const int s = slot_of(tile, kb);
          const Wait w = wait(me, w_empty[s], (use_of(tile, kb) & 1) ^ 1);
          if (w == kBlocked) return false;
          if (w == kLeave) { a[me].done = true; return true; }
          slot[s][quad] = tile * KB + kb; w_full[s].arrive(); have = false;
        }
        kb += kGroups;
        if (kb >= KB + g) { kb = g; if (++tile == tiles) a[me].done = true; }
        return true; }; }
    { const int me = n++; int tile = 0, kb = -1; bool x = false;      // MMA issuer
      a[me].move = [=, this]() mutable {
        Wait w;
        if (kb < 0) { w = wait(me, t_empty[tile & 1], ((tile >> 1) & 1) ^ 1); if (w == kPass) kb = 0; }
        else if (!x) { const int it = tile * KB + kb; w = wait(me, x_full[it % kX], (it / kX) & 1); x = w == kPass; }
        else {
          const int s = slot_of(tile, kb), it = tile * KB + kb;
          w = wait(me, w_full[s], use_of(tile, kb) & 1);
          if (w == kPass) {
            inflight.push_back([=, this]() { for (int q = 0; q < 4; ++q) wrong += slot[s][q] != it; x_empty[it % kX].arrive(); w_empty[s].arrive(); });
            x = false;
            if (++kb == KB) { const int b = tile & 1; inflight.push_back([=, this]() { t_full[b].arrive(); }); kb = -1; if (++tile == tiles) a[me].done = true; }
          }
        }
        if (w == kLeave) a[me].done = true;
        return w != kBlocked; }; }
    for (int q = 0; q < 4; ++q) {                          // epilogue warps: wait, with SiLU two named barriers, arrive
      const int me = n++; int tile = 0, state = 0, gen = 0; bool fail = false;
      static bool any_fail; any_fail = false;
      a[me].move = [=, this]() mutable {
        auto join = [&]() { gen = bar_gen; if (++at_bar == 4) { at_bar = 0; ++bar_gen; } };
        if (state == 0) {
          const Wait w = wait(me, t_full[tile & 1], (tile >> 1) & 1);
          if (w == kBlocked) return false;
          fail = w == kLeave;
          if (silu && !one_by_one) { any_fail = any_fail || fail; join(); state = 1; return true; }   // a vote: OR of the four
          if (fail) { a[me].done = true; return true; }
          state = 2;
        } else if (state == 1) {
          if (bar_gen == gen) return false;
          if (any_fail) { a[me].done = true; return true; }
          state = 2;
        } else if (state == 2) {
          if (silu) join();
          state = 3;
        } else if (state == 3) {
          if (silu && bar_gen == gen) return false;
          if (silu) join();
          state = 4;
        } else {
          if (silu && bar_gen == gen) return false;
          t_empty[tile & 1].arrive(); state = 0;
          if (++tile == tiles) a[me].done = true;
        }
        return true; }; }
    { const int me = n++;                                  // the tensor core: completes what was issued, in order
      a[me].move = [=, this]() {
        if (completed < inflight.size()) { inflight[completed++](); return true; }
        return false; }; }
    const int raise_at = raise_abort ? (int)(rng() % (unsigned)(total * 40)) : -1;
    int slow = -1, held = 0, idle = 0;
    const int actors = n;
    for (long step = 0;; ++step) {
      if (step == raise_at) abort_flag = true;
      if (held-- <= 0) { slow = rng() % 3 == 0 ? (int)(rng() % actors) : -1; held = 1 + rng() % 200; }   // an actor that is late for a while
      bool left = false;
      for (int i = 0; i < actors - 1; ++i) left = left || !a[i].done;
      if (!left) return 0;
      const int i = rng() % actors;
      if (i == slow || a[i].done) continue;
      if (a[i].move()) idle = 0;
      else if (++idle > 4000) { if (raise_at > step) { abort_flag = true; idle = 0; continue; } return 1; }
    }
  }
};

int main(int argc, char** argv) {
  const int first = atoi(argv[1]), last = atoi(argv[2]), trials = atoi(argv[3]);
  const bool by_step = atoi(argv[4]), one_by_one = atoi(argv[5]), aborts = atoi(argv[6]);
  long wrong = 0, stuck = 0;
  for (int KB = first; KB <= last; ++KB)
    for (int t = 0; t < trials; ++t) {
      Run r;
      r.rng.seed(KB * 1000 + t);
      r.KB = KB; r.tiles = 1 + t % 4; r.by_step = by_step; r.one_by_one = one_by_one;
      stuck += r.go(aborts, aborts || t % 2);
      wrong += r.wrong;
    }
  std::printf("%ld %ld\n", wrong, stuck);
  return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("w4")
    (d / "model.cpp").write_text(MODEL)
    subprocess.run(["g++", "-std=c++20", "-O2", f"-I{CSRC}", str(d / "model.cpp"), "-o", str(d / "model")], check=True)

    def run(first, last, trials, by_step=0, one_by_one=0, aborts=0):
        out = subprocess.run([str(d / "model"), *map(str, (first, last, trials, by_step, one_by_one, aborts))], check=True, text=True,
                             stdout=subprocess.PIPE, timeout=300).stdout
        return tuple(map(int, out.split()))

    return run


def test_every_product_reads_its_own_weights(model):
    """1 to 48 K steps, one to four tiles of a CTA."""
    assert model(1, 48, 60) == (0, 0)


def test_failed_waits_end_every_role(model):
    """A role that gives up at any moment: every other one ends, with the barriers of the SiLU epilogue between its warps."""
    wrong, stuck = model(1, 9, 400, aborts=1)
    assert stuck == 0


@pytest.mark.parametrize("steps", [5, 6, 7, 45])
def test_model_sees_slots_that_follow_the_running_step(model, steps):
    wrong, stuck = model(steps, steps, 400, by_step=1)
    assert wrong + stuck > 0


def test_model_sees_epilogue_warps_that_leave_one_by_one(model):
    assert model(1, 9, 400, one_by_one=1, aborts=1)[1] > 0
