"""Turn order of the softmax groups of the attention forward kernel (csrc/attn_turns.h), every interleaving of two groups of
two warps: no warp is left waiting, and no wait is answered by the parity of another turn.  The rule itself is compiled."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "frankentorch_b200" / "csrc"

MODEL = r"""
#include <array>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
#include "attn_turns.h"

struct Op { bool wait; unsigned parity; int turn; };      // wait for the other group's `turn`, or arrive
typedef std::vector<Op> Prog;
typedef std::vector<std::array<int, 2>> Items;

static Prog program(int t, const Items& items) {
  Prog p;
  ftk::AttnTurns turns;
  int taken = 0;
  for (const auto& it : items) {
    turns.item(it[0], it[1]);
    for (int j = 0; j < it[t]; ++j) {
      unsigned par;
      if (turns.waits(t, j, par)) p.push_back({true, par, taken - (t == 0)});
      if (turns.takes(j)) { p.push_back({false, 0, 0}); ++taken; }
    }
  }
  return p;
}
// The same without a wait at an item's first block and with every block counted.
static Prog loose(int t, const Items& items) {
  Prog p;
  int other = 0;
  for (const auto& it : items) {
    const int mine = it[t], theirs = it[t ^ 1], other0 = other;
    other += theirs;
    for (int j = 0; j < mine; ++j) {
      if (t == 0 ? (j > 0 && theirs > 0) : j < theirs) {
        const int want = other0 + (t == 0 ? j - 1 : j);
        p.push_back({true, (unsigned)(want & 1), want});
      }
      p.push_back({false, 0, 0});
    }
  }
  return p;
}
// 0: sound, 1: a warp waits for good, 2: a wait is answered by another turn's parity
static int explore(const Prog* g, int& states) {
  const int W = 2;
  typedef std::array<short, 4> S;      // program counters: two warps of group 0, two of group 1
  std::set<S> seen;
  std::vector<S> todo{S{0, 0, 0, 0}};
  seen.insert(todo[0]);
  std::vector<int> arrivals[2];
  for (int t = 0; t < 2; ++t) {
    arrivals[t].push_back(0);
    for (const Op& o : g[t]) arrivals[t].push_back(arrivals[t].back() + !o.wait);
  }
  int bad = 0;
  while (!todo.empty()) {
    const S s = todo.back();
    todo.pop_back();
    bool moved = false, done = true;
    for (int w = 0; w < 4; ++w) {
      const int t = w / W, u = t ^ 1;
      if (s[w] == (short)g[t].size()) continue;
      done = false;
      const Op& o = g[t][s[w]];
      if (o.wait) {
        const int c = (arrivals[u][s[u * W]] + arrivals[u][s[u * W + 1]]) / W;      // completed phases
        if (c != o.turn && c != o.turn + 1) bad = bad ? bad : 2;
        if ((unsigned)(c & 1) == o.parity) continue;                                // reads as not complete
      }
      moved = true;
      S n = s;
      ++n[w];
      if (seen.insert(n).second) todo.push_back(n);
    }
    if (!moved && !done) bad = 1;
  }
  states += (int)seen.size();
  return bad;
}
int main(int argc, char** argv) {
  const bool rule = atoi(argv[1]) == 0;
  // key blocks of an item's two tiles: causal, unmasked, and without a second tile
  const int kinds[7][2] = {{1, 2}, {1, 0}, {1, 1}, {2, 2}, {3, 4}, {3, 0}, {2, 0}};
  int states = 0, n_bad[3] = {0, 0, 0};
  for (int len = 1; len <= 3; ++len) {
    int combos = 1;
    for (int i = 0; i < len; ++i) combos *= 7;
    for (int c = 0; c < combos; ++c) {
      Items items;
      for (int i = 0, r = c; i < len; ++i, r /= 7) items.push_back({kinds[r % 7][0], kinds[r % 7][1]});
      const Prog g[2] = {rule ? program(0, items) : loose(0, items), rule ? program(1, items) : loose(1, items)};
      ++n_bad[explore(g, states)];
    }
  }
  printf("%d %d %d %d\n", n_bad[0], n_bad[1], n_bad[2], states);
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("turns")
    (d / "model.cpp").write_text(MODEL)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(CSRC), str(d / "model.cpp"), "-o", str(d / "model")], check=True,
                   capture_output=True)
    return lambda mode: [int(v) for v in
                         subprocess.run([str(d / "model"), str(mode)], check=True, capture_output=True, text=True).stdout.split()]


def test_turns_hold_in_every_interleaving(model):
    sound, stuck, lapped, states = model(0)
    assert (stuck, lapped) == (0, 0) and sound == 7 + 49 + 343
    assert states > 5000


def test_the_model_sees_a_turn_that_only_time_keeps(model):
    _, stuck, lapped, _ = model(1)
    assert stuck > 0
