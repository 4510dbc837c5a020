"""The drain of the tensor-core kernels after a wait that ran out (no GPU).

A kernel frees its TMEM only when the MMAs it issued have ended. The order in which it waits
for the phases of its mbarrier is TcPhase's (delta_b200/csrc/tcphase.h), compiled here for the
host and run against a model of the mbarrier: one arrival per commit, each completing the open
phase; a wait for a parity is over when the open phase has the other one. Every layer in turn
is made late, by less and by more than the limit of the drain. The sources are checked for the
two kernels using it, and for no commit between the wait that ran out and the drain.
"""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "delta_b200" / "csrc"

MODEL = r"""
#include <cstdio>
#include <deque>
#include "tcphase.h"

struct Barrier {          // count 1; commits arrive in order
  uint32_t open = 0;      // parity of the open phase
  long now = 0;
  std::deque<long> due;   // arrival times of the commits in flight
  void commit(long duration) { due.push_back((due.empty() || due.back() < now ? now : due.back()) + duration); }
  void tick() {
    ++now;
    while (!due.empty() && due.front() <= now) {
      due.pop_front();
      open ^= 1u;
    }
  }
  bool wait(uint32_t parity, int spin) {
    for (int i = 0; i < spin; ++i, tick())
      if (open != parity) return true;
    return false;
  }
};

constexpr int kSpin = 100;

// a kernel of `layers` layers, of which layer `slow` takes `duration`; returns 0 if it ends with
// nothing in flight and says so, 1 if with work in flight and says so, 2 if it claims an end
// that has not come, 3 if it waited for work that had ended, 4 if it did not notice
int kernel(int layers, int slow, long duration) {
  Barrier b;
  delta::TcPhase phase;
  auto bounded = [&](uint32_t parity) { return b.wait(parity, kSpin); };
  bool ok = true;
  for (int l = 0; l < layers && ok; ++l) {
    b.commit(l == slow ? duration : 3);
    ok = phase.wait(bounded);
    if (ok && !b.due.empty()) return 2;  // went on before the layer had ended
  }
  if (ok) return slow < 0 || duration < kSpin ? 0 : 4;
  const bool drained = phase.drain(bounded);
  if (drained && !b.due.empty()) return 2;
  if (!drained && b.due.empty()) return 3;
  return drained ? 0 : 1;
}

// the order that flips the parity whatever the wait returned and drains with one more commit
bool flipping_ends_clean(int layers, int slow, long duration) {
  Barrier b;
  uint32_t parity = 0;
  bool ok = true;
  for (int l = 0; l < layers && ok; ++l) {
    b.commit(l == slow ? duration : 3);
    ok = b.wait(parity, kSpin);
    parity ^= 1u;
  }
  b.commit(1);
  b.wait(parity, kSpin);
  return b.due.empty();
}

int main() {
  int bad = 0;
  for (int layers = 1; layers <= 9; ++layers) {
    bad += kernel(layers, -1, 0) != 0;
    for (int slow = 0; slow < layers; ++slow) {
      bad += kernel(layers, slow, kSpin - 1) != 0;      // in time
      bad += kernel(layers, slow, kSpin + 1) != 0;      // late, drained
      bad += kernel(layers, slow, 2 * kSpin - 2) != 0;  // late, drained at the last moment
      bad += kernel(layers, slow, 3 * kSpin) != 1;      // lost, and reported
    }
  }
  // the model tells the two orders apart
  if (flipping_ends_clean(5, 2, kSpin + 50)) return 90;
  std::printf("%d\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_nothing_is_in_flight_after_the_drain(tmp_path):
    src, exe = tmp_path / "drain.cpp", tmp_path / "drain"
    src.write_text(MODEL)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "0\n")


@pytest.mark.parametrize("file,wait", [("mlp_train.cu", "tr_wait"), ("mlp.cu", "tc_layer")])
def test_the_kernels_follow_the_phase(file, wait):
    text = (CSRC / file).read_text()
    body = text[text.index(f"__device__ __forceinline__ bool {wait}("):]
    body = body[:body.index("\n}\n")]
    assert "phase.wait(" in body and not re.search(r"phase\s*\^=", text)
    # after the wait that ran out: the drain, and no commit before it
    drain = text.index("phase.drain(")
    last = text.rindex("if (!ok", 0, drain)
    assert "tc_commit" not in text[last:drain]
    assert text.index("tcgen05.dealloc", drain) > drain
