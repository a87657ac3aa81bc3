"""The ring of state planes of the 3D reconstruction (plane_ring.h) on the host, with the
kernel's order of loads and waits: no plane overwrites one that is still to be read, each is
waited for with its own phase, and where any of the waits gives up, every load that was issued
and not seen to land is waited for once more before the block leaves."""
import subprocess

import pytest

import conftest

PROGRAM = r"""
#include <cstdio>
#include "%s/csrc/plane_ring.h"

// KEEP: plane k0 - 2's slot is filled again before the march, and plane k - 1 is not read at k
template <int RING, bool KEEP>
struct March {
  using Ring = kfvm::PlaneRing<RING>;
  int k0, last, failAt, waits = 0, lowest;   // planes below `lowest` have been read
  int plane[RING], armed[RING], landed[RING];   // of each slot: its plane, loads issued, loads seen to land
  bool drained[RING];
  bool wrong = false;

  March(int k0_, int k1, int failAt_) : k0(k0_), last(k1 + 1), failAt(failAt_), lowest(k0_ - 2) {
    for (int s = 0; s < RING; s++) plane[s] = armed[s] = landed[s] = 0, drained[s] = false;
  }
  void issue(int p) {
    const int s = Ring::slot(k0, p);
    if (p > last || armed[s] != landed[s] || (armed[s] && plane[s] >= lowest)) wrong = true;
    plane[s] = p;
    armed[s]++;
  }
  bool wait(int p) {
    const int s = Ring::slot(k0, p);
    // the phase of this parity is the one the slot's newest load completes
    if (!armed[s] || plane[s] != p || ((unsigned)(armed[s] - 1) & 1u) != Ring::parity(k0, p)) wrong = true;
    if (waits++ == failAt) return false;
    landed[s] = armed[s];
    return true;
  }
  // 0: every load was waited for
  int missed() {
    int n = 0;
    for (int s = 0; s < RING; s++) n += armed[s] != landed[s] && !drained[s];
    return wrong ? -1 : n;
  }
  int run(int k1) {
    for (int p = k0 - 2; p <= Ring::started(k0, last); p++) issue(p);
    bool ok = wait(k0 - 2) && wait(k0 - 1) && wait(k0) && wait(k0 + 1);
    lowest = k0 - 1;
    if (KEEP && ok) issue(k0 + 2);
    for (int k = k0; k < k1; k++) {
      ok = ok && wait(k + 2);
      if (!ok) {
        for (int p = Ring::flying_from(k0, k); p <= Ring::flying_to(k, last); p++) {
          // a wait for the slot's load in flight, or for a phase that is over
          const int s = Ring::slot(k0, p);
          if (((unsigned)(armed[s] - 1) & 1u) == Ring::parity(k0, p)) drained[s] = true;
        }
        return missed();
      }
      lowest = KEEP ? k : k - 1;
      if (k + 3 <= last) issue(k + 3);
    }
    return missed();
  }
};

int main() {
  int bad = 0, runs = 0;
  for (int n = 1; n <= 12; n++)
    for (int f = -1; f < n + 4; f++) {
      bad += March<4, true>(3, 3 + n, f).run(3 + n) != 0;
      bad += March<5, false>(3, 3 + n, f).run(3 + n) != 0;
      runs += 2;
    }
  printf("%%d %%d\n", runs, bad);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text(PROGRAM % conftest.PKG)
    subprocess.run(["g++", "-O1", "-std=c++17", str(d / "ring.cpp"), "-o", str(d / "ring")], check=True)
    return str(d / "ring")


def test_every_load_is_waited_for(program):
    runs, bad = (int(x) for x in subprocess.run([program], capture_output=True, text=True, check=True).stdout.split())
    assert runs > 200 and bad == 0
