"""The warp reconstruction's bookkeeping of its double buffer (copy_phases.h) on
the CPU, against barriers that are played here: a wait that gives up must leave
the parity of the copy in flight, so that the drain before the block's end waits
for that copy and does not return at once."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lowrank_gpu_fastest_b200", "csrc")

# The walk of recon_warp_body: the next chunk's copy is issued into the other
# buffer, then this chunk's is waited for. Copy ``late`` and the one after it
# (already issued then) only land after the walk. ``skip``: every skip-th chunk
# has no rows to copy.
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "copy_phases.h"

struct Barrier {  // mbarrier: ``done`` phases are complete
  int done = 0, asked = 0;
  bool passes(unsigned parity) const { return ((done & 1) != 0) != (parity != 0); }
};

int main(int, char** argv) {
  const int chunks = atoi(argv[1]), late = atoi(argv[2]), skip = atoi(argv[3]);
  lrd::CopyPhases ph;
  Barrier bar[2];
  int landed[2] = {0, 0}, gave_up = -1;
  auto rows = [&](int c) { return c < chunks && (skip == 0 || c % skip != skip - 1); };
  auto copy = [&](int c) {
    if (!rows(c) || !ph.ok) return;
    const int b = c & 1;
    if (ph.in_flight(b)) return (void)(printf("chunk %d overwrites buffer %d\n", c, b), exit(1));
    ph.issued(b);
    ++bar[b].asked;
    if (gave_up < 0 && (late < 0 || c < late)) ++bar[b].done;  // lands before it is waited for
  };
  copy(0);
  for (int c = 0; c < chunks; ++c) {
    copy(c + 1);
    if (!rows(c) || !ph.ok) continue;
    const int b = c & 1;
    const bool arrived = bar[b].passes(ph.parity(b));
    if (arrived != (bar[b].done == bar[b].asked)) return printf("chunk %d: waited for the wrong phase\n", c), 1;
    if (!arrived) gave_up = c;
    ph.waited(b, arrived);
  }
  for (int b = 0; b < 2; ++b) {
    const bool flying = bar[b].done < bar[b].asked;
    if (flying && !ph.in_flight(b)) return printf("buffer %d: a copy in flight is not waited for\n", b), 1;
    if (!ph.in_flight(b)) continue;
    if (bar[b].passes(ph.parity(b)) == flying) return printf("buffer %d: the drain asks for the wrong phase\n", b), 1;
    bar[b].done = bar[b].asked;
    if (!bar[b].passes(ph.parity(b))) return printf("buffer %d: the drain would wait for ever\n", b), 1;
  }
  printf("%d\n", gave_up);
  return 0;
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("copy_phases")
    (d / "walk.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", CSRC, str(d / "walk.cpp"), "-o", str(d / "walk")], check=True)
    return str(d / "walk")


@pytest.mark.parametrize("skip", [0, 2, 3, 5])
def test_drain_waits_for_the_copy_in_flight(walk, skip):
    for chunks in (1, 2, 3, 8, 9):
        for late in range(-1, chunks):
            p = subprocess.run([walk, str(chunks), str(late), str(skip)], capture_output=True, text=True)
            assert p.returncode == 0, (chunks, late, p.stdout)
            copied = [c for c in range(chunks) if skip == 0 or c % skip != skip - 1]
            stuck = [c for c in copied if c >= late] if late >= 0 else []
            assert int(p.stdout) == (stuck[0] if stuck else -1)
