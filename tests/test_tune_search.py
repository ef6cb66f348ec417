"""The autotuner's search, compiled for the host, on made-up run times: it finds the small claims that the walk kernels
default to, and it does not move the knobs on times that do not hold up against the starting ones. No GPU."""
import subprocess
from pathlib import Path

import pytest

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "tune_search.h"
using namespace bingo;
static unsigned calls = 0;
static const char* form;
// Milliseconds of a run under t.
static double once(const Tuning& t) {
  ++calls;
  if (!strcmp(form, "small")) return t.walk_chunk == 4 || t.walk_chunk == 0 ? 10 : t.walk_chunk < 4 ? 11 : 12 - t.walk_chunk / 64. * .1 + (t.walk_chunk == 8);
  if (!strcmp(form, "two")) return t.walk_chunk == 2 ? 8 : t.walk_chunk == 32 ? 9 : 10;
  if (!strcmp(form, "warming")) return 10. + 5. * 30 / (calls + 30);     // every run faster than the one before
  if (!strcmp(form, "late")) return calls < 60 && t.walk_chunk == 64 ? 8 : 10 + (t.walk_chunk == 64);  // a lucky spell
  if (!strcmp(form, "split")) return 10 - 2. * t.walk_split + (t.walk_order == 0);
  if (!strcmp(form, "update")) return t.apply_blocks_per_sm == 16 ? 3 : 4;
  return 10;
}
int main(int, char** a) {
  form = a[1];
  Tuning start;
  start.walk_chunk = atoi(a[2]);
  KnobSearch<double (*)(const Tuning&)> s(start, 3, once);
  if (!strcmp(form, "update"))
    search_update_knobs(s, 100000);
  else
    search_walk_knobs(s, true, true);
  printf("%u %u %u %u %u %d\n", s.best.walk_chunk, s.best.walk_split, s.best.walk_order, s.best.walk_blocks_per_sm,
         s.best.apply_blocks_per_sm, s.ms_best <= s.ms_start);
}
"""


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    (d / "tune.cpp").write_text(PROGRAM)
    csrc = Path(__file__).resolve().parent.parent / "bingo_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-I", str(csrc), str(d / "tune.cpp"), "-o", str(d / "tune")], check=True)

    def run(form, start=0):
        out = subprocess.run([str(d / "tune"), form, str(start)], capture_output=True, text=True, check=True)
        return tuple(map(int, out.stdout.split()))
    return run


@pytest.mark.parametrize("form,start,chunk", [("small", 32, (0, 4)), ("small", 256, (0, 4)), ("small", 8, (0, 4)),
                                              ("small", 0, (0,)), ("two", 0, (2,)), ("two", 32, (2,))])
def test_small_claims_are_found(search, form, start, chunk):
    assert search(form, start)[0] in chunk


@pytest.mark.parametrize("form", ["flat", "warming", "late"])
def test_knobs_stay_without_a_lasting_gain(search, form):
    assert search(form, 16) == (16, 0, 1, 0, 8, 1)


def test_other_knobs(search):
    assert search("split") == (0, 1, 1, 0, 8, 1)
    assert search("update") == (0, 0, 1, 0, 16, 1)
