"""Claim sizes of mixed walk tables, compiled for the host, in a model of one warp: 32 lanes, each on a walk of some
length, refilled from the warp's claims. Short walks must not go to the counter at every step, long ones must not be
held unstarted, and a table that changes from one to the other is followed. No GPU."""
import subprocess
from pathlib import Path

import pytest

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include "claim.h"
using namespace bingo;
// argv: mean lengths of the walks in turn, 3000 steps each -> per part: claims per 1000 steps, mean size held
int main(int n, char** a) {
  std::mt19937 rng(1);
  unsigned left[32] = {0}, turn = 0, claim = kClaimMin, claimed = 0, held = 0;
  for (int p = 1; p < n; ++p) {
    const double mean = atof(a[p]);
    std::geometric_distribution<unsigned> len(1 / mean);
    unsigned claims = 0, steps = 0;
    double waiting = 0;
    for (unsigned s = 0; s < 3000; ++s) {
      for (unsigned& l : left)
        if (!l) {
          if (!held) {
            claim = turn ? next_claim(claim, turn - claimed) : kClaimMin;
            if (claim < kClaimMin || claim > kClaimMax) return 1;
            claimed = turn, held = claim;
            claims += s >= 500;
          }
          --held;
          l = 1 + len(rng);
        }
      for (unsigned& l : left) --l;
      ++turn;
      if (s >= 500) waiting += held, ++steps;
    }
    printf("%.1f %.2f\n", claims * 1000. / steps, waiting / steps);
  }
}
"""


@pytest.fixture(scope="module")
def warp(tmp_path_factory):
    d = tmp_path_factory.mktemp("claims")
    (d / "claims.cpp").write_text(PROGRAM)
    csrc = Path(__file__).resolve().parent.parent / "bingo_b200" / "csrc"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(csrc), str(d / "claims.cpp"), "-o", str(d / "claims")],
                   check=True)

    def run(*means):
        out = subprocess.run([str(d / "claims"), *map(str, means)], capture_output=True, text=True, check=True)
        return [tuple(map(float, line.split())) for line in out.stdout.splitlines()]
    return run


@pytest.mark.parametrize("mean", [1.5, 3, 6.7, 10])
def test_short_walks_claim_seldom(warp, mean):
    """At four per claim a step of walks of mean length m takes 8 / m claims: every step one or more for these."""
    (claims, _), = warp(mean)
    assert claims < 1000 * max(32 / mean / 32 * 1.2, 0.45)


@pytest.mark.parametrize("mean", [80, 150, 400])
def test_long_walks_are_not_held(warp, mean):
    (_, held), = warp(mean)
    assert held < 4


def test_sizes_follow_the_table(warp):
    parts = warp(150, 5, 150, 5)
    alone = [warp(150)[0], warp(5)[0]]
    for got, want in zip(parts, alone * 2):
        assert got[0] == pytest.approx(want[0], rel=0.15, abs=5) and got[1] == pytest.approx(want[1], rel=0.2, abs=1)
