"""Handing walks out near the largest total of a launch (2^32 - 1 walks): the claim arithmetic of the walk kernels,
compiled for the host, against Python integers. No GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "claim.h"
using namespace bingo;
// argv: total warps chunk start -> the share, then every claim of warps that take turns until each has been refused.
int main(int, char** a) {
  const uint32_t total = strtoul(a[1], 0, 10), warps = strtoul(a[2], 0, 10), chunk = strtoul(a[3], 0, 10);
  WalkQueue q{strtoull(a[4], 0, 10), 0, 0};
  printf("%u\n", walk_share(total, warps));
  uint32_t running = warps, rounds = 0;
  while (running && ++rounds < 1000) {
    const uint32_t turn = running;
    for (uint32_t w = 0; w < turn; ++w) {
      const unsigned long long base = q.next;
      q.next += chunk;
      uint32_t b, e;
      if (claim_range(base < total ? base : total, total, chunk, &b, &e))
        printf("%u %u\n", b, e);
      else
        --running;
    }
  }
  printf("%s\n", running ? "still running" : "all refused");
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("claim")
    src = d / "claim.cpp"
    src.write_text(PROGRAM)
    exe = d / "claim"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "bingo_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True)
    return str(exe)


TOP = 2 ** 32


@pytest.mark.parametrize("chunk", [1, 4, 32, 1000, 1024])
@pytest.mark.parametrize("warps", [1, 8, 4736, 9472])
@pytest.mark.parametrize("total", [1, 31, 4737, TOP - 9472, TOP - 4736, TOP - 4735, TOP - 33, TOP - 32, TOP - 1])
def test_every_walk_is_claimed_once_and_every_warp_stops(program, total, warps, chunk):
    """The last 20 rounds of claims of a launch: shares stay in range, the claims tile [start, total) and every warp
    is refused in the end, also where the counter runs past 2^32."""
    start = max(0, total - total % chunk - 20 * warps * chunk) // chunk * chunk
    if (total - start) // chunk > 300_000:
        start = total // chunk * chunk - 300_000 * chunk
    start = max(0, start)
    out = subprocess.run([program, str(total), str(warps), str(chunk), str(start)], capture_output=True, text=True,
                         check=True, timeout=60).stdout.split("\n")
    assert int(out[0]) == -(-total // warps)
    assert 1 <= min(32, int(out[0]))
    at = start
    rows = [tuple(map(int, r.split())) for r in out[1:] if r and r[0].isdigit()]
    for b, e in rows:
        assert b == at and b < e <= total and e - b <= chunk
        at = e
    assert at == total
    assert "all refused" in out
