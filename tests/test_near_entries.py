"""The back-pointers that a delete brings near lie inside the edge's own run, for every number of set bits: the
function of the delete kernel, compiled for the host. No GPU."""
import subprocess
from pathlib import Path

PROGRAM = r"""
#include <cstdio>
#include "near.h"
int main() {
  unsigned w;
  while (scanf("%u", &w) == 1) printf("%u\n", bingo::near_last(w));
}
"""


def test_inside_the_run(tmp_path):
    root = Path(__file__).resolve().parent.parent
    (tmp_path / "near.cpp").write_text(PROGRAM)
    exe = tmp_path / "near"
    subprocess.run(["g++", "-std=c++17", "-I", str(root / "bingo_b200" / "csrc"), str(tmp_path / "near.cpp"), "-o",
                    str(exe)], check=True)
    words = [0] + [(1 << b) - 1 for b in range(1, 33)] + [1 << b for b in range(32)] + [0xAAAAAAAA, 0x80000001]
    out = subprocess.run([str(exe)], input="\n".join(map(str, words)), capture_output=True, text=True, check=True)
    for w, last in zip(words, map(int, out.stdout.split()), strict=True):
        run = bin(w).count("1")
        assert last == max(0, min(8, run) - 1), (w, last)
    # The kernel asks for these entries only, and only of an edge that is there.
    body = (root / "bingo_b200" / "csrc" / "engine.cu").read_text().split("k_apply_delete(", 1)[1].split("\n}\n", 1)[0]
    asked = [line.strip() for line in body.splitlines() if "prefetch_l2" in line and "S.bp" in line]
    assert len(asked) == 2 and "near_last(e.w)" in asked[1]
