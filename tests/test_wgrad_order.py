"""The order the weight gradients' work items are walked in (csrc/wgrad_order.cuh, compiled for the host):
every item has one place, whatever the schedule and however the list's length divides by the four items that
are read at a time, and every run's rows are covered once."""
import os
import random
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <vector>
#include "wgrad_order.cuh"

// lines of "ks_rows fixed_rows n start[0..n]" (fixed_rows -1: routed) -> per item "group row0 blocks place"
int main() {
  int ks, fixed, n;
  while (std::scanf("%d %d %d", &ks, &fixed, &n) == 3) {
    std::vector<int> start(n + 1), blocks, group, row0;
    for (int& s : start) std::scanf("%d", &s);
    const moe::WgradRuns runs{start.data(), fixed};
    for (int g = 0; g < n; ++g) {
      const int chunks = moe::wgrad_chunks(fixed >= 0 ? fixed : start[g + 1] - start[g], ks);
      for (int c = 0; c < chunks; ++c) {
        const moe::WgradRows w = moe::wgrad_rows(runs, ks, g, c);
        group.push_back(g);
        row0.push_back(w.row0);
        blocks.push_back(w.blocks);
      }
    }
    const int items = int(blocks.size());
    for (int i = 0; i < 3; ++i) blocks.push_back(moe::WGRAD_NO_ITEM);
    for (int i = 0; i < items; ++i) {
      int place = 0;
      for (int k = 0; k < items; k += 4)
        for (int u = 0; u < 4; ++u) place += moe::wgrad_before(blocks[k + u], k + u, blocks[i], i);
      std::printf("%d %d %d %d ", group[i], row0[i], blocks[i], place);
    }
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    where = tmp_path_factory.mktemp("wgrad_order")
    (where / "main.cpp").write_text(HARNESS)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", "-I",
                    os.path.join(ROOT, "nanospeaker_b200", "csrc"), str(where / "main.cpp"), "-o",
                    str(where / "main")], check=True)
    return str(where / "main")


def test_every_item_has_one_place_and_covers_its_rows(harness):
    rng = random.Random(0)
    lists = [(ks, rows, [0] * n + [rows]) for n in (1, 2, 9, 10, 13, 37, 256)      # the fixed schedule
             for ks, rows in [(256, 576), (128, 640), (64, 1), (3072, 4096), (64, 0)]]
    for n in (1, 9, 34, 78):                                                        # routed, empty runs too
        lens = [128 * rng.choice([0, 1, 1, 2, 3, 9, 33]) for _ in range(n)]
        lists.append((rng.choice([64, 1024, 3072]), -1, [sum(lens[:g]) for g in range(n + 1)]))
    asked = "".join(" ".join(map(str, [ks, fixed, len(start) - 1, *start])) + "\n" for ks, fixed, start in lists)
    out = subprocess.run([harness], input=asked, check=True, capture_output=True, text=True,
                         timeout=60).stdout.splitlines()
    assert len(out) == len(lists)
    for (ks, fixed, start), line in zip(lists, out):
        v = list(map(int, line.split()))
        items = [tuple(v[i:i + 4]) for i in range(0, len(v), 4)]
        assert sorted(i[3] for i in items) == list(range(len(items)))
        walked = sorted(items, key=lambda i: i[3])
        assert [i[2] for i in walked] == sorted((i[2] for i in items), reverse=True)
        for g in range(len(start) - 1):
            lo, hi = (0, fixed) if fixed >= 0 else (start[g], start[g + 1])
            mine = [i for i in items if i[0] == g]
            assert [i[1] for i in mine] == [lo + c * ks for c in range(len(mine))]
            ends = [min(i[1] + ks, hi) for i in mine]
            assert [i[2] for i in mine] == [max(0, -(-(e - i[1]) // 64)) for i, e in zip(mine, ends)]
            assert ends[-1] == hi
