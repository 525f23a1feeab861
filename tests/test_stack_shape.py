"""Which shapes and devices the decode stack takes (csrc/stack_shape.cuh, compiled for the host): its CTAs
wait on one another, so that a grid which is not resident as a whole must be declined, device by device."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "stack_shape.cuh"

// lines of "sms blocks_per_sm cooperative T E" -> "taken grid items"; then the values of devices 0 .. 3
// (sms = 10 + device) as eight threads see them, and how often each was asked for
int main() {
  int sms, blocks, coop, T, E;
  while (std::scanf("%d %d %d %d %d", &sms, &blocks, &coop, &T, &E) == 5) {
    moe::StackDevice dev{sms, blocks, coop != 0};
    moe::StackShape o{};
    const bool ok = moe::stack_shape(dev, T, 576, 128, E, 2, 6, &o);
    std::printf("%d %d %d\n", ok, dev.grid(), ok ? o.n_items : 0);
  }
  static moe::PerDevice<moe::StackDevice> devices;
  static std::atomic<int> asked[4];
  std::atomic<bool> same{true};
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i)
    threads.emplace_back([&] {
      for (int d = 0; d < 4; ++d)
        if (devices.get(d, [](int dev) {
              ++asked[dev];
              return moe::StackDevice{10 + dev, 1, true};
            })->grid() != 10 + d)
          same = false;
    });
  for (auto& t : threads) t.join();
  std::printf("%d %d %d %d %d %d\n", int(same), int(asked[0]), int(asked[1]), int(asked[2]), int(asked[3]),
              devices.get(-1, [](int) { return moe::StackDevice{}; }) == nullptr);
}
"""
DEVICES = [((148, 1, 1, 64, 76), (1, 148, 336)),
           ((148, 1, 1, 256, 76), (1, 148, 368)),
           ((148, 0, 1, 64, 76), (0, 0, 0)),      # no room for its shared memory
           ((148, 1, 0, 64, 76), (0, 0, 0)),      # no cooperative launch
           ((42, 1, 1, 64, 76), (1, 42, 336)),    # a part of the SMs: eight items each
           ((41, 1, 1, 64, 76), (0, 41, 0)),      # more than that
           ((41, 1, 1, 64, 32), (1, 41, 160)),
           ((16, 1, 1, 65, 8), (0, 16, 0))]       # more tokens than slots


@pytest.fixture(scope="module")
def answers(tmp_path_factory):
    where = tmp_path_factory.mktemp("stack_shape")
    (where / "main.cpp").write_text(HARNESS)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", "-pthread", "-I",
                    os.path.join(ROOT, "nanospeaker_b200", "csrc"), str(where / "main.cpp"), "-o",
                    str(where / "main")], check=True)
    asked = "".join(" ".join(map(str, q)) + "\n" for q, _ in DEVICES)
    out = subprocess.run([str(where / "main")], input=asked, check=True, capture_output=True, text=True,
                         timeout=60).stdout.splitlines()
    return [tuple(map(int, line.split())) for line in out]


def test_a_grid_that_would_not_be_resident_is_declined(answers):
    assert answers[:-1] == [want for _, want in DEVICES]


def test_every_device_answers_for_itself(answers):
    assert answers[-1] == (1, 1, 1, 1, 1, 1)
