"""The give-up protocol of waits that a group of threads acts on together (csrc/agree.cuh), compiled for
the host: whatever another thread writes meanwhile, all of the group go on or all leave."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <atomic>
#include <barrier>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "agree.cuh"

// argv[1]: when an outsider raises the abort flag: 0 never, 1 before the leader looks, 2 behind the
// barrier, when the first thread has its answer and the others have not
int main(int, char** argv) {
  const int when = std::atoi(argv[1]);
  constexpr int N = 4;
  std::barrier<> gate(N);
  volatile int answer = -1;
  std::atomic<int> abort_flag{when == 1}, first_out{0}, reads_behind{0};
  int got[N];
  std::vector<std::thread> group;
  for (int i = 0; i < N; ++i)
    group.emplace_back([&, i] {
      bool behind = false;
      got[i] = moe::agree(i == 0, &answer, [&] {
        if (behind || i != 0) ++reads_behind;
        return abort_flag.load() == 0;
      }, [&] {
        gate.arrive_and_wait();
        behind = true;
        if (i == 0) return;
        while (!first_out) std::this_thread::yield();
        if (when == 2) abort_flag = 1;
      });
      if (i == 0) first_out = 1;
    });
  for (auto& t : group) t.join();
  for (int i = 0; i < N; ++i) std::printf("%d ", got[i]);
  std::printf("%d\n", reads_behind.load());
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    where = tmp_path_factory.mktemp("agree")
    (where / "main.cpp").write_text(HARNESS)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++20", "-O1", "-pthread", "-I",
                    os.path.join(ROOT, "nanospeaker_b200", "csrc"), str(where / "main.cpp"), "-o",
                    str(where / "main")], check=True)
    return str(where / "main")


@pytest.mark.parametrize("when,go", [(0, 1), (1, 0), (2, 1)])
def test_a_group_goes_on_or_leaves_as_one(harness, when, go):
    out = subprocess.run([harness, str(when)], check=True, capture_output=True, text=True, timeout=60)
    *got, reads_behind = map(int, out.stdout.split())
    assert got == [go] * 4            # (an abort raised behind the barrier counts at the next wait)
    assert reads_behind == 0
