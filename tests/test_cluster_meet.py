"""The exchange of the Newton norms' cluster (csrc/cluster_meet.h) on host threads, a thread per block:
no block may touch the first one's shared memory before that block has started, however late it
does, and the first block sees every value."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xyce_b200", "csrc")

# A cluster on host threads: arrive and wait of a split barrier, and a record of the blocks that run.
HARNESS = r"""
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
#include "cluster_meet.h"

struct Shared {
  int blocks, arrived = 0, phase = 0;
  std::mutex m;
  std::condition_variable cv;
  std::vector<std::atomic<int>> started;
  std::atomic<int> early{0};
  std::vector<double> slots;
  explicit Shared(int n) : blocks(n), started(n), slots(n, 0.0) {}
};

struct Cluster {
  Shared *s;
  int rank, mine = 0;
  void barrier_arrive() {
    std::lock_guard<std::mutex> l(s->m);
    mine = s->phase;
    if (++s->arrived == s->blocks) {
      s->arrived = 0;
      ++s->phase;
      s->cv.notify_all();
    }
  }
  void barrier_wait() {
    std::unique_lock<std::mutex> l(s->m);
    s->cv.wait(l, [&] { return s->phase != mine; });
  }
  void sync() { barrier_arrive(); barrier_wait(); }
  int block_rank() const { return rank; }
  double *map_shared_rank(double *p, int r) {
    if (!s->started[r]) ++s->early;  // memory of a block that does not run yet
    return p;
  }
};

int main(int, char **argv) {
  const int n = atoi(argv[1]), late = atoi(argv[2]);
  Shared s(n);
  double sum = 0.0;
  std::vector<std::thread> t;
  for (int b = 0; b < n; ++b)
    t.emplace_back([&, b] {
      if (b == late) std::this_thread::sleep_for(std::chrono::milliseconds(50));
      s.started[b] = 1;
      ClusterMeet<Cluster> meet(Cluster{&s, b}, true);
      meet.put(b + 1.0, s.slots.data(), true);
      if (b == 0)
        for (double v : s.slots) sum += v;
    });
  for (auto &x : t) x.join();
  if (s.early) return 2;
  return sum == n * (n + 1) / 2.0 ? 0 : 3;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("meet")
    (d / "meet.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(d / "meet.cpp"), "-o", str(d / "meet")], check=True)
    return str(d / "meet")


@pytest.mark.parametrize("blocks", [2, 8])
@pytest.mark.parametrize("late", [0, 1])
def test_no_store_before_the_first_block_runs(program, blocks, late):
    assert subprocess.run([program, str(blocks), str(late)], timeout=60).returncode == 0
