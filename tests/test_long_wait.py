"""The wait of a long-read strip for the strip above it, on the CPU.

csrc/pairhmm_wait.h is compiled for the host with 32 threads as a warp's lanes.  The
word moves on with every read of it, as it does while another warp publishes blocks, so
lanes that read it for themselves would come back with different counts; every lane has
to return the same word, and give up together.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "vardepth_b200" / "csrc"

PROGRAM = r"""
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>
#include "pairhmm_wait.h"

constexpr int kLanes = 32;
struct Shared {
  std::atomic<unsigned long long> word{0};
  std::atomic<int> loads{0}, error{0};
  bool moving = true;
  unsigned long long handed = 0;
  std::mutex mu;
  std::condition_variable cv;
  int arrived = 0, round = 0;
  void meet() {
    std::unique_lock<std::mutex> lk(mu);
    const int r = round;
    if (++arrived == kLanes) { arrived = 0; ++round; cv.notify_all(); }
    else cv.wait(lk, [&] { return round != r; });
  }
};
struct HostWarp {
  Shared& s;
  int lane;
  unsigned long long load() const { ++s.loads; return s.moving ? ++s.word : s.word.load(); }
  bool stopped() const { return s.error != 0; }
  void give_up() const { s.error = 2; }
  void pause() const {}
  unsigned long long from_leader(unsigned long long v) const {
    if (lane == 0) s.handed = v;
    s.meet();
    v = s.handed;
    s.meet();
    return v;
  }
};

int main() {
  int bad = 0;
  for (int mode = 0; mode < 2; ++mode) {  // 0: the word advances; 1: another wait has given up
    Shared s;
    s.moving = mode == 0;
    s.error = mode;
    for (int need = 1; need < (mode == 0 ? 40 : 2); ++need) {
      std::vector<std::thread> lanes;
      unsigned long long got[kLanes];
      bool ok[kLanes];
      for (int l = 0; l < kLanes; ++l)
        lanes.emplace_back([&, l] {
          HostWarp w{s, l};
          ok[l] = true;
          got[l] = vd::wait_word(w, need, ok[l]);
        });
      for (auto& t : lanes) t.join();
      for (int l = 0; l < kLanes; ++l) {
        bad += got[l] != got[0] || ok[l] != ok[0];
        bad += ok[l] != (mode == 0) || (ok[l] && vd::task_blocks(got[l]) < need);
      }
    }
  }
  std::printf("%d\n", bad);
  return bad != 0;
}
"""


def test_every_lane_returns_the_same_word(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "wait.cpp", tmp_path / "wait"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout
