"""The ring that the one-launch decode step's keys come through (``csrc/key_ring.cuh``), compiled here with threads in place of
warps and counters in place of barriers: no stage is filled again under a warp that still reads it, whichever warp is slow."""
import ctypes
import subprocess

import pytest

from llm_serving_engine_b200.csrc import build

_TRIAL = '''
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>
#include "key_ring.cuh"
using namespace std::chrono;
// A barrier that counts arrivals and goes through phases, as those in shared memory do.
struct Barrier {
  int count = 0, pending = 0;
  unsigned phase = 0;
  std::mutex lock;
  std::condition_variable changed;
  void init(int n) { count = pending = n; }
  void arrive() {
    std::lock_guard<std::mutex> hold(lock);
    if (--pending == 0) { pending = count; ++phase; changed.notify_all(); }
  }
  bool wait(unsigned parity) {
    std::unique_lock<std::mutex> hold(lock);
    return changed.wait_for(hold, seconds(5), [&] { return (phase & 1u) != parity; });
  }
};
// Stages that were not what a warp began to read, and waits that gave up; warp `slow` takes long over its first tile, and the data
// of stage `late` lands late.
extern "C" int trial(int warps, int tiles, int a_stage, int stages, int slow, int late) {
  std::vector<Barrier> full(stages), empty(stages);
  for (int i = 0; i < stages; ++i) { full[i].init(1); empty[i].init(warps); }
  std::vector<std::atomic<int>> held(stages);
  for (auto& h : held) h = -1;
  std::atomic<int> wrong{0};
  std::vector<std::thread> threads;
  threads.emplace_back([&] {
    Slot slot;
    for (int first = 0; first < tiles; first += a_stage) {
      if (!empty[slot.at].wait(slot.parity ^ 1u)) { ++wrong; return; }
      if (first / a_stage == late) std::this_thread::sleep_for(milliseconds(40));
      held[slot.at] = first / a_stage;
      full[slot.at].arrive();
      slot.step(stages);
    }
  });
  for (int warp = 0; warp < warps; ++warp)
    threads.emplace_back([&, warp] {
      Slot slot;
      bool first = true;
      walk_key_stages(warp, warps, tiles, a_stage, stages, slot, [&](const Slot& at) { if (!full[at.at].wait(at.parity)) ++wrong; },
                      [&](const Slot& at, int, int t) {
                        if (held[at.at] != t / a_stage) ++wrong;
                        if (first && warp == slow) std::this_thread::sleep_for(milliseconds(80));
                        first = false;
                        if (held[at.at] != t / a_stage) ++wrong;
                      },
                      [&](const Slot& at) { empty[at.at].arrive(); });
    });
  for (auto& thread : threads) thread.join();
  return wrong;
}
'''


@pytest.fixture(scope="module")
def trial(tmp_path_factory):
    folder = tmp_path_factory.mktemp("ring")
    (folder / "trial.cpp").write_text(_TRIAL)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", f"-I{build.CSRC}", str(folder / "trial.cpp"), "-o",
                    str(folder / "trial.so")], check=True)
    return ctypes.CDLL(str(folder / "trial.so")).trial


# as the kernel has it (eight warps, three tiles a stage, four to six stages): fewer stages than the ring has, one more, many
@pytest.mark.parametrize("stages", [4, 6])
@pytest.mark.parametrize("tiles", [1, 18, 19, 24, 79])
@pytest.mark.parametrize("slow", range(8))
def test_no_stage_is_filled_again_under_a_slow_warp(trial, stages, tiles, slow):
    assert trial(8, tiles, 3, stages, slow, -1) == 0


@pytest.mark.parametrize("late", [0, 1, 5, 6, 9])
def test_no_stage_is_given_back_before_its_data_is_there(trial, late):
    assert trial(8, 40, 3, 6, 2, late) == 0
