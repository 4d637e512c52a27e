"""The rule that keeps cooperative launches away from serving loops
(csrc/loop_gate.h), run on the host with stand-ins for the launches."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "madmax_b200", "csrc")

MAIN = r"""
#include <atomic>
#include <chrono>
#include <thread>
#include "loop_gate.h"
using namespace sp;

int main() {
  LoopGate gate;
  bool taken = false;
  // none counts: the launch is made, and its error comes back
  if (gate.launch_alone([] { return 5; }, &taken) != 5 || !taken) return 1;
  // a loop on its way: a launch asked for meanwhile waits for the count, and is
  // not made
  std::atomic<int> made{0}, asked{0};
  bool meanwhile = true;
  std::thread other;
  const int rc = gate.start_loop([&] {
    other = std::thread([&] {
      gate.launch_alone([&] { return made++, 0; }, &meanwhile);
      asked = 1;
    });
    std::this_thread::sleep_for(std::chrono::milliseconds(100));
    return asked.load() ? 9 : 0;
  });
  other.join();
  if (rc || meanwhile || made.load()) return 2;
  // two loops, then one, then none
  if (gate.start_loop([] { return 0; })) return 3;
  gate.stop_loop();
  if (gate.launch_alone([&] { return made++, 0; }, &taken) || taken || made.load()) return 4;
  gate.stop_loop();
  // a loop that could not be launched does not count
  if (gate.start_loop([] { return 7; }) != 7) return 5;
  if (gate.launch_alone([&] { return made++, 0; }, &taken) || !taken || made.load() != 1) return 6;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_no_cooperative_launch_behind_a_loop(tmp_path):
    src, exe = tmp_path / "gate.cpp", tmp_path / "gate"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
