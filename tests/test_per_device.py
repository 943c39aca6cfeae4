"""What is remembered per device (`csrc/per_device.h`): host code, compiled here on its own."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

int main() {
  hl::PerDevice pairs, allowed;
  int asked = 0;
  auto ask = [&](int answer) { return [&asked, answer] { ++asked; return answer; }; };
  // each device is asked once and keeps its own answer
  assert(pairs.value(0, ask(74)) == 74 && pairs.value(1, ask(70)) == 70 && pairs.value(0, ask(9)) == 74 && pairs.value(1, ask(9)) == 70);
  assert(asked == 2);
  // no answer is not remembered, nor is one for an ordinal past the table
  assert(pairs.value(2, ask(0)) == 0 && pairs.value(2, ask(66)) == 66 && pairs.value(2, ask(9)) == 66);
  assert(pairs.value(64, ask(5)) == 5 && pairs.value(64, ask(6)) == 6 && pairs.value(-1, ask(7)) == 7);
  // an action is repeated until it has succeeded on that device
  int runs = 0;
  auto act = [&](int result) { return [&runs, result] { ++runs; return result; }; };
  assert(allowed.once(3, act(2)) == 2 && allowed.once(3, act(0)) == 0 && allowed.once(3, act(2)) == 0 && runs == 2);
  assert(allowed.once(4, act(0)) == 0 && runs == 3);
  // threads
  hl::PerDevice shared;
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 100000; ++i) assert(shared.value((t + i) % 5, [&] { return 100 + (t + i) % 5; }) == 100 + (t + i) % 5);
    });
  for (auto& t : threads) t.join();
  puts("per device ok");
}
"""


def test_values_and_actions_are_per_device(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{ROOT / 'heirloom_b200' / 'csrc'}", "-o", str(exe), str(tmp_path / "main.cpp")],
                   check=True)
    assert "per device ok" in subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout
