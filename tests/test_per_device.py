"""What a launcher does once per device: again on every further device, and again after it failed."""

import re
import shutil
import subprocess
from pathlib import Path

KERNELS = Path(__file__).resolve().parent.parent / "kv_cache_optimization_for_llm_b200" / "csrc" / "kernels"

PROGRAM = """
#include "per_device.h"
#include <cstdio>
int main() {
  OncePerDevice once;
  int calls = 0, answer = 7;
  auto set = [&] { ++calls; return answer; };
  const int failed = once(0, set), first_calls = calls;          // fails: not remembered
  answer = 0;
  once(0, set), once(0, set);                                      // done, then remembered
  const int one_device = calls;
  once(1, set), once(63, set), once(1, set), once(0, set);         // every further device once
  const int three_devices = calls;
  once(64, set), once(64, set), once(-1, set);                     // beyond what is remembered
  std::printf("%d %d %d %d %d", failed, first_calls, one_device, three_devices, calls);
}
"""


def test_once_per_device(tmp_path):
    source, program = tmp_path / "once.cpp", tmp_path / "once"
    source.write_text(PROGRAM)
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-I", str(KERNELS), str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)], capture_output=True, text=True, check=True).stdout == "7 1 2 4 7"


def test_no_launcher_remembers_a_kernels_attributes_for_all_devices():
    for path in sorted(KERNELS.glob("*.cu*")):
        for found in re.finditer(r"static (bool|int) (\w+) = (false|0);", path.read_text()):
            assert found.group(2) == "max_threads", (path.name, found.group(0))      # (registers of a kernel: the same on every device)
