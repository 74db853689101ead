"""Kernel attributes are set once on each device, not once in a process."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "them_bones_b200", "csrc")


def test_every_launcher_sets_its_kernels_attributes_by_device():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        assert not re.search(r"static bool \w+ = false;", text), name          # a flag of the process
        outside = re.sub(r"BONES_ONCE\(\w+, \{.*?\n *\}\);", "", text, flags=re.S)
        if "struct NoAllocDevice" in text:                                        # keeps its own table by device
            outside = re.sub(r"static int noalloc_setup\(.*?\n\}", "", outside, flags=re.S)
        assert "cudaFuncSetAttribute" not in outside, name


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_once_on_each_device(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text('''
#include "per_device.h"
#include <cstdio>
static bones::OncePerDevice once;
int main() {
  int calls = 0;
  auto fine = [&] { ++calls; return 0; };
  auto fails = [&] { ++calls; return 7; };
  if (once(0, fails) != 7 || calls != 1) return 1;            // an error is handed on, and the next call tries again
  if (once(0, fine) || calls != 2 || once(0, fine) || calls != 2) return 2;
  if (once(1, fine) || calls != 3 || once(1, fails) || calls != 3) return 3;      // another device has its own turn
  if (once(63, fine) || calls != 4 || once(63, fine) || calls != 4) return 4;
  const int past[] = {64, 1000, -1};                          // past the table: every time
  for (int dev : past) {
    const int before = calls;
    if (once(dev, fine) || once(dev, fine) || calls != before + 2) return 5;
  }
  return 0;
}
''')
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
