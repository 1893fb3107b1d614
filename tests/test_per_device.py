"""Kernel attributes are set on every device that a process uses, not on its first one alone."""

import re
import shutil
import subprocess

import pytest

from shrike_b200.ops import build

PROGRAM = """
#include "per_device.cuh"
#include <initializer_list>
int main() {
  PerDevice flag;
  int calls[80] = {}, fail_next = 0;
  auto on = [&](int device) { return flag.once(device, [&] { ++calls[device < 0 ? 79 : device]; return fail_next; }); };
  for (int round = 0; round < 3; ++round)
    for (int device : {0, 1, 63}) if (on(device) != 0) return 1;
  if (calls[0] != 1 || calls[1] != 1 || calls[63] != 1) return 2;   // once each, whatever another device has had
  fail_next = 7;
  if (on(2) != 7) return 3;
  fail_next = 0;
  if (on(2) != 0 || on(2) != 0 || calls[2] != 2) return 4;           // a failure is not remembered as done
  for (int round = 0; round < 2; ++round)
    for (int device : {64, -1}) if (on(device) != 0) return 5;
  if (calls[64] != 2 || calls[79] != 2) return 6;                    // devices that are not kept track of: every time
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_once_per_device(tmp_path):
    source, program = tmp_path / "once.cpp", tmp_path / "once"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-x", "c++", f"-I{build.CSRC}", str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0


def test_no_launcher_keeps_one_flag_for_all_devices():
    for path in sorted(build.CSRC.glob("*.cu")):
        text = path.read_text()
        assert not re.search(r"static\s+(bool|size_t|int)\s+\w*(configured|raised)", text), path.name
