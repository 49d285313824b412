"""The record of kernel attributes (csrc/tms_attr.cuh): the CUDA runtime keeps a
kernel's shared-memory limit per device, so every context sets what its device
needs, once, and a refusal is not taken for done."""
import glob
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nissa_b200", "csrc")

PROGRAM = r"""
#include "tms_attr.cuh"
#include <cassert>
enum Status { OK = 0, REFUSED = 1 };
int main()
{
  int kernel[2], calls[2] = {0, 0};
  tms_int::KernelAttrs ctx[2]; // contexts on two devices
  auto set = [&](int c, int k, int attr, int value, Status answer) {
    return ctx[c].once(&kernel[k], attr, value, [&] { ++calls[c]; return answer; });
  };
  for (int rep = 0; rep < 3; rep++)
    for (int c = 0; c < 2; c++) assert(set(c, 0, 8, 66560, OK) == OK);
  assert(calls[0] == 1 && calls[1] == 1);                       // once on each device
  assert(set(0, 0, 9, 100, OK) == OK && calls[0] == 2);         // another attribute
  assert(set(0, 1, 8, 66560, REFUSED) == REFUSED && calls[0] == 3);
  assert(set(0, 1, 8, 66560, OK) == OK && calls[0] == 4);       // a refusal is tried again
  assert(set(0, 1, 8, 66560, REFUSED) == OK && calls[0] == 4);  // done
  assert(set(0, 1, 8, 70000, OK) == OK && calls[0] == 5);       // another value
  assert(set(0, 0, 8, 66560, REFUSED) == OK && calls[0] == 5 && calls[1] == 1);
  return 0;
}
"""


def test_attributes_are_set_once_per_context(tmp_path):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)])
    subprocess.check_call([str(exe)])


def test_every_launch_sets_attributes_through_the_record():
    calls = []
    for f in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = open(f).read()
        assert not re.search(r"static[^;]*cudaFuncSetAttribute", text), f
        calls += re.findall(r"cudaFuncSetAttribute\(", text)
    assert len(calls) == 1  # kernel_attr
