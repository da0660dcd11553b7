"""Host-side launch rules of the library, compiled on their own with the host compiler."""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynlplus_b200", "csrc")


def run_cpp(tmp_path, body):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(body.lstrip())
    subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_a_kernel_attribute_is_set_once_on_each_device(tmp_path):
    run_cpp(tmp_path, r"""
#include <cassert>
#include <initializer_list>
#include "per_device.h"
int main() {
  std::atomic<uint64_t> a{0}, b{0};
  int calls[70] = {0};
  bool ok = true;
  auto use = [&](std::atomic<uint64_t> &d, int dev) { return dlp::once_per_device(d, dev, [&] { ++calls[dev]; return ok; }); };
  for (int k = 0; k < 3; ++k)
    for (int dev : {0, 1, 63}) assert(use(a, dev));
  assert(calls[0] == 1 && calls[1] == 1 && calls[63] == 1);
  assert(use(b, 1) && calls[1] == 2);          // another kernel
  ok = false;
  assert(!use(a, 2) && !use(a, 2) && calls[2] == 2);  // a refusal is asked again
  assert(use(a, 0) && calls[0] == 1);
  ok = true;
  assert(use(a, 2) && use(a, 2) && calls[2] == 3);
  assert(use(a, 69) && use(a, 69) && calls[69] == 2);  // past the bits: set every time
}
""")


def test_no_kernel_attribute_is_set_once_per_process():
    """cudaFuncSetAttribute acts on the current device: it is called where the devices are told apart only."""
    where = [(os.path.basename(f), n) for f in glob.glob(os.path.join(CSRC, "*.cu*"))
             for n in [len(re.findall(r"cudaFuncSetAttribute\(", open(f).read()))] if n]
    assert where == [("common.cuh", 1)]
