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
    subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
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


def test_resident_kernels_run_on_as_many_blocks_as_the_device_holds(tmp_path):
    run_cpp(tmp_path, r"""
#include <cassert>
#include <vector>
#include "resident.h"
using dlp::Launch;
int main() {
  std::vector<int> grids;
  int plain = 0;
  auto on = [&](int holds, Launch beyond) {  // a device that holds `holds` blocks
    return [&grids, holds, beyond](int g) { grids.push_back(g); return g <= holds ? Launch::ok : beyond; };
  };
  auto one = [&] { ++plain; return Launch::ok; };
  auto run = [&](int grid, int holds, Launch beyond) { grids.clear(); plain = 0; return dlp::launch_resident(grid, on(holds, beyond), one); };
  assert(run(296, 296, Launch::too_large) == Launch::ok && grids == std::vector<int>{296} && plain == 0);
  assert(run(296, 40, Launch::too_large) == Launch::ok && (grids == std::vector<int>{296, 148, 74, 37}) && plain == 0);
  assert(run(3, 0, Launch::too_large) == Launch::ok && (grids == std::vector<int>{3, 1}) && plain == 1);
  assert(run(296, 0, Launch::refused) == Launch::ok && grids == std::vector<int>{296} && plain == 1);
  assert(run(296, 0, Launch::failed) == Launch::failed && grids == std::vector<int>{296} && plain == 0);
}
""")


def test_every_cooperative_launch_has_another_form():
    """cudaLaunchCooperativeKernel is called in one place, which tells a refusal from an error; its callers launch
    another form of the work or a smaller grid then."""
    where = [(os.path.basename(f), n) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
             for n in [len(re.findall(r"cudaLaunchCooperativeKernel\(", open(f).read()))] if n]
    assert where == [("common.cuh", 1)]


def test_a_host_read_waits_for_the_stream_of_the_tensors_device(monkeypatch):
    """A wait for another device's stream is that stream's own: the handle of a default stream names the current
    device's."""
    import torch
    from dynlplus_b200 import backend
    waited = []

    class Stream:
        def __init__(self, dev):
            self.dev = dev

        def synchronize(self):
            waited.append(self.dev)
    monkeypatch.setattr(backend, "have_cuda", lambda: True)
    monkeypatch.setattr(backend, "stream", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: Stream(str(dev)))
    monkeypatch.setattr(backend._lib, "call", lambda name, handle: waited.append((name, handle)))
    backend.sync()
    backend.sync(torch.device("cuda", 0))
    backend.sync("cuda")
    backend.sync(torch.device("cuda", 1))
    here = ("dlp_stream_synchronize", 0)
    assert waited == [here, here, here, "cuda:1"]


def test_host_blocks_are_kept_per_call_at_once_not_per_thread(tmp_path):
    run_cpp(tmp_path, r"""
#include <atomic>
#include <cassert>
#include <memory>
#include <thread>
#include "block_pool.h"
int main() {
  dlp::BlockPool<int> pool;
  std::atomic<int> made{0}, in{0};
  auto alloc = [&]() -> int * { ++made; return new int(0); };
  for (int t = 0; t < 100; ++t)
    std::thread([&] { int *p = pool.borrow(alloc); *p = 1; pool.give(p); }).join();
  assert(made == 1);
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&] {
      for (int k = 0; k < 2000; ++k) {
        int *p = pool.borrow(alloc);
        const int v = ++*p;
        std::this_thread::yield();
        assert(*p == v);  // nobody else has the block
        pool.give(p);
      }
    });
  for (auto &t : ts) t.join();
  assert(made >= 1 && made <= 8);
  int *none = pool.borrow([]() -> int * { return nullptr; });
  pool.give(none);
  for (int k = 0; k < 9; ++k) none = pool.borrow([]() -> int * { return nullptr; });
  assert(none == nullptr);
  pool.give(none);
  assert(pool.borrow([]() -> int * { return nullptr; }) == nullptr);
}
""")


def test_no_pinned_block_belongs_to_a_thread_of_the_amg_loop():
    src = open(os.path.join(CSRC, "amg_pcg.cu")).read()
    assert "thread_local" not in src and "BlockPool" in src
