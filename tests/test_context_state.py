"""State the library keeps per CUDA context (csrc/xc_once.h): what was set or
allocated once must be so again on another device and after a
cudaDeviceReset, and a failure must not be remembered."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "xc_once.h"

int main() {
  xc::PerKey<int> a;
  int* p = nullptr;
  int calls = 0;
  // a failure is passed on and not remembered; a second key is made anew
  if (a.get(1, &p, [&](int*) { ++calls; return 7; }) != 7 || p) return 1;
  if (a.get(1, &p, [&](int* v) { ++calls; *v = 10; return 0; }) != 0 || *p != 10 || calls != 2) return 2;
  int* first = p;
  if (a.get(2, &p, [&](int* v) { ++calls; *v = 20; return 0; }) != 0 || *p != 20 || calls != 3) return 3;
  if (a.get(1, &p, [&](int*) { ++calls; return 7; }) != 0 || p != first || *p != 10 || calls != 3) return 4;
  // many threads, three keys: made once each
  xc::PerKey<int> b;
  std::atomic<int> made{0}, bad{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 16; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 2000; ++i) {
        int* q = nullptr;
        const int key = (t + i) % 3;
        if (b.get(key, &q, [&](int* v) { made.fetch_add(1); *v = 100 + key; return 0; }) != 0 || *q != 100 + key) bad.fetch_add(1);
      }
    });
  for (auto& t : ts) t.join();
  if (made != 3 || bad != 0) return 5;
  std::printf("ok\n");
  return 0;
}
"""


def test_state_per_key(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "once.cpp"
    src.write_text(PROBE)
    exe = tmp_path / "once"
    subprocess.run([gxx, "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "xcore.jl_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)


# forward (more than 48 KB of shared memory) and weight gradient of 128 channels, all memory by the runtime itself,
# before and after the process gives its context back
RESET = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import xcore_gb300 as xc
lib = xc.lib()
rt = ctypes.CDLL("libcudart.so.13")
B, H, W, C = 1, 8, 128, 128
rng = np.random.default_rng(0)
bf16 = lambda a: (np.ascontiguousarray(a, np.float32).view(np.uint32) >> 16).astype(np.uint16)
x, w = bf16(rng.standard_normal((B, H, W, C))), bf16(rng.standard_normal((C, 9, C)))

def put(a):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, ctypes.c_void_p(a.ctypes.data), ctypes.c_size_t(a.nbytes), 1) == 0
    return p

def calls():
    y, dw = np.zeros((B, H, W, C), np.float32), np.zeros((C, 9, C), np.float32)
    px, pw, py, pd = put(x), put(w), put(y), put(dw)
    rc = lib.xc_nn_conv3x3(px, pw, None, None, py, B, H, W, C, C, 0, None)
    assert rc == 0, lib.xc_last_error()
    rc = lib.xc_nn_conv3x3_wgrad(px, px, pd, B, H, W, C, C, None)
    assert rc == 0, lib.xc_last_error()
    for p, a in ((py, y), (pd, dw)):
        assert rt.cudaMemcpy(ctypes.c_void_p(a.ctypes.data), p, ctypes.c_size_t(a.nbytes), 2) == 0
    return y, dw

first = calls()
assert np.abs(first[0]).max() > 0 and np.abs(first[1]).max() > 0
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    for a, b in zip(first, calls()):
        assert np.array_equal(a, b)
print("ok")
"""


@pytest.mark.gpu
def test_convolutions_after_a_context_reset():
    r = subprocess.run([sys.executable, "-c", RESET, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), (r.returncode, r.stdout, r.stderr[-2000:])
