"""CPU check of csrc/smem_limit.h with a stand-in for the CUDA runtime: the
shared-memory limit of a kernel belongs to one device, so it is raised on every
device that launches the kernel, once; a failure is returned and not kept.
And every kernel that needs it goes through there."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mscomplex_gb300", "csrc")

RUNTIME = r"""
#pragma once
#include <mutex>
#include <set>
#include <tuple>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
inline thread_local int fake_device = 0;
inline int fake_calls = 0, fake_failures = 0;
inline std::mutex fake_lock;
inline std::set<std::tuple<int, const void *, int>> fake_limits;  // device, kernel, bytes
inline cudaError_t cudaGetDevice(int *d) { *d = fake_device; return cudaSuccess; }
template <class K> cudaError_t cudaFuncSetAttribute(K *k, cudaFuncAttribute, int bytes) {
  std::lock_guard<std::mutex> g(fake_lock);
  ++fake_calls;
  if (fake_failures > 0) { --fake_failures; return cudaErrorInvalidValue; }
  fake_limits.insert({fake_device, (const void *)k, bytes});
  return cudaSuccess;
}
"""

PROGRAM = r"""
#include "smem_limit.h"
#include <cstdio>
#include <thread>
#include <vector>
static int fails = 0;
static void expect(bool ok, const char *what) { if (!ok) { std::printf("FAIL %s\n", what); ++fails; } }
static void k1(int) {}
static void k2(float, int) {}
static cudaError_t launch(int device) {
  static dmsc::SmemLimit limit;
  fake_device = device;
  return limit.raise(100000, k1, k2);
}
static bool raised(int d) { return fake_limits.count({d, (const void *)k1, 100000}) && fake_limits.count({d, (const void *)k2, 100000}); }

int main() {
  expect(launch(0) == cudaSuccess && raised(0) && fake_calls == 2, "the first device");
  expect(launch(1) == cudaSuccess && raised(1) && fake_calls == 4, "a second device of the process");
  expect(launch(0) == cudaSuccess && launch(1) == cudaSuccess && fake_calls == 4, "once per device");
  fake_failures = 1;
  expect(launch(5) == cudaErrorInvalidValue && !raised(5), "a failure is returned");
  expect(launch(5) == cudaSuccess && raised(5), "and tried again");
  expect(launch(63) == cudaSuccess && raised(63) && launch(64) == cudaSuccess && raised(64) && launch(70) == cudaSuccess && raised(70),
         "many devices");
  std::vector<std::thread> t;
  for (int i = 0; i < 8; ++i) t.emplace_back([i] { expect(launch(10 + i % 4) == cudaSuccess && raised(10 + i % 4), "threads"); });
  for (auto &x : t) x.join();
  return fails != 0;
}
"""


def test_limit_is_raised_on_every_device(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", str(tmp_path), "-I", CSRC, str(src), "-o", str(exe)],
                   check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_every_raised_limit_goes_through_it():
    users = [f for f in sorted(os.listdir(CSRC)) if "cudaFuncSetAttribute(" in open(os.path.join(CSRC, f)).read()]
    assert users == ["smem_limit.h"]
