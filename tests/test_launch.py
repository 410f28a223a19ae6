"""The kernels' limits of dynamic shared memory (lm_launch.cu), on the CPU: the
file is compiled against a runtime of the test's own, which keeps the limits and
lets the threads meet where they could lose one another's."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <thread>
#include "lm_internal.h"

static thread_local int t_dev = 0;
static std::mutex g_mu;
static std::map<std::pair<const void *, int>, int> g_limit;
static std::atomic<int> g_sets{0}, g_hold{0}, g_applied{0};

extern "C" cudaError_t cudaGetDevice(int *d) { *d = t_dev; return cudaSuccess; }
static thread_local cudaError_t t_last = cudaSuccess;
extern "C" cudaError_t cudaGetLastError() {
  const cudaError_t e = t_last;
  t_last = cudaSuccess;
  return e;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void *k, cudaFuncAttribute,
                                            int v) {
  g_sets++;
  if (v > 227 << 10) return t_last = cudaErrorInvalidValue;
  // the call that is to lose: applied after the other thread's, if that one
  // comes through meanwhile
  if (v == g_hold)
    for (int i = 0; i < 300 && !g_applied; ++i)
      std::this_thread::sleep_for(std::chrono::milliseconds(1));
  std::lock_guard<std::mutex> lock(g_mu);
  g_limit[{k, t_dev}] = v;
  if (v != g_hold) g_applied = 1;
  return cudaSuccess;
}
extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(
    int *n, const void *, int, size_t) {
  *n = 2;
  return cudaSuccess;
}

static int limit(const void *k, int dev) {
  std::lock_guard<std::mutex> lock(g_mu);
  auto it = g_limit.find({k, dev});
  return it == g_limit.end() ? 48 * 1024 : it->second;
}
// a launch: prepared, and refused by the driver above the kernel's limit
static void launch(const void *k, lm::LaunchCache &c, int smem) {
  cudaError_t err;
  if (lm::prepare_launch(k, c, smem, 256, &err) != 2 || err != cudaSuccess ||
      limit(k, t_dev) < smem) {
    printf("refused: %d bytes on device %d, limit %d\n", smem, t_dev,
           limit(k, t_dev));
    exit(1);
  }
}
"""


def _run(tmp_path, body):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    src = tmp_path / "launches.cpp"
    src.write_text(FAKE + "int main() {\n" + body + "\n  return 0;\n}\n")
    csrc = os.path.join(ROOT, "libmarshal_gb300", "csrc")
    exe = str(tmp_path / "launches")
    subprocess.check_call(
        [cxx, "-std=c++17", "-O1", "-I", csrc, "-I",
         os.path.join(cuda, "include"), str(src), "-x", "c++",
         os.path.join(csrc, "lm_launch.cu"), "-o", exe, "-lpthread"])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_first_launches_of_two_threads(tmp_path):
    """Two threads launch one kernel for the first time, the one with less
    shared memory held back in its call of the driver: the larger limit is the
    one that stays."""
    _run(tmp_path, r"""
  static lm::LaunchCache c;
  static char k;
  g_hold = 70 << 10;
  std::thread less([] {
    cudaError_t err;
    lm::prepare_launch(&k, c, 70 << 10, 256, &err);
  });
  while (!g_sets) std::this_thread::yield();
  std::thread more([] {
    cudaError_t err;
    lm::prepare_launch(&k, c, 108 << 10, 256, &err);
  });
  less.join();
  more.join();
  launch(&k, c, 108 << 10);
  launch(&k, c, 70 << 10);
  launch(&k, c, 108 << 10);""")


def test_limit_only_grows(tmp_path):
    _run(tmp_path, r"""
  static lm::LaunchCache c;
  static char k;
  for (int kb : {1, 60, 100, 50, 100, 227, 60}) launch(&k, c, kb << 10);
  if (g_sets != 3) return printf("%d calls of the driver\n", (int)g_sets), 1;""")


def test_devices_have_their_own(tmp_path):
    """Devices past the eighth do not pass for one of the first eight."""
    _run(tmp_path, r"""
  static lm::LaunchCache c;
  static char k;
  for (int dev : {0, 8, 15, 7, 63}) {
    t_dev = dev;
    launch(&k, c, 100 << 10);
  }""")


def test_a_refused_limit_leaves_no_error(tmp_path):
    """A size that the driver refuses is reported by its caller alone: the error
    is not left for the check of the next launch to find."""
    _run(tmp_path, r"""
  static lm::LaunchCache c;
  static char k;
  cudaError_t err;
  if (lm::prepare_launch(&k, c, 300 << 10, 256, &err) != 0 ||
      err != cudaErrorInvalidValue || cudaGetLastError() != cudaSuccess)
    return puts("an error is pending"), 1;
  launch(&k, c, 100 << 10);
  if (lm::grow_smem_limit(&k, 300 << 10) != cudaErrorInvalidValue ||
      cudaGetLastError() != cudaSuccess)
    return puts("an error is pending"), 1;
  launch(&k, c, 200 << 10);""")
