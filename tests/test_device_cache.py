"""The host code's memory of what a device answered, compiled and run here."""
import re
import shutil
import subprocess

import pytest

from sonicboom_b200.csrc.build import ARCH_FLAGS, SRC_DIR, BuildError, _nvcc

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "device_cache.h"
int main() {
  static SbDeviceCache c;
  int asked = 0;
  auto ask = [&](int v) { return [&asked, v] { ++asked; return v; }; };
  if (c.get(0, ask(-1)) != -1 || c.get(0, ask(18)) != 18) return 1;      // a failed query is asked again
  if (c.get(0, ask(7)) != 18 || asked != 2) return 2;                    // an answer is kept
  if (c.get(1, ask(0)) != 0 || c.get(1, ask(5)) != 0) return 3;          // for its device only, also when it is none
  if (c.get(-1, ask(4)) != 4 || c.get(-1, ask(3)) != 3 || c.get(SbDeviceCache::DEVICES, ask(2)) != 2) return 4;
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] {
      for (int d = 2; d < 60; ++d) wrong += c.get(d, [d] { return 100 + d; }) != 100 + d;
    });
  for (auto& t : threads) t.join();
  return wrong ? 5 : 0;
}
"""


def test_device_cache(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(SRC_DIR), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t"),
                    "-pthread"], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0

ONCE = r"""
#include <cuda_runtime.h>
static int g_device = 0, g_fails = 0, g_set[2] = {0, 0}, g_cleared = 0;
static cudaError_t fake_device(int* d) { *d = g_device; return cudaSuccess; }
static cudaError_t fake_attribute(const void*, cudaFuncAttribute, int) {
  if (g_fails > 0) { --g_fails; return cudaErrorInvalidValue; }
  ++g_set[g_device];
  return cudaSuccess;
}
static cudaError_t fake_last() { ++g_cleared; return cudaSuccess; }
#define cudaGetDevice fake_device
#define cudaFuncSetAttribute(k, a, v) fake_attribute((const void*)(k), a, v)
#define cudaGetLastError fake_last
#include "common.cuh"
template <int N> __global__ void some_kernel() {}
int main() {
  g_fails = 1;
  if (sb_allow_shared<some_kernel<1>>(1024) == cudaSuccess || g_cleared != 1) return 1;       // reported, and cleared
  for (int i = 0; i < 3; ++i)
    if (sb_allow_shared<some_kernel<1>>(1024) != cudaSuccess) return 2;                       // tried again, then kept
  if (g_set[0] != 1) return 3;
  g_device = 1;
  if (sb_allow_shared<some_kernel<1>>(1024) != cudaSuccess || g_set[1] != 1) return 4;        // another device
  g_device = 0;
  if (sb_allow_shared<some_kernel<2>>(1024) != cudaSuccess || g_set[0] != 2) return 5;        // another kernel
  return g_cleared == 1 ? 0 : 6;
}
"""


def test_a_kernels_attributes_are_set_once_per_device(tmp_path):
    try:
        nvcc = _nvcc()
    except BuildError:
        pytest.skip("no nvcc")
    (tmp_path / "t.cu").write_text(ONCE)
    subprocess.run([nvcc, *ARCH_FLAGS, "-std=c++17", "-I", str(SRC_DIR), str(tmp_path / "t.cu"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


RESIDENT = r"""
#include <cuda_runtime.h>
static int g_bad = 0, g_last = 0;                  // which query fails; the runtime's last error
static cudaError_t answer(int query) { return g_bad == query ? (cudaError_t)(g_last = cudaErrorInvalidValue) : cudaSuccess; }
static cudaError_t fake_device(int* device) { *device = 0; return answer(1); }
static cudaError_t fake_blocks(int* n, const void*, int, size_t) { *n = 2; return answer(2); }
static cudaError_t fake_attribute(int* n, cudaDeviceAttr, int) { *n = 148; return answer(3); }
static cudaError_t fake_last() { const int e = g_last; g_last = 0; return (cudaError_t)e; }
#define cudaGetDevice fake_device
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, k, t, s) fake_blocks(n, (const void*)(k), t, s)
#define cudaDeviceGetAttribute fake_attribute
#define cudaGetLastError fake_last
#include "gemm_mma.cu"
int sb_check_linear_args(const char*, int, int, int, int, const void*, const float*, int) { return 0; }
int main() {
  for (g_bad = 2; g_bad <= 3; ++g_bad)
    if (skinny_resident<gemm_skinny_stream_kernel<5, float>>() != 0 || g_last) return g_bad;
  g_bad = 0;
  return skinny_resident<gemm_skinny_stream_kernel<5, float>>() == 296 ? 0 : 4;
}
"""


def test_a_failed_occupancy_query_leaves_no_error_for_the_launch_that_follows(tmp_path):
    """The weight-streaming product then runs a block per group, and that launch is checked with the runtime's last error."""
    try:
        nvcc = _nvcc()
    except BuildError:
        pytest.skip("no nvcc")
    (tmp_path / "t.cu").write_text(RESIDENT)
    subprocess.run([nvcc, *ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-O0", "-Xptxas", "-O0", "-I", str(SRC_DIR),
                    str(tmp_path / "t.cu"), str(SRC_DIR / "error.cu"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


@pytest.mark.parametrize("path", sorted(SRC_DIR.glob("*.cu*")), ids=lambda p: p.name)
def test_no_attribute_or_cluster_count_is_kept_for_all_devices(path):
    """A flag or number of the whole process beside a query or attribute of one device."""
    kept = re.compile(r"^ +static (?:bool|int) \w+(?:\[\d+\])? = [^;]*;\n(?:.*\n){0,4}?.*(?:cudaFuncSetAttribute|cudaOccupancy)", re.M)
    assert not kept.findall(path.read_text())
