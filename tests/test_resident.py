"""Launch limits per device (resident.hpp), built with the host compiler on a runtime that records the
calls: the shared-memory limit is raised and the occupancy asked on each device that a kernel is
launched on, once, and errors are returned."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "meltpooldg_b200",
                    "csrc")

RUNTIME = r"""
#pragma once
#include <stddef.h>
enum cudaError_t { cudaSuccess, cudaErrorInvalidDevice, cudaErrorLaunchOutOfResources, cudaErrorFake };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize, cudaDevAttrMultiProcessorCount };
static int device, attribute_calls[64], limit[64], occupancy_calls[64];
static cudaError_t next_error = cudaSuccess;
static int resident = 3;
inline cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
template <typename K> cudaError_t cudaFuncSetAttribute(K, int, int bytes)
{
  if (next_error != cudaSuccess) return next_error;
  ++attribute_calls[device];
  limit[device] = bytes;
  return cudaSuccess;
}
template <typename K>
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, K, int, size_t)
{
  ++occupancy_calls[device];
  *n = resident;
  return cudaSuccess;
}
inline cudaError_t cudaDeviceGetAttribute(int *v, int, int d) { *v = 100 + d; return cudaSuccess; }
"""

MAIN = r"""
#include <stdio.h>
#include "cuda_runtime.h"
#include "resident.hpp"
static void kernel(int) {}
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main()
{
  using namespace mpdg;
  static ResidentBlocks blocks, small, failing;
  int b = 0;
  const int order[] = {0, 1, 0, 1, 1, 0};
  for (int d : order) {
    device = d;
    CHECK(blocks.get(kernel, 64, 52352, &b) == cudaSuccess && b == 3 * (100 + d));
    CHECK(attribute_calls[d] == 1 && limit[d] == 52352 && occupancy_calls[d] == 1);
  }
  CHECK(small.get(kernel, 64, 48 * 1024, &b) == cudaSuccess && attribute_calls[0] == 1);
  device = 64;
  CHECK(blocks.get(kernel, 64, 52352, &b) == cudaErrorInvalidDevice);
  device = 2;
  next_error = cudaErrorFake;
  CHECK(failing.get(kernel, 64, 52352, &b) == cudaErrorFake);
  next_error = cudaSuccess;
  resident = 0;
  CHECK(failing.get(kernel, 64, 52352, &b) == cudaErrorLaunchOutOfResources);
  resident = 3;
  CHECK(failing.get(kernel, 64, 52352, &b) == cudaSuccess && b == 3 * 102);
  static SharedLimit raise;
  const int others[] = {5, 6};
  for (int d : others) {
    device = d;
    CHECK(raise.raise(kernel, 70000) == cudaSuccess && limit[d] == 70000);
    CHECK(raise.raise(kernel, 60000) == cudaSuccess && limit[d] == 70000);
    CHECK(raise.raise(kernel, 90000) == cudaSuccess && limit[d] == 90000);
    CHECK(attribute_calls[d] == 2);
  }
  next_error = cudaErrorFake;
  CHECK(raise.raise(kernel, 99000) == cudaErrorFake);
  next_error = cudaSuccess;
  CHECK(raise.raise(kernel, 99000) == cudaSuccess && limit[6] == 99000);
  return 0;
}
"""


def test_limits_are_set_on_every_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", str(tmp_path), "-I", CSRC,
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_no_launch_limit_is_kept_per_process():
    """Every limit is raised through resident.hpp."""
    for f in sorted(os.listdir(CSRC)):
        if f != "resident.hpp":
            assert "cudaFuncSetAttribute" not in open(os.path.join(CSRC, f)).read(), f
