"""A device allocation or copy that fails leaves nothing half-made behind for the
next call: csrc/host/engine.cpp on the host, over a CUDA runtime whose n-th call
fails (allocations are host memory, launches do nothing)."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import PKG, REPO

PROGRAM = r"""
#include "engine.cpp"

#include <cstdio>
#include <cstdlib>

static int calls_left = -1;  // calls of the failing kind until one fails; -1: none does
static bool fails() { return calls_left >= 0 && calls_left-- == 0; }
static bool fail_copies = false;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
  if (!fail_copies && fails()) return cudaErrorMemoryAllocation;
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (fail_copies && fails()) return cudaErrorUnknown;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "as asked"; }
}

namespace slaph {
namespace dev {
cudaError_t upload_gamma(cudaStream_t) { return cudaSuccess; }
cudaError_t upload_gamma_tc(cudaStream_t) { return cudaSuccess; }
cudaError_t momenta(double2 *, int32_t const *, int32_t, Geometry, cudaStream_t) { return cudaSuccess; }
cudaError_t phase_fixed(longlong2 *, double2 const *, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t unit_roots(double2 *, int32_t, cudaStream_t) { return cudaSuccess; }
std::vector<int2> vdaggerv_tc_tiles(std::vector<VdvFamily> const &, int32_t, int32_t, int32_t, int32_t,
                                    VdvColumns &) {
  return std::vector<int2>(1);
}
}  // namespace dev
}  // namespace slaph

using namespace slaph;

template <typename F>
static bool throws(F &&f) {
  try {
    f();
  } catch (std::exception const &) {
    return true;
  }
  return false;
}

#define EXPECT(c) \
  if (!(c)) return std::printf("line %d: %s\n", __LINE__, #c), 1

// Q1 factors that share their products: two of them with six gammas each.
static int shared_q1(int fail) {
  Schedule s;
  for (int r = 0; r < 2; ++r)
    for (int g = 0; g < 6; ++g) s.q1.push_back({0, 0, r, 1, g, 6 * r + g});
  DeviceSchedule ds;
  calls_left = fail;
  EXPECT(throws([&] { plan_shared_q1(ds, s, nullptr); }));
  calls_left = -1;
  plan_shared_q1(ds, s, nullptr);
  EXPECT(ds.x1_ready && ds.x1_max == 2 && ds.x1_batches.size() == 1);
  EXPECT(ds.x1_batches[0].n_x == 2 && ds.x1_batches[0].n_p == 12);
  auto const *x = ds.x1.as<dev::X1Inst>();
  auto const *p = ds.q1_picks.as<dev::Q1Pick>();
  EXPECT(x && p);
  EXPECT(x[1].r == 1 && x[1].r2 == 1);
  for (int k = 0; k < 12; ++k) EXPECT(p[k].x == k / 6 && p[k].gamma == k % 6 && p[k].slot == k);
  return 0;
}

// A table of operators, then a larger one that fails: neither is in place.
static int operators(int fail) {
  Engine e(slaph_dims{2, 4, 4, 4, 5, 1, 2, 2});
  std::vector<slaph_vdv_op> ops(5);
  for (int k = 0; k < 5; ++k) ops[k] = slaph_vdv_op{k, {k, 1, 0}, 0, {}};
  e.set_operators(ops.data(), 1, -1);
  calls_left = fail;
  bool const failed = throws([&] { e.set_operators(ops.data(), 5, -1); });
  calls_left = -1;
  if (!failed) return 2;  // fewer calls than that
  bool state = false;
  try {
    e.vdaggerv_build(SLAPH_MIXED);
  } catch (StateError const &) {
    state = true;
  }
  EXPECT(state);
  e.set_operators(ops.data(), 5, -1);
  return 0;
}

int main(int, char **argv) {
  fail_copies = std::atoi(argv[2]) != 0;
  int const fail = std::atoi(argv[3]);
  return argv[1][0] == 'q' ? shared_q1(fail) : operators(fail);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent / "include"
    assert os.path.isdir(cuda)
    d = tmp_path_factory.mktemp("failed_allocation")
    (d / "main.cpp").write_text(PROGRAM)
    host = PKG / "csrc" / "host"
    # what the two calls do not reach stays unresolved
    subprocess.run(["g++", "-std=c++17", "-O1", "-no-pie", f"-I{host}", f"-I{REPO / 'include'}",
                    f"-I{cuda}", str(d / "main.cpp"), str(host / "schedule.cpp"),
                    str(host / "vdv_families.cpp"), "-Wl,--unresolved-symbols=ignore-all",
                    "-o", str(d / "run")], check=True, capture_output=True)
    return lambda *a: subprocess.run([str(d / "run"), *map(str, a)], capture_output=True,
                                     text=True, timeout=60)


@pytest.mark.parametrize("copies", [0, 1], ids=["malloc", "memcpy"])
@pytest.mark.parametrize("fail", [0, 1])
def test_shared_q1_plan(program, copies, fail):
    r = program("q1", copies, fail)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("copies", [0, 1], ids=["malloc", "memcpy"])
def test_operator_table(program, copies):
    tried = 0
    for fail in range(20):
        r = program("operators", copies, fail)
        if r.returncode == 2:
            break
        assert r.returncode == 0, (fail, r.returncode, r.stdout)
        tried += 1
    assert tried >= 3
