"""GPU: a wait on an mbarrier phase that nobody completes gives up within about a second; what a driver warp awaits
before it leaves -- its copies and its products -- is answered at once when nothing is in flight."""
import ctypes as C
import os
import subprocess

import pytest

from util import ROOT

pytestmark = pytest.mark.gpu

SRC = r"""
#include "tcgen05.cuh"
__device__ bool drained(uint32_t b) {  // the end of a driver that gave up, with no copy and no product outstanding
  sphkv::cp_async_wait_all();
  __syncwarp();
  if (sphkv::elect_one()) sphkv::mma_commit(b);
  __syncwarp();
  return sphkv::mbar_wait(b, 0);
}
__global__ void wait_kernel(unsigned long long* out, int drain) {
  __shared__ __align__(8) unsigned long long bar;
  const uint32_t b = sphkv::smem_u32(&bar);
  if (threadIdx.x == 0) sphkv::mbar_init(b, 1);
  __syncwarp();
  unsigned long long t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  const bool ok = drain ? drained(b) : sphkv::mbar_wait(b, 0);
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
  if (threadIdx.x == 0) { out[0] = ok; out[1] = t1 - t0; }
}
extern "C" int run_wait(unsigned long long* host, int drain) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
  wait_kernel<<<1, 32>>>(d, drain);
  const int rc = (int)cudaMemcpy(host, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return rc;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    (d / "wait.cu").write_text(SRC)
    pkg_dir = os.path.join(ROOT, "spherical-kv_b200")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                           "-fPIC", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(pkg_dir, "csrc"),
                           str(d / "wait.cu"), "-o", str(d / "wait.so")])
    lib = C.CDLL(str(d / "wait.so"))

    def call(drain):
        out = (C.c_uint64 * 2)()
        assert lib.run_wait(out, drain) == 0
        return int(out[0]), int(out[1])
    return call


def test_a_lost_phase_ends_the_wait_in_about_a_second(run):
    ok, ns = run(0)
    assert not ok
    assert 5e6 <= ns <= 4e9, ns  # not sooner than any work of a CTA takes, not later than a host should wait


def test_nothing_in_flight_is_awaited_at_once(run):
    ok, ns = run(1)
    assert ok and ns <= 1e6, ns
