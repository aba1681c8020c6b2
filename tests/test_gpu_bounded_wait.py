"""GPU: a wait on an mbarrier phase that nobody completes gives up within about a second."""
import ctypes as C
import os
import subprocess

import pytest

from util import ROOT

pytestmark = pytest.mark.gpu

SRC = r"""
#include "tcgen05.cuh"
__global__ void wait_kernel(unsigned long long* out) {
  __shared__ __align__(8) unsigned long long bar;
  const uint32_t b = sphkv::smem_u32(&bar);
  if (threadIdx.x == 0) sphkv::mbar_init(b, 1);
  __syncwarp();
  unsigned long long t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  const bool ok = sphkv::mbar_wait(b, 0);
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
  if (threadIdx.x == 0) { out[0] = ok; out[1] = t1 - t0; }
}
extern "C" int run_wait(unsigned long long* host) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 16) != cudaSuccess) return 1;
  wait_kernel<<<1, 32>>>(d);
  const int rc = (int)cudaMemcpy(host, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return rc;
}
"""


def test_a_lost_phase_ends_the_wait_in_about_a_second(tmp_path):
    src, so = tmp_path / "wait.cu", tmp_path / "wait.so"
    src.write_text(SRC)
    pkg_dir = os.path.join(ROOT, "spherical-kv_b200")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                           "-fPIC", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(pkg_dir, "csrc"), str(src), "-o", str(so)])
    out = (C.c_uint64 * 2)()
    assert C.CDLL(str(so)).run_wait(out) == 0
    assert out[0] == 0
    assert 5e6 <= out[1] <= 4e9, out[1]  # ns: not sooner than any work of a CTA takes, not later than a host should wait
