"""The lead that settles a tensor-core search covers twice what its sums can be off.

CPU: the constants of search.cuh, compiled for the host, against what bf16 pairs are off, over every mantissa.  GPU: the tensor
core's own sums against float64, from terms of one size to terms that are cut off."""
import ctypes as C
import os
import shutil
import subprocess

import pytest
import torch

from util import ROOT

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "include"),
         "-I", os.path.join(ROOT, "spherical-kv_b200", "csrc")]


def test_the_lead_covers_the_pairs(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not found")
    src, exe = tmp_path / "bound.cu", tmp_path / "bound"
    src.write_text('#include <cstdio>\n#include "search.cuh"\nusing namespace sphkv;\n'
                   'int main() { printf("%.17g %.17g %.17g %.17g", (double)kGap, kPairError, kSumError, kChainError); }\n')
    subprocess.check_call([NVCC, *FLAGS, str(src), "-o", str(exe)])
    gap, pair, sums, chains = map(float, subprocess.check_output([str(exe)], text=True).split())
    x = (torch.arange(1 << 23, dtype=torch.int32) + (127 << 23)).view(torch.float32)  # every mantissa
    hi = x.bfloat16().float()
    lo = (x - hi).bfloat16().float()
    off = ((x.double() - hi.double() - lo.double()).abs() / x.double()).max().item()
    assert 0.9 * pair < off <= pair
    assert (lo.abs() / x).max().item() <= 2.0 ** -8  # lo * lo is a product of its own: 2^-16 is more than a third of the lead
    assert sums >= 17 * 2.0 ** -25 + 2.0 ** -23 and chains >= 32 * 2.0 ** -24
    assert 2 * (2 * pair + 8 * sums + chains) < gap


SRC = r"""
#include "search.cuh"
using namespace sphkv;
// d[128][16] = sum over `n` products of a[i][128][16] b[i][16][16]^T, values that bf16 holds
__global__ void __launch_bounds__(128) sums_kernel(const float* a, const float* b, float* d, int n) {
  __shared__ __align__(128) uint8_t op[512];
  __shared__ __align__(8) unsigned long long bar_word;
  __shared__ uint32_t base_word;
  const int warp = threadIdx.x >> 5;
  const uint32_t bar = smem_u32(&bar_word);
  if (warp == 0) tmem_alloc(smem_u32(&base_word), 32);
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *(volatile uint32_t*)&base_word, mine = tmem + ((uint32_t)(32 * warp) << 16);
  bool ok = true;
  for (int i = 0; i < n && ok; ++i) {
    for (int e = threadIdx.x; e < 256; e += 128) {
      const int r = e >> 4, c = e & 15;
      *reinterpret_cast<__nv_bfloat16*>(op + (r >> 3) * 256 + (r & 7) * 16 + (c >> 3) * 128 + (c & 7) * 2) = __float2bfloat16_rn(b[i * 256 + e]);
    }
    uint32_t w[8];
    for (int e = 0; e < 8; ++e) {
      const float* row = a + (i * 128 + threadIdx.x) * 16 + 2 * e;
      const __nv_bfloat162 v = __floats2bfloat162_rn(row[0], row[1]);
      w[e] = *reinterpret_cast<const uint32_t*>(&v);
    }
    tmem_st_x8(mine + 16, w);
    tmem_wait_st();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
      if (elect_one()) {
        mma_ts(tmem, tmem + 16, smem_desc(smem_u32(op), 128, 256, 0), (1u << 4) | (1u << 7) | (1u << 10) | (2u << 17) | (8u << 24), i > 0);
        mma_commit(bar);
      }
      __syncwarp();
    }
    ok = __syncthreads_and(mbar_wait(bar, i & 1));
    tc_fence_after();
  }
  float v[16];
  tmem_ld_x16(mine, v);
  tmem_wait_ld();
  for (int e = 0; e < 16; ++e) d[threadIdx.x * 16 + e] = ok ? v[e] : __int_as_float(0x7fc00000);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 32);
}
extern "C" int run_sums(const float* a, const float* b, float* d, int n) {
  sums_kernel<<<1, 128>>>(a, b, d, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.gpu
@pytest.mark.parametrize("low", [0, -12, -18, -24, -30])
def test_tensor_core_sums(tmp_path, low):
    """four products of 16 terms with exponents from 0 down to `low`: each loses at most 17 x 2^-25 of its largest addend and one
    place of the fp32 sum"""
    (tmp_path / "sums.cu").write_text(SRC)
    subprocess.check_call([NVCC, *FLAGS, "-shared", "-Xcompiler", "-fPIC", str(tmp_path / "sums.cu"), "-o", str(tmp_path / "sums.so")])
    lib = C.CDLL(str(tmp_path / "sums.so"))
    lib.run_sums.argtypes = [C.c_void_p] * 3 + [C.c_int]
    g = torch.Generator().manual_seed(-low)
    n = 4
    a = torch.randn(n, 128, 16, generator=g).bfloat16().float()
    a *= 2.0 ** torch.randint(low, 1, a.shape, generator=g).float()
    a[:, ::2] = a[:, ::2].abs()  # of one sign: what is cut off adds up
    b = (1 + torch.rand(n, 16, 16, generator=g)).bfloat16().float()
    d = torch.empty(128, 16, device="cuda")
    ad, bd = a.cuda(), b.cuda()
    assert lib.run_sums(ad.data_ptr(), bd.data_ptr(), d.data_ptr(), n) == 0
    terms = a.double()[:, :, None, :] * b.double()[:, None, :, :]  # [n, 128, 16, 16]
    part = terms.sum(3).cumsum(0)
    largest = torch.maximum(terms.abs().amax(3), torch.cat([part[:1] * 0, part[:-1].abs()]))
    bound = (17 * 2.0 ** -25 * largest + 2.0 ** -23 * torch.maximum(part.abs(), largest)).sum(0)
    assert ((d.cpu().double() - part[-1]).abs() <= bound).all()
