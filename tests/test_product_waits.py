"""CPU: what a warp that issues tensor-core products still awaits after a wait has run out.

The waits of the search kernels (ProductWaits) are compiled for the host and driven by a model of a barrier: a
batch of products is issued, then awaited; the model lets a batch be late by any number of waits.  When the warp leaves
and its last wait was answered, nothing that it issued may be outstanding: its shared and tensor memory are given back."""
import os
import shutil
import subprocess

import pytest

from util import ROOT

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "tcgen05.cuh"
struct Barrier {  // one arrival completes a phase; products complete in order
  int issued = 0, done = 0, late = 0;
  bool wait(unsigned parity) {  // true: the phase with this parity has completed, as mbarrier.try_wait.parity
    if (done < issued && late-- <= 0) ++done;
    return ((unsigned)done & 1u) != parity;
  }
};
int main() {
  int bad = 0, answered = 0;
  for (int seed = 0; seed < 20000; ++seed) {
    srand(seed);
    Barrier b;
    sphkv::ProductWaits w;
    bool last = true;
    auto wait = [&](unsigned parity) { return last = b.wait(parity); };
    const int batches = 1 + rand() % 6;
    b.issued = 1;
    for (int i = 0; i < batches; ++i) {
      if (rand() % 3 == 0 && b.late <= 0) b.late = 1 + rand() % 2;
      w.next(wait);
      if (i + 1 < batches && !w.lost) ++b.issued;
    }
    w.leave(wait);
    answered += last;
    bad += last && b.done != b.issued;
    bad += !w.lost && b.done != b.issued;
  }
  printf("%d %d\n", bad, answered);
  return 0;
}
"""


def test_nothing_is_outstanding_after_a_lost_wait(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src, exe = tmp_path / "waits.cu", tmp_path / "waits"
    src.write_text(SRC)
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(ROOT, "spherical-kv_b200", "csrc"), str(src), "-o", str(exe)])
    bad, answered = map(int, subprocess.check_output([str(exe)], text=True).split())
    assert answered > 5000 and bad == 0
