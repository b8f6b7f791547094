"""A residue GEMM that fails is not repeated on a C it may have changed.

``gemm`` of csrc/dense_multi.cuh may fall back to FP64 tiles only when the scratch
is too small, which rg_dense finds before its first launch.  The test compiles that
header against a stand-in for rg_dense that returns a chosen status and counts the
launches (none of which needs a GPU)."""
import os
import subprocess

import pytest

from emustack_b200 import _lib
from emustack_b200.build import ARCH, CSRC, FLAGS, nvcc

EMU_E_CUDA = 7
SRC = r'''
#include <cstdio>
#include <cstdlib>
#include "dense_multi.cuh"
static int g_status, g_launches;
namespace emu {
int sm_count() { return 148; }
void note_launch(int n) { g_launches += n; }
int rg_dense(const RgDense &, void *, size_t, cudaStream_t) { return g_status; }
size_t rg_dense_scratch(int, int, int, int) { return 1 << 20; }
}
int main(int, char **argv) {
  g_status = atoi(argv[1]);
  int status = EMU_OK;
  const RgScratch rg{(void *)4096, 1 << 20, &status};
  cd *p = (cd *)65536;
  for (int i = 0; i < 2; ++i) {
    gemm(512, 512, 512, cd{-1.0, 0.0}, p, 0, 512, p, 0, 512, cd{1.0, 0.0}, p, 0, 512, 1, rg, nullptr);
    if (i == 0) g_status = atoi(argv[2]);
  }
  printf("%d %d\n", g_launches, status);
}
'''


@pytest.fixture(scope='module')
def prog(tmp_path_factory):
    d = tmp_path_factory.mktemp('gemm')
    (d / 'g.cu').write_text(SRC)
    out = str(d / 'g')
    r = subprocess.run([nvcc()] + ARCH + FLAGS + ['-I' + CSRC, '-cudart', 'static', '-o', out, str(d / 'g.cu')],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize('first,second,launches,status', [
    (_lib.EMU_OK, _lib.EMU_OK, 0, _lib.EMU_OK),
    (_lib.EMU_E_WORKSPACE, _lib.EMU_E_WORKSPACE, 2, _lib.EMU_OK),   # FP64 tiles instead
    (EMU_E_CUDA, _lib.EMU_OK, 0, EMU_E_CUDA),             # partly written C: an error, no second product
    (_lib.EMU_E_ARG, EMU_E_CUDA, 0, _lib.EMU_E_ARG),           # the first error is the one reported
])
def test_only_a_small_scratch_falls_back(prog, first, second, launches, status):
    r = subprocess.run([prog, str(first), str(second)], capture_output=True, text=True,
                       env=dict(os.environ, CUDA_VISIBLE_DEVICES=''))
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == [str(launches), str(status)]
