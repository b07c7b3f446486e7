"""The bound of a relax's wait for a neighbouring plane (tlq_mg_wait.cuh): a
wait for a flag that nothing sets ends after a second, after the polls of a
short limit, or at once when another block has given up; the kernel returns
and the context stays usable."""
import ctypes as C
import os
import subprocess

import pytest

from tlaloque_gb300 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cuda_runtime.h>
#include "tlq_mg_wait.cuh"
struct Ctl { int abort; long long wait_limit; };
__global__ void k_wait(const Ctl* c, const volatile int* flag, long long* polls) {
  tlq::MgWait w;
  while (*flag == 0)
    if (w.out(c)) break;
  *polls = w.polls;
}
extern "C" int wait_once(int abort, long long limit, double* ms, long long* polls) {
  struct Mem { Ctl c; int flag; long long polls; } h = {{abort, limit < 0 ? tlq::MG_WAIT_LIMIT : limit}, 0, 0};
  Mem* d = nullptr;
  cudaEvent_t a, b;
  if (cudaMalloc(&d, sizeof h) || cudaMemcpy(d, &h, sizeof h, cudaMemcpyHostToDevice)) return 1;
  if (cudaEventCreate(&a) || cudaEventCreate(&b)) return 2;
  cudaEventRecord(a);
  k_wait<<<1, 1>>>(&d->c, &d->flag, &d->polls);
  cudaEventRecord(b);
  if (cudaEventSynchronize(b)) return 3;
  float t = 0.f;
  cudaEventElapsedTime(&t, a, b);
  *ms = t;
  if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost)) return 4;
  *polls = h.polls;
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return cudaFree(d) ? 5 : 0;
}
"""


@pytest.fixture(scope="module")
def wait_once(tmp_path_factory):
    d = tmp_path_factory.mktemp("mgwait")
    src, lib = d / "wait.cu", d / "wait.so"
    src.write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared", f"-I{build.CSRC}",
                    str(src), "-o", str(lib)], check=True)
    f = C.CDLL(str(lib)).wait_once
    f.argtypes = [C.c_int, C.c_longlong, C.POINTER(C.c_double), C.POINTER(C.c_longlong)]

    def run(abort, limit):
        ms, polls = C.c_double(), C.c_longlong()
        assert f(abort, limit, C.byref(ms), C.byref(polls)) == 0
        return ms.value, polls.value

    return run


def test_ends_after_a_second(wait_once):
    ms, polls = wait_once(0, 1 << 40)  # (more polls than fit into the time)
    assert 1000.0 <= ms < 1500.0 and polls > 256
    ms, polls = wait_once(0, -1)  # the default: whichever comes first
    assert ms < 1500.0


@pytest.mark.parametrize("limit", [0, 1, 255, 256, 257, 1000])
def test_ends_after_the_polls(wait_once, limit):
    assert wait_once(0, limit)[1] == limit + 1


def test_ends_when_another_gave_up(wait_once):
    assert wait_once(1, -1)[1] == 0
