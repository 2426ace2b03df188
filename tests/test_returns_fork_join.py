"""The fork and join of the plastic returns that run beside the next step's sort: the code of
every CUDA call of theirs reaches the caller, by its first failure, and after a failed event
record the wait is not attempted.  Compiled for the host against fakes of the two calls."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
static int calls = 0, fail_at = 0;
static cudaStream_t rec_on, waiter;
static cudaError_t fake_record(cudaEvent_t, cudaStream_t s) { rec_on = s; return ++calls == fail_at ? cudaErrorInvalidResourceHandle : cudaSuccess; }
static cudaError_t fake_wait(cudaStream_t s, cudaEvent_t, unsigned) { waiter = s; return ++calls == fail_at ? cudaErrorStreamCaptureIsolation : cudaSuccess; }
#define cudaEventRecord fake_record
#define cudaStreamWaitEvent fake_wait
#include "mpm_kernels.h"
int main() {
  mpm_b200::StepArgs a{};
  cudaStream_t st = (cudaStream_t)1;
  a.side = (cudaStream_t)2;
  for (fail_at = 0; fail_at < 3; ++fail_at)
    for (int join = 0; join < 2; ++join) {
      calls = 0;
      const cudaError_t e = join ? mpm_b200::join_side(a, st) : mpm_b200::fork_side(a, st);
      std::printf("%d %d %d %d %d\n", fail_at, join, (int)e, calls, rec_on == (join ? a.side : st) && (fail_at == 1 || waiter == (join ? st : a.side)));
    }
}
"""


def test_codes_reach_the_caller(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "fork_join.cpp", tmp_path / "fork_join"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"),
                           "-I", os.path.join(ROOT, "mpm_b200", "csrc"), str(src), "-o", str(exe)])
    rows = [tuple(map(int, r.split())) for r in subprocess.check_output([str(exe)], text=True).splitlines()]
    handle, isolation = 400, 905  # cudaErrorInvalidResourceHandle, cudaErrorStreamCaptureIsolation
    assert rows == [(0, 0, 0, 2, 1), (0, 1, 0, 2, 1), (1, 0, handle, 1, 1), (1, 1, handle, 1, 1),
                    (2, 0, isolation, 2, 1), (2, 1, isolation, 2, 1)]
