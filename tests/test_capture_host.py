"""capture_graph (csrc/cuda/capture.hpp) against a runtime whose calls can be made to fail: whichever step
fails, the caller gets no graph and no pending error (it then launches one by one and asks for the last
error after that)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "capture.hpp"
static int failing, destroyed;
static cudaError_t last;
static cudaError_t ret(int call) { return call == failing ? last = cudaErrorStreamCaptureUnsupported : cudaSuccess; }
extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return ret(1); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = failing == 2 ? nullptr : (cudaGraph_t)0x10;
  return ret(2);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  if (failing != 3) *e = (cudaGraphExec_t)0x20;
  return ret(3);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { ++destroyed; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
}
int main(int, char** v) {
  failing = std::atoi(v[1]);
  int enqueued = 0;
  cudaGraphExec_t e = dpm::gpu::capture_graph(nullptr, [&] { ++enqueued; });
  std::printf("%d %d %d %d\n", e != nullptr, enqueued, destroyed, (int)last);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("capture")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INC, "-I", os.path.join(ROOT, "dopamine_b200", "csrc", "cuda"),
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("failing,expect", [(0, "1 1 1 0"), (1, "0 0 0 0"), (2, "0 1 0 0"), (3, "0 1 1 0")])
def test_failing_step_leaves_no_graph_and_no_error(program, failing, expect):
    out = subprocess.run([program, str(failing)], capture_output=True, text=True, check=True).stdout.strip()
    assert out == expect
