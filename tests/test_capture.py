"""The host helper that builds CUDA graphs (euler3d_b200/csrc/common.hpp), compiled for the CPU against a
recording stand-in for the runtime: a capture is ended and its graph destroyed however the queued work
ends, so an error leaves the stream usable."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = r"""
#include "common.hpp"
static int capturing, graphs, fail;
extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing++; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    capturing--;
    if (fail == 2) { *g = nullptr; return cudaErrorStreamCaptureInvalidated; }
    graphs++;
    *g = (cudaGraph_t)&graphs;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { graphs--; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    if (fail == 3) return cudaErrorMemoryAllocation;
    *e = (cudaGraphExec_t)&fail;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
// 0: a graph, 1: an error that left nothing behind, 2: anything else
int build(int how) {
    fail = how;
    int result = 0;
    try {
        if (!e3d::capture_graph(nullptr, [] { if (fail == 1) throw e3d::Error(E3D_ERR_CUDA, "launch"); })) result = 2;
    } catch (const e3d::Error &) {
        result = 1;
    }
    return capturing || graphs ? 2 : result;
}
}
"""


@pytest.fixture(scope="module")
def build_graph(tmp_path_factory):
    from euler3d_b200 import build

    d = tmp_path_factory.mktemp("capture")
    (d / "capture.cpp").write_text(SOURCE)
    root = os.path.dirname(HERE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{root}/euler3d_b200/csrc",
                    f"-I{root}/include", f"-I{cuda}", "-o", str(d / "capture.so"), str(d / "capture.cpp")], check=True)
    return C.CDLL(str(d / "capture.so")).build


@pytest.mark.parametrize("fail", [0, 1, 2, 3], ids=["none", "launch", "end of capture", "instantiation"])
def test_capture_ends(build_graph, fail):
    assert build_graph(fail) == (1 if fail else 0)
