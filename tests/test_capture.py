"""The capture of a restart chunk as a graph, on the CPU against a fake of the CUDA runtime's calls: whichever of them
fails, and where a launch inside throws, the capture has ended, nothing leaks and no error is left."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "capture.cuh"
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <string>

static std::string fail;
static int capturing = 0, graphs = 0, execs = 0, launched = 0;
static cudaError_t last = cudaSuccess;
static cudaError_t result(const char *call) { return last = fail == call ? cudaErrorStreamCaptureInvalidated : cudaSuccess; }
extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    if (result("begin") == cudaSuccess) ++capturing;
    return last;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    --capturing;
    *g = nullptr;
    if (fail == "launch") return last = cudaErrorStreamCaptureInvalidated; // as a failed launch leaves the capture
    if (result("end") != cudaSuccess) return last;
    ++graphs;
    *g = reinterpret_cast<cudaGraph_t>(&graphs);
    return last;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
    if (result("instantiate") != cudaSuccess) return last;
    ++execs;
    *e = reinterpret_cast<cudaGraphExec_t>(&execs);
    return last;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { --graphs; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
}

int main(int, char **argv)
{
    fail = argv[1];
    const auto exec = mhd::capture_graph(nullptr, [] {
        ++launched;
        if (fail == "launch" || fail == "throw") throw std::runtime_error("launch failed");
    });
    std::printf("exec %d capturing %d graphs %d execs %d launched %d error %d\n", exec != nullptr, capturing, graphs, execs, launched, (int)last);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("capture")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-I" + os.path.join(ROOT, "mpcns_uns_b200", "csrc", "gpu"),
                    "-I/usr/local/cuda/include", "-o", str(d / "t"), str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("fail", ["none", "begin", "launch", "throw", "end", "instantiate"])
def test_capture_always_ends(program, fail):
    out = subprocess.run([program, fail], check=True, capture_output=True, text=True).stdout.split()
    got = dict(zip(out[::2], map(int, out[1::2])))
    ok = fail == "none"
    assert got == dict(exec=ok, capturing=0, graphs=0, execs=ok, launched=fail != "begin", error=0)
