"""CPU test of csrc/stream_fork.h against a fake of the CUDA runtime's event and stream calls: a scope
that is left by an exception between fork and join still makes the main stream (in whose order the
buffers are freed) wait for every auxiliary stream, and a failing call of the join leaves no stream out.
"""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "gammcor-integrals_b200" / "csrc"
CUDA_INCLUDE = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

HARNESS = r"""
#include "stream_fork.h"
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <stdexcept>

// streams and events are small numbers; each call prints one line
static int id(const void* p) { return (int)(intptr_t)p; }
static int fail_record_of = -1, fail_wait_of = -1;   // a stream's id
extern "C" cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    if (id(s) == fail_record_of) return cudaErrorUnknown;
    std::printf("record %d %d\n", id(e), id(s));
    return cudaSuccess;
}
extern "C" cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    if (id(s) == fail_wait_of) return cudaErrorUnknown;
    std::printf("wait %d %d\n", id(s), id(e));
    return cudaSuccess;
}
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    std::printf("sync %d\n", id(s));
    return cudaSuccess;
}
struct Buffer { ~Buffer() { std::printf("free\n"); } };

int main(int argc, char** argv)
{
    const char* what = argc > 1 ? argv[1] : "";
    const cudaStream_t main_s = (cudaStream_t)1, aux[2] = {(cudaStream_t)2, (cudaStream_t)3};
    const cudaEvent_t ev = (cudaEvent_t)10, join[2] = {(cudaEvent_t)12, (cudaEvent_t)13};
    if (!std::strcmp(what, "begin")) fail_wait_of = 3;
    try {
        Buffer b;
        gci::StreamFork f(main_s, aux, 2, ev, join);
        if (f.begin() != cudaSuccess) throw std::runtime_error("begin");
        std::printf("launch\n");
        if (!std::strcmp(what, "record")) fail_record_of = 2;
        if (!std::strcmp(what, "throw")) throw std::runtime_error("launch failed");
        std::printf("join %d\n", (int)f.join());
    } catch (const std::exception& e) {
        std::printf("caught\n");
    }
    return 0;
}
"""

FORK = ["record 10 1", "wait 2 10", "wait 3 10"]
JOIN = ["record 12 2", "wait 1 12", "record 13 3", "wait 1 13"]


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime_api.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("fork")
    (d / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(CUDA_INCLUDE), str(d / "harness.cpp"), "-o",
                    str(d / "harness")], check=True)
    return lambda what: subprocess.run([str(d / "harness"), what], check=True, capture_output=True,
                                       text=True).stdout.split("\n")[:-1]


@pytest.mark.parametrize("what,calls", [
    ("", FORK + ["launch"] + JOIN + ["join 0", "free"]),
    ("throw", FORK + ["launch"] + JOIN + ["free", "caught"]),
    ("record", FORK + ["launch", "sync 2"] + JOIN[2:] + ["join 999", "free"]),
    ("begin", FORK[:2] + ["free", "caught"]),
])
def test_every_auxiliary_stream_is_joined(harness, what, calls):
    assert harness(what) == calls
