"""The side stream of a factorisation (SideScope) against a runtime that records its calls and fails on demand:
the work beside a handle's stream is joined to it, and a join that fails is an error, not an unordered call."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "internal.cuh"
#include <cstdio>
#include <cstring>
#include <string>

static const char* g_fail = "";  // the call that fails
static int g_made = 0;
static const char* name(const void* p) {  // handles in the order of their creation; the handle's own stream
    static char b[4][16];
    static int k = 0;
    char* o = b[++k % 4];
    if ((size_t)p == 0x1000) return "own";
    std::snprintf(o, 16, "%zu", (size_t)p);
    return o;
}
static cudaError_t call(const std::string& what) {
    std::puts(what.c_str());
    return what == g_fail ? cudaErrorUnknown : cudaSuccess;
}
extern "C" {
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)(size_t)++g_made;
    return call("stream");
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t)(size_t)++g_made;
    return call("event");
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return call(std::string("record ") + name(e) + " on " + name(s)); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    return call(std::string(name(s)) + " waits for " + name(e));
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return call(std::string("synchronise ") + name(s)); }
}

int main(int, char** argv) {
    using namespace gwb200;
    const std::string mode = argv[1];
    g_fail = argv[2];
    SideStream side;
    cudaStream_t own = (cudaStream_t)(size_t)0x1000;
    try {
        if (mode == "unused") return 0;
        if (mode == "none") {
            SideScope beside(nullptr, own);
            std::printf("on %s\n", name(beside.stream()));
            beside.join();
            return 0;
        }
        if (mode == "twice") {
            SideScope first(&side, own);
            first.stream();
            first.join();
        }
        SideScope beside(&side, own);
        beside.stream();
        std::puts("work");
        if (mode == "throws") fail(GWB200_CUDA_ERROR, "launch");
        beside.join();
        std::puts("joined");
    } catch (const Failure& f) {
        std::printf("error %d\n", f.code);
    }
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("side")
    (d / "side.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-w", "-x", "c++", f"-I{ROOT / 'minigw_b200' / 'csrc'}", "-I/usr/local/cuda/include",
                    str(d / "side.cpp"), "-o", str(d / "side")], check=True)

    def go(mode, fails=""):
        out = subprocess.run([str(d / "side"), mode, fails], check=True, capture_output=True, text=True).stdout
        return out.splitlines()

    return go


MADE = ["stream", "event", "event"]  # stream 1, events 2 (fork) and 3 (join)
BEGIN = MADE + ["record 2 on own", "1 waits for 2", "work"]


def test_joined_once(run):
    assert run("normal") == BEGIN + ["record 3 on 1", "own waits for 3", "joined"]


@pytest.mark.parametrize("fails", ["record 3 on 1", "own waits for 3"])
def test_a_join_that_fails_is_reported(run, fails):
    out = run("normal", fails)
    assert "joined" not in out
    assert out[-2:] == ["synchronise 1", "error 6"]


def test_left_by_an_exception(run):
    assert run("throws") == BEGIN + ["record 3 on 1", "own waits for 3", "error 6"]
    assert run("throws", "own waits for 3")[-2:] == ["synchronise 1", "error 6"]


def test_made_by_the_first_scope_alone(run):
    assert run("unused") == []
    assert run("none") == ["on own"]
    twice = run("twice")
    assert twice[:3] == MADE and not {"stream", "event"} & set(twice[3:])
