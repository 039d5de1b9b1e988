"""The events of an instrumented render (host/profile_events.h, compiled against a stub runtime):
a render that fails between its launches gives back every event it made, and the times and
launch counts of one that finishes add up per kernel class."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pathtracerglsl_b200", "csrc")

STUB = """
#pragma once
typedef int cudaStream_t;
typedef int* cudaEvent_t;
enum cudaError_t { cudaSuccess, cudaErrorUnknown };
cudaError_t cudaEventCreate(cudaEvent_t*);
cudaError_t cudaEventDestroy(cudaEvent_t);
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t);
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t);
"""
PROGRAM = """
#include "host/profile_events.h"
#include <cstdio>
static int live = 0, tick = 0;
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = new int(0); ++live; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --live; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { *e = ++tick * tick; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t a, cudaEvent_t b) { *t = (float)(*b - *a); return cudaSuccess; }
int render(bool fails, float* ms, int* n) {
    ptx_host::ProfList prof;
    for (int w = 0; w < 3; ++w) {
        prof.begin(2, 10 * w, 0);
        prof.end(10 * w + 4, 0);
        prof.begin(4, 10 * w + 4, 0);
        if (fails && w == 1) return 1;
        prof.end(10 * w + 5, 0);
    }
    prof.fold(ms, n);
    return 0;
}
int main() {
    float ms[6] = {};
    int n[6] = {};
    std::printf("%d ", render(true, ms, n));
    std::printf("%d ", live);
    tick = 0;
    std::printf("%d ", render(false, ms, n));
    std::printf("%d %.0f %.0f %d %d %d", live, ms[2], ms[4], n[2], n[4], n[0]);
}
"""


def test_events_are_given_back(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(STUB)
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout
    # the event of tick k reads k^2: class 2 gets (4 - 1) + (36 - 25) + (100 - 81), class 4 (16 - 9) + (64 - 49) + (144 - 121)
    assert out == "1 0 0 0 33 45 12 3 0"


def test_the_library_makes_its_profile_events_there():
    src = open(os.path.join(CSRC, "ptx_rt.cu")).read()
    assert not re.search(r"cudaEventCreate|cudaEventDestroy", src)
