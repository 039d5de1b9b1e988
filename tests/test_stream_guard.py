"""Host memory behind asynchronous copies (host/stream_guard.h, compiled against a stub runtime
that logs its calls): every way out of a scope that holds such memory waits for the stream
before the memory goes, an error's included; and the calls that copy from memory of their own
take the guard."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pathtracerglsl_b200", "csrc")

STUB = """
#pragma once
typedef int cudaStream_t;
enum cudaError_t { cudaSuccess, cudaErrorUnknown };
cudaError_t cudaStreamSynchronize(cudaStream_t);
"""
PROGRAM = """
#include "host/stream_guard.h"
#include <cstdio>
cudaError_t cudaStreamSynchronize(cudaStream_t s) { std::printf("wait%d ", s); return cudaSuccess; }
struct Image { ~Image() { std::printf("free "); } };
int call(bool fails) {
    Image image;
    ptx_host::StreamGuard guard(7);
    std::printf("copy ");
    if (fails) return 1;
    cudaStreamSynchronize(7);
    guard.waited();
    return 0;
}
int main() {
    call(true);
    std::printf("| ");
    call(false);
}
"""


def test_memory_outlives_its_copies(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(STUB)
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout
    assert out == "copy wait7 free | copy wait7 free "


def test_calls_with_host_images_take_the_guard():
    src = open(os.path.join(CSRC, "ptx_rt.cu")).read()
    for function, memory in (("int ptr_render_batch(", "image(n_tables);"), ("int build_mesh_device_core(", "root_task ="),
                             ("int ptr_trace_closest(", "const float* rays")):
        body = src[src.index(function):]
        body = body[:re.search(r"\n\}\n", body).end()]
        at, guard, copy = body.index(memory), body.index("StreamGuard guard("), body.index("cudaMemcpyAsync(")
        assert at < guard < copy, function
