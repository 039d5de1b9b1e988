"""Device memory of the contexts (host/device_memory.h, compiled against a stub runtime): devices
of any ordinal, and devices that make no memory pool, allocate; contexts on one device share
a pool that goes with the last of them; every block is given back the way it was taken."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pathtracerglsl_b200", "csrc")

STUB = """
#pragma once
#include <cstddef>
typedef int* cudaStream_t;
typedef int* cudaMemPool_t;
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorNotSupported = 801 };
enum { cudaDevAttrMemoryPoolsSupported, cudaMemAllocationTypePinned, cudaMemLocationTypeDevice, cudaMemPoolAttrReleaseThreshold,
       cudaMemPoolReuseAllowInternalDependencies };
struct cudaMemPoolProps { int allocType; struct { int type, id; } location; };
cudaError_t cudaDeviceGetAttribute(int*, int, int);
cudaError_t cudaMemPoolCreate(cudaMemPool_t*, const cudaMemPoolProps*);
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, int, void*);
cudaError_t cudaMemPoolDestroy(cudaMemPool_t);
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t);
cudaError_t cudaMalloc(void**, size_t);
cudaError_t cudaFree(void*);
cudaError_t cudaMallocFromPoolAsync(void**, size_t, cudaMemPool_t, cudaStream_t);
cudaError_t cudaFreeAsync(void*, cudaStream_t);
cudaError_t cudaDeviceSynchronize();
enum { cudaStreamNonBlocking = 1 };
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned);
cudaError_t cudaStreamDestroy(cudaStream_t);
cudaError_t cudaGetLastError();
"""
RUNTIME = """
#include "host/device_memory.h"
#include <cstdio>
static bool supported = true, creates = true;
static size_t left = ~(size_t)0, idle = 0;   // bytes the device has free; bytes its pool holds unused
static int next = 0;
cudaError_t cudaDeviceGetAttribute(int* v, int, int) { *v = supported; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* q) {
    std::printf("pool%d ", q->location.id);
    *p = creates ? new int(q->location.id) : nullptr;
    return creates ? cudaSuccess : cudaErrorNotSupported;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, int a, void* v) {
    if (a == cudaMemPoolAttrReleaseThreshold) std::printf("keep%llu ", *(unsigned long long*)v >> 20);
    else std::printf(*(int*)v ? "tied " : "apart ");
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { std::printf("~pool%d ", *p); return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t n) { std::printf("trim%zu ", n); left += idle; idle = 0; return cudaSuccess; }
static cudaError_t take(void** out, size_t n, const char* how) {
    std::printf("%s%s ", how, n <= left ? "" : "!");
    if (n > left) return cudaErrorMemoryAllocation;
    left -= n;
    *out = (void*)(size_t)++next;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, "malloc"); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return take(p, n, "pooled"); }
cudaError_t cudaFree(void* p) { std::printf("free%zu ", (size_t)p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::printf("async%zu ", (size_t)p); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { std::printf("wait "); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { std::printf("stream "); *s = new int(0); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { std::printf("~stream "); return cudaSuccess; }
using ptx_host::DeviceMemory;
using ptx_host::DevicePools;
int main() {
    void *a, *b;
    %s
}
"""


def _run(tmp_path, body):
    (tmp_path / "cuda_runtime.h").write_text(STUB)
    (tmp_path / "t.cpp").write_text(RUNTIME.replace("%s\n}", body + "\n}"))
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t"), "-pthread"], check=True)
    return subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout.split()


def test_contexts_share_a_devices_pool(tmp_path):
    out = _run(tmp_path, """
    DeviceMemory m, n, o;
    m.open(0, nullptr); n.open(0, nullptr); o.open(1, nullptr);
    m.alloc(&a, 100); n.alloc(&b, 257u << 20);
    m.free(a); n.free(b); n.free(nullptr);
    m.close(); n.close(); o.close();
    m.open(0, nullptr); m.close();
    """)
    assert out == "pool0 keep512 apart pool1 keep512 apart pooled malloc async1 free2 ~pool0 ~pool1 pool0 keep512 apart ~pool0".split()


def test_any_ordinal_and_no_pools(tmp_path):
    use = "m.alloc(&a, 100); m.alloc(&b, 1u << 30); m.free(a); m.free(b); m.close();"
    assert _run(tmp_path, "DeviceMemory m; m.open(71, nullptr); " + use) == \
        "pool71 keep512 apart pooled malloc async1 free2 ~pool71".split()
    assert _run(tmp_path, "supported = false; DeviceMemory m; m.open(0, nullptr); " + use) == "malloc malloc free1 free2".split()
    assert _run(tmp_path, "creates = false; DeviceMemory m; m.open(0, nullptr); " + use) == "pool0 malloc malloc free1 free2".split()


def test_a_block_that_does_not_fit_is_null(tmp_path):
    out = _run(tmp_path, """
    DeviceMemory m; m.open(0, nullptr);
    left = 1000;
    a = &a;
    std::printf("%d ", (int)m.alloc(&a, 2000));
    std::printf("%s ", a ? "set" : "null");
    m.free(a);
    std::printf("%d ", (int)m.alloc(&a, 500));
    m.free(a);
    m.close();
    """)
    assert "2 null" in " ".join(out) and out[-4:] == ["pooled", "0", "async1", "~pool0"]


def test_idle_pool_memory_does_not_refuse_a_block(tmp_path):
    """A block fits as long as it fits beside the blocks in use: what the pool keeps idle is given
    back first, and a block that does not fit then is refused."""
    out = _run(tmp_path, """
    DeviceMemory m; m.open(0, nullptr);
    left = 300u << 20; idle = 400u << 20;
    std::printf("%d ", (int)m.alloc(&a, 600u << 20));
    std::printf("%d ", (int)m.alloc(&b, 200u << 20));
    idle = 150u << 20;
    std::printf("%d ", (int)m.alloc(&b, 200u << 20));
    m.free(a); m.free(b); m.close();
    """)
    assert out == ("pool0 keep512 apart malloc! wait trim0 malloc 0 pooled! wait trim0 pooled! 2 "
                   "pooled! wait trim0 pooled 0 free1 async2 ~pool0").split()


def test_contexts_share_a_devices_upload_stream(tmp_path):
    out = _run(tmp_path, """
    DeviceMemory m, n;
    m.open(2, nullptr); n.open(2, nullptr);
    std::printf("%s ", DevicePools::all().upload_stream(2) == DevicePools::all().upload_stream(2) ? "same" : "other");
    m.close();
    std::printf("| ");
    n.close();
    m.open(2, nullptr); m.close();
    """)
    assert out == "pool2 keep512 apart stream same | ~stream ~pool2 pool2 keep512 apart ~pool2".split()
