"""The wide node test (bvh.cuh cw_node), its source compiled for the host: a child that the slab
test with unfolded offsets accepts (each plane one FMA of the quantized byte and the rounded
(p - o) / d) is accepted, from inside the node to 10^7 cells away, where the folded offset's own
rounding exceeds a fixed share of a cell.  Rays aim at the edges and corners of the children,
most of them one cell thin, where a rounding decides."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

BVH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pathtracerglsl_b200", "csrc", "device", "bvh.cuh")

HARNESS = r"""
#include <cmath>
#include <cstring>
#include <cstdint>
#define __device__
#define __forceinline__ inline
struct uint4 { unsigned x, y, z, w; };
struct f3 {
    float x, y, z;
    f3() : x(0), y(0), z(0) {}
    f3(float a, float b, float c) : x(a), y(b), z(c) {}
};
static f3 operator+(f3 a, f3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
static f3 operator-(f3 a, f3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
static f3 operator*(f3 a, f3 b) { return f3(a.x * b.x, a.y * b.y, a.z * b.z); }
static f3 operator*(f3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
static uint4 __ldg(const uint4* p) { return *p; }
static float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static int __ffs(int v) { return __builtin_ffs(v); }
static unsigned __byte_perm(unsigned x, unsigned y, unsigned s) {
    const uint64_t both = ((uint64_t)y << 32) | x;
    unsigned r = 0;
    for (int k = 0; k < 4; ++k) r |= (unsigned)((both >> (8 * ((s >> (4 * k)) & 7u))) & 0xFFu) << (8 * k);
    return r;
}
@SOURCE@
// The test without the fold: planes in the order of the box's faces, each one FMA.
static float gmin(float a, float b) { return b < a ? b : a; }
static float gmax(float a, float b) { return a < b ? b : a; }
// widen: the planes moved apart by 0.05 cells and 2^-20 of the offset, more than twice what the
// node test's pad (2^-7 of a cell and 5 * 2^-24 of the folded offset) can come to.
static bool slab(const uint32_t* w, int s, f3 ro, const CwRay& cr, float tmax, bool widen) {
    const unsigned char* q = (const unsigned char*)(w + 8);
    const float o[3] = {ro.x, ro.y, ro.z}, inv[3] = {cr.inv.x, cr.inv.y, cr.inv.z};
    float tn = 0.0f, tf = tmax;
    for (int a = 0; a < 3; ++a) {
        const float dq = __uint_as_float(((w[3] >> (8 * a)) & 0xFFu) << 23) * inv[a];
        const float oq = (__uint_as_float(w[a]) - o[a]) * inv[a];
        const float lo = std::fma((float)q[8 * a + s], dq, oq), hi = std::fma((float)q[24 + 8 * a + s], dq, oq);
        const float by = widen ? 0.05f * std::fabs(dq) + 9.5367432e-7f * std::fabs(oq) : 0.0f;
        tn = gmax(gmin(lo, hi) - by, tn);
        tf = gmin(gmax(lo, hi) + by, tf);
    }
    return !(tf * kBvhTfarPad < tn);
}
// The children a ray meets, bit s for slot s: the node test's, the unfolded test's and those of
// the unfolded test with wider boxes.
extern "C" void verdicts(const uint32_t* nodes, const float* rays, int n, float tmax, unsigned char* folded, unsigned char* unfolded, unsigned char* wide) {
    for (int i = 0; i < n; ++i) {
        uint32_t w[20];
        std::memcpy(w, nodes + 20 * (size_t)i, sizeof(w));
        const float* r = rays + 6 * (size_t)i;
        const f3 ro(r[0], r[1], r[2]);
        const CwRay cr = cw_ray(f3(r[3], r[4], r[5]));
        const CwNodeHits h = cw_node((const uint4*)w, ro, cr, tmax);
        unsigned a = 0, b = 0, c = 0;
        for (int s = 0; s < 8; ++s) {
            if ((h.hits >> (((unsigned)s ^ cr.octinv) & 7u)) & 1u) a |= 1u << s;
            if (slab(w, s, ro, cr, tmax, false)) b |= 1u << s;
            if (slab(w, s, ro, cr, tmax, true)) c |= 1u << s;
        }
        folded[i] = (unsigned char)a;
        unfolded[i] = (unsigned char)b;
        wide[i] = (unsigned char)c;
    }
}
"""


@pytest.fixture(scope="module")
def node_test(tmp_path_factory):
    src = open(BVH).read()
    pad = re.search(r"constexpr float kBvhTfarPad = [^;]+;", src).group(0)
    clamp = re.search(r"__device__ __forceinline__ float clamp_dir[^\n]+\n", src).group(0)
    body = src[src.index("struct CwRay"):src.index("// The next child of a node group")]
    d = tmp_path_factory.mktemp("cw_node")
    (d / "cw_node.cpp").write_text(HARNESS.replace("@SOURCE@", "\n".join((pad, clamp, body))))
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC",
                    str(d / "cw_node.cpp"), "-o", str(d / "cw_node.so")], check=True)
    return C.CDLL(str(d / "cw_node.so")).verdicts


def _cases(rng, n, reach):
    """n nodes of eight inner children and one ray each, `reach` cells from the node, aimed at an edge
    or a corner of a child of it."""
    e = rng.randint(-12, 4, (n, 3))
    cell = 2.0 ** e
    p = (rng.uniform(-4, 4, (n, 3)) * 255 * cell).astype(np.float32)
    lo = rng.randint(0, 256, (n, 3, 8))
    hi = np.minimum(255, lo + np.where(rng.uniform(size=(n, 3, 8)) < 0.7, rng.randint(0, 2, (n, 3, 8)), rng.randint(0, 256, (n, 3, 8))))
    nodes = np.zeros((n, 20), np.uint32)
    nodes[:, :3] = p.view(np.uint32)
    exps = (e + 127).astype(np.uint32)
    nodes[:, 3] = exps[:, 0] | (exps[:, 1] << 8) | (exps[:, 2] << 16) | np.uint32(0xFF000000)
    nodes[:, 6:8] = np.frombuffer(bytes(32 + 24 + s for s in range(8)), np.uint32)
    nodes[:, 8:14] = lo.astype(np.uint8).reshape(n, 24).view(np.uint32)
    nodes[:, 14:20] = hi.astype(np.uint8).reshape(n, 24).view(np.uint32)
    child, k = rng.randint(8, size=n), np.arange(n)
    face = rng.randint(3, size=(n, 3))          # per axis the low face, the high face or a point between
    face[k, rng.randint(3, size=n)] = 0
    l, h = lo[k, :, child], hi[k, :, child]
    at = p + cell * np.where(face == 0, l, np.where(face == 1, h, l + (h - l) * rng.uniform(size=(n, 3))))
    u = rng.normal(size=(n, 3)) * np.where(rng.uniform(size=(n, 3)) < 0.15, 1e-9, 1.0)
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    o = (at + u * (reach * cell.max(axis=1))[:, None]).astype(np.float32)
    d = at - o
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)
    return nodes, np.ascontiguousarray(np.concatenate([o, d.astype(np.float32)], axis=1), np.float32)


@pytest.mark.parametrize("reach", [0.3, 30.0, 1e3, 1e4, 1e5, 1e6, 1e7])
def test_no_child_of_the_unfolded_test_is_lost(node_test, reach):
    n = 1_000_000
    nodes, rays = _cases(np.random.RandomState(int(reach) % 99991), n, reach)
    folded, unfolded, wide = (np.zeros(n, np.uint8) for _ in range(3))
    node_test(*(v.ctypes.data_as(C.c_void_p) for v in (nodes, rays)), n, C.c_float(1e20),
              *(v.ctypes.data_as(C.c_void_p) for v in (folded, unfolded, wide)))
    assert (unfolded != 0).mean() > 0.2
    lost = unfolded & ~folded
    assert not lost.any(), f"{(lost != 0).sum()} rays lose a child"
    assert not (folded & ~wide).any()   # nor is a box widened beyond its pad
