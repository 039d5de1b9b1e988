// bvh.cuh — acceleration-structure arms of the scene queries: triangle meshes (binary BVH
// or compressed wide BVH BLAS) and instanced batches (binary TLAS over placements).
//
// Triangle leaf: Moller-Trumbore as the reference's mesh_tri_test
//   (src/components/intersection/mesh/mesh.glsl:41-59), flat geometric normal.
// Binary walk: the stack-DFS of mesh_nearest_bvh (mesh.glsl:162-191) with the padded slab
//   test bvh_aabb_hit (accel/bvh/bvh.glsl:28-36), near child first by the split axis.
// Wide walk: the octant-ordered CWBVH walk (intersection/index.ts:99-158): per-node ray
//   transform, one-FMA quantized slabs, find-MSB child order, node groups on a small stack.
//   Nodes are fetched as five 128-bit loads.
// Placements (intersection/instancing/placement.glsl:19-41): world -> rigid frame by the
//   stored quaternion q and ts = (t_rigid, s); mesh prototypes are intersected in their
//   local frame with the t-preserving (un-normalised) direction.
#pragma once
#include "scene.cuh"

namespace ptx {

constexpr float kBvhTfarPad = 1.00000024f;   // BVH_TFAR_PAD (Ize 2013 far-plane pad)
constexpr int kBvhStack = 64;                // BVH_STACK_DEPTH
constexpr int kCwStack = 24;                 // CWBVH_STACK_DEPTH
constexpr unsigned kErrBvhStack = 1u;        // a binary walk dropped a subtree (stack full)
constexpr unsigned kErrCwStack = 2u;         // a wide walk dropped a node group
constexpr unsigned kErrCwGuard = 4u;         // a wide walk hit its iteration guard

struct HitRec { float t, u, v; int region, element, prim; };

// Per-thread work tally (instrumented pass only): the timed kernels pass a null tally,
// which the inlined walks fold away.
struct Work { unsigned nodes, tris, tlas, inst; };

__device__ __forceinline__ void flag_error(const DevScene& S, unsigned bit) {
    if (S.err_flags) atomicOr(S.err_flags, bit);
}

// ---- placement algebra ------------------------------------------------------------------
__device__ __forceinline__ f3 qrot(float4 q, f3 v) {
    f3 qv(q.x, q.y, q.z);
    return v + 2.0f * cross(qv, cross(qv, v) + q.w * v);
}
__device__ __forceinline__ f3 placement_rigid(float4 q, float4 ts, f3 p) { return qrot(q, p) + f3(ts.x, ts.y, ts.z); }
__device__ __forceinline__ f3 placement_normal(float4 q, f3 n) { return qrot(make_float4(-q.x, -q.y, -q.z, q.w), n); }

// ---- triangle leaf --------------------------------------------------------------------
__device__ __forceinline__ bool tri_test(f3 ro, f3 rd, f3 a, f3 e1, f3 e2, float& t) {
    f3 gnorm = cross(e1, e2);
    float det = -dot(rd, gnorm);
    if (fabsf(det) < 1e-12f) return false;
    float invdet = 1.0f / det;
    f3 ao = ro - a;
    f3 dao = cross(ao, rd);
    float u = dot(e2, dao) * invdet;
    float v = -dot(e1, dao) * invdet;
    t = dot(ao, gnorm) * invdet;
    float w = 1.0f - u - v;
    const float E = 1e-6f;
    return u >= -E && v >= -E && w >= -E;
}
__device__ __forceinline__ void load_tri(const float4* tri, int i, f3& a, f3& e1, f3& e2) {
    float4 t0 = __ldg(tri + 3 * i), t1 = __ldg(tri + 3 * i + 1), t2 = __ldg(tri + 3 * i + 2);
    a = xyz(t0); e1 = xyz(t1); e2 = xyz(t2);
}
// The caller's index of the triangle in leaf slot i (stored in the record's first w).
__device__ __forceinline__ int tri_orig(const float4* tri, int i) { return __float_as_int(__ldg(&tri[3 * (size_t)i].w)); }

// Hits at equal t resolve in one order whatever the traversal visits first: the lower
// region index, then the lower instance index (the caller's placement order), then the
// lower triangle index of the caller's mesh.  The oracle's ordered scans give that order,
// so hit IDs agree at ties too.  Node tests keep boxes entered exactly at the current t
// (a tied triangle may sit on the box's near face); leaf tests take t == tmax only when
// it wins the tie.  NoTie: no tie with the incoming tmax is won (a plain mesh region;
// its incoming tmax belongs to an earlier region).
struct NoTie { __device__ __forceinline__ bool operator()() const { return false; } };

// ---- binary BVH walk --------------------------------------------------------------------
__device__ __forceinline__ bool aabb_hit(float4 n0, float4 n1, f3 ro, f3 inv, float tmax) {
    float tx0 = (n0.x - ro.x) * inv.x, tx1 = (n1.x - ro.x) * inv.x;
    float ty0 = (n0.y - ro.y) * inv.y, ty1 = (n1.y - ro.y) * inv.y;
    float tz0 = (n0.z - ro.z) * inv.z, tz1 = (n1.z - ro.z) * inv.z;
    float tn = gmax(gmax(gmin(tx0, tx1), gmin(ty0, ty1)), gmin(tz0, tz1));
    float tf = gmin(gmin(gmax(tx0, tx1), gmax(ty0, ty1)), gmax(tz0, tz1)) * kBvhTfarPad;
    float tenter = gmax(tn, 0.0f);
    return tf >= tenter && tenter <= tmax;
}

// Leaf(off, cnt) -> for nearest walks updates the caller's tmax itself; returns true to
// stop the walk (any-hit found).
template <class Leaf>
__device__ __forceinline__ bool walk_binary(const DevScene& S, const float4* nodes, f3 ro, f3 rd, const float& tmax, Leaf leaf,
                                            unsigned* visits = nullptr) {
    f3 inv(1.0f / rd.x, 1.0f / rd.y, 1.0f / rd.z);
    int stack[kBvhStack];
    int ptr = 0;
    stack[0] = 0;
    while (ptr >= 0) {
        int ni = stack[ptr];
        ptr--;
        if (visits) (*visits)++;
        float4 n0 = __ldg(nodes + 2 * ni), n1 = __ldg(nodes + 2 * ni + 1);
        if (!aabb_hit(n0, n1, ro, inv, tmax)) continue;
        if (n0.w >= 0.0f) {
            if (leaf((int)n1.w, (int)n0.w)) return true;
        } else {
            int axis = (int)(-n0.w - 1.0f);
            int L = ni + 1, R = (int)n1.w;
            bool nf = (axis == 0 ? rd.x : (axis == 1 ? rd.y : rd.z)) >= 0.0f;
            if (ptr + 2 < kBvhStack) {
                stack[++ptr] = nf ? R : L;
                stack[++ptr] = nf ? L : R;
            } else {
                flag_error(S, kErrBvhStack);
            }
        }
    }
    return false;
}

// ---- compressed wide BVH walk ---------------------------------------------------------------
__device__ __forceinline__ int find_msb24(unsigned v) { return 31 - __clz(v); }
__device__ __forceinline__ float clamp_dir(float d) { return fabsf(d) < 1e-20f ? (d < 0.0f ? -1e-20f : 1e-20f) : d; }

// Per-ray set-up of a wide walk: the direction with zero components clamped (slab
// reciprocals stay finite), its reciprocal and the inverted octant that orders children.
struct CwRay { f3 inv; unsigned octinv; };
__device__ __forceinline__ CwRay cw_ray(f3 rd) {
    f3 rdc(clamp_dir(rd.x), clamp_dir(rd.y), clamp_dir(rd.z));
    CwRay c;
    c.octinv = 7u - ((rdc.x < 0.0f ? 1u : 0u) | (rdc.y < 0.0f ? 2u : 0u) | (rdc.z < 0.0f ? 4u : 0u));
    c.inv = f3(1.0f / rdc.x, 1.0f / rdc.y, 1.0f / rdc.z);
    return c;
}
// One CWBVH node against the ray: the hit internal children as an octant-ordered bit mask
// (hits, with the node's child base and internal-child mask for the group) and the hit
// leaf triangles as bits above the node's triangle base (leaf_bits, leaf_base).
//
// The walk is bound by instruction issue, so a child costs as few instructions as the test
// allows, and no branch: the ray's octant picks the near and the far plane of each axis once
// per node; a quantized byte b becomes the float 1 + b 2^-15 by one byte permute and its
// plane's distance by one FMA with the offset c = (p - o) / d - 2^15 dq folded in (dq: a cell's
// distance); internal and leaf children are told apart on the 8-bit hit mask.
//
// No child is lost to the fold.  The slab test without it takes a plane at fma(b, dq, (p - o) / d);
// folded, c, c -+ pad and the plane round once more each, and |plane| <= |c| + 33023 |dq|, so
// with u = 2^-24 the two differ by less than pad if that is 4 u |c| + 66046 u |dq| and a little for
// the roundings' own products.  kCwPad (2^-7 > 66046 u) of a cell and kCwPadOffset (5 u) of |c|
// are: near planes lie before the unfolded ones, far planes behind, from any distance.  (The
// share of |c| costs three FMAs a node; 1920 x 1080 x 16 spp of 16 instanced meshes took 65.9 ms
// with it and without.)
struct CwNodeHits { unsigned hits, leaf_bits, child_base, imask, leaf_base; };
constexpr float kCwPad = 0.0078125f, kCwPadOffset = 2.9802322e-7f;
__device__ __forceinline__ float cw_plane(unsigned word, unsigned k, float scale, float offset) {
    return __fmaf_rn(__uint_as_float(__byte_perm(word, 0x3F800000u, 0x7604u | (k << 4))), scale, offset);
}
__device__ __forceinline__ CwNodeHits cw_node(const uint4* nd, f3 ro, const CwRay& cr, float tmax) {
    const uint4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2), n3 = __ldg(nd + 3), n4 = __ldg(nd + 4);
    const f3 p(__uint_as_float(n0.x), __uint_as_float(n0.y), __uint_as_float(n0.z));
    const f3 dq = f3(__uint_as_float((n0.w & 0xFFu) << 23), __uint_as_float(((n0.w >> 8) & 0xFFu) << 23),
                     __uint_as_float(((n0.w >> 16) & 0xFFu) << 23)) * cr.inv;
    const f3 sc = dq * 32768.0f;
    const f3 c = (p - ro) * cr.inv - sc;
    const f3 pad(__fmaf_rn(fabsf(c.x), kCwPadOffset, fabsf(dq.x) * kCwPad), __fmaf_rn(fabsf(c.y), kCwPadOffset, fabsf(dq.y) * kCwPad),
                 __fmaf_rn(fabsf(c.z), kCwPadOffset, fabsf(dq.z) * kCwPad));
    const f3 cn = c - pad, cf = c + pad;
    const bool px = (cr.octinv & 1u) != 0u, py = (cr.octinv & 2u) != 0u, pz = (cr.octinv & 4u) != 0u;   // direction >= 0
    unsigned hm = 0u;
#pragma unroll
    for (unsigned half = 0u; half < 2u; ++half) {
        const unsigned lx = half ? n2.y : n2.x, ly = half ? n2.w : n2.z, lz = half ? n3.y : n3.x;
        const unsigned hx = half ? n3.w : n3.z, hy = half ? n4.y : n4.x, hz = half ? n4.w : n4.z;
        const unsigned nx = px ? lx : hx, ny = py ? ly : hy, nz = pz ? lz : hz;
        const unsigned fx = px ? hx : lx, fy = py ? hy : ly, fz = pz ? hz : lz;
#pragma unroll
        for (unsigned k = 0u; k < 4u; ++k) {
            const float tn = fmaxf(fmaxf(cw_plane(nx, k, sc.x, cn.x), cw_plane(ny, k, sc.y, cn.y)),
                                   fmaxf(cw_plane(nz, k, sc.z, cn.z), 0.0f));
            const float tf = fminf(fminf(cw_plane(fx, k, sc.x, cf.x), cw_plane(fy, k, sc.y, cf.y)),
                                   fminf(cw_plane(fz, k, sc.z, cf.z), tmax)) * kBvhTfarPad;
            if (!(tf < tn)) hm |= 1u << (4u * half + k);
        }
    }
    CwNodeHits o;
    o.child_base = n1.x;
    o.leaf_base = n1.y;
    o.imask = (n0.w >> 24) & 0xFFu;
    o.leaf_bits = 0u;
    // hit leaf children: their items' bits (an empty slot has none)
    for (unsigned lm = hm & ~o.imask; lm != 0u; lm &= lm - 1u) {
        const unsigned sl = (unsigned)__ffs((int)lm) - 1u;
        const unsigned m = ((sl < 4u ? n1.z : n1.w) >> (8u * (sl & 3u))) & 0xFFu;
        o.leaf_bits |= (m >> 5) << (m & 0x1Fu);
    }
    // hit internal children, slot s at bit s ^ octinv
    unsigned h = hm & o.imask;
    if (cr.octinv & 1u) h = ((h & 0x55u) << 1) | ((h >> 1) & 0x55u);
    if (cr.octinv & 2u) h = ((h & 0x33u) << 2) | ((h >> 2) & 0x33u);
    if (cr.octinv & 4u) h = ((h & 0x0Fu) << 4) | (h >> 4);
    o.hits = h;
    return o;
}
// The next child of a node group: pops the highest hit bit and maps it to the child index.
__device__ __forceinline__ unsigned cw_next_child(unsigned& g_hits, unsigned g_base, unsigned g_imask, unsigned octinv) {
    int bit = find_msb24(g_hits);
    g_hits &= ~(1u << (unsigned)bit);
    unsigned slot = ((unsigned)bit ^ octinv) & 7u;
    return g_base + __popc(g_imask & ((1u << slot) - 1u));
}

// Leaf(item) for one leaf item index (wide-order); returns true to stop.
template <class Leaf>
__device__ __forceinline__ bool walk_wide(const DevScene& S, const uint4* nodes, f3 ro, f3 rd, const float& tmax, Leaf leaf,
                                          unsigned* visits = nullptr) {
    const CwRay cr = cw_ray(rd);
    // node-group stack in thread-local memory (a wide TLAS walk nests a BLAS walk inside
    // its leaves, each with its own stack)
    uint2 stack[kCwStack];
    int ptr = -1;
    unsigned g_base = 0u, g_hits = 1u << (cr.octinv & 7u), g_imask = 1u;
    for (int guard = 0; guard < 65536; guard++) {
        if (g_hits == 0u) {   // pop a group and go on to its next node in the same iteration
            if (ptr < 0) return false;
            const uint2 top = stack[ptr];
            g_base = top.x;
            g_hits = top.y & 0xFFu;
            g_imask = top.y >> 8;
            ptr--;
        }
        const unsigned child = cw_next_child(g_hits, g_base, g_imask, cr.octinv);
        if (g_hits != 0u) {
            if (ptr + 1 < kCwStack) { ptr++; stack[ptr] = make_uint2(g_base, g_hits | (g_imask << 8)); }
            else flag_error(S, kErrCwStack);
        }
        if (visits) (*visits)++;
        const CwNodeHits nh = cw_node(nodes + 5 * (size_t)child, ro, cr, tmax);
        unsigned leaf_bits = nh.leaf_bits;
        while (leaf_bits != 0u) {
            int lb = find_msb24(leaf_bits);
            leaf_bits &= ~(1u << (unsigned)lb);
            if (leaf((int)nh.leaf_base + lb)) return true;
        }
        if (nh.hits != 0u) { g_base = nh.child_base; g_hits = nh.hits; g_imask = nh.imask; }
        else g_hits = 0u;
    }
    flag_error(S, kErrCwGuard);
    return false;
}

// Whether the program walks this mesh's compressed wide BVH (else its binary one).
__device__ __forceinline__ bool walks_cwbvh(const DevScene& S, const DevMesh& m) {
    return (PTR_SPEC_ACCEL < 0 ? S.accel : PTR_SPEC_ACCEL) == PTR_ACCEL_CWBVH && m.cwbvh;
}

// ---- one mesh BLAS in a given frame (ro/rd already in the mesh's local frame) --------------
// tie_in(): whether this walk wins a tie with the incoming tmax (a lower instance index
// than the hit that set it); ties inside the walk go to the lower triangle index.
template <class Tie = NoTie>
__device__ __forceinline__ bool mesh_nearest(const DevScene& S, const DevMesh& m, f3 ro, f3 rd, float& tmax, int& prim,
                                             Work* w = nullptr, Tie tie_in = Tie{}) {
    bool found = false;
    const float4* tri = walks_cwbvh(S, m) ? m.tri_w : m.tri;
    auto take = [&](int i, float t) {
        return t > 0.0f && (t < tmax || (t == tmax && (found ? tri_orig(tri, i) < tri_orig(tri, prim) : tie_in())));
    };
    if (walks_cwbvh(S, m)) {
        walk_wide(S, m.cwbvh, ro, rd, tmax, [&](int i) {
            f3 a, e1, e2;
            if (w) w->tris++;
            load_tri(tri, i, a, e1, e2);
            float t;
            if (tri_test(ro, rd, a, e1, e2, t) && take(i, t)) { tmax = t; prim = i; found = true; }
            return false;
        }, w ? &w->nodes : nullptr);
    } else {
        walk_binary(S, m.bvh, ro, rd, tmax, [&](int off, int cnt) {
            for (int i = off; i < off + cnt; ++i) {
                f3 a, e1, e2;
                if (w) w->tris++;
                load_tri(tri, i, a, e1, e2);
                float t;
                if (tri_test(ro, rd, a, e1, e2, t) && take(i, t)) { tmax = t; prim = i; found = true; }
            }
            return false;
        }, w ? &w->nodes : nullptr);
    }
    return found;
}
__device__ __forceinline__ bool mesh_any(const DevScene& S, const DevMesh& m, f3 ro, f3 rd, float max_dist, Work* w = nullptr) {
    if (walks_cwbvh(S, m)) {
        const float4* tri = m.tri_w;
        return walk_wide(S, m.cwbvh, ro, rd, max_dist, [&](int i) {
            f3 a, e1, e2;
            if (w) w->tris++;
            load_tri(tri, i, a, e1, e2);
            float t;
            return tri_test(ro, rd, a, e1, e2, t) && t > 0.0f && t < max_dist;
        }, w ? &w->nodes : nullptr);
    }
    const float4* tri = m.tri;
    return walk_binary(S, m.bvh, ro, rd, max_dist, [&](int off, int cnt) {
        for (int i = off; i < off + cnt; ++i) {
            f3 a, e1, e2;
            if (w) w->tris++;
            load_tri(tri, i, a, e1, e2);
            float t;
            if (tri_test(ro, rd, a, e1, e2, t) && t > 0.0f && t < max_dist) return true;
        }
        return false;
    }, w ? &w->nodes : nullptr);
}

// ---- instanced meshes: TLAS over BLAS as one flat loop --------------------------------------
// The nested form (accel_closest / accel_any) runs each instance's BLAS walk to the end
// inside the TLAS leaf that reached it, so in a warp every lane whose TLAS step did not
// enter an instance waits for the other lanes' whole BLAS walks.  Here one loop advances
// each lane by one node, whichever tree the node belongs to: TLAS and BLAS are walked in the
// same node format by the same code (wide: compressed nodes of the wide TLAS and the CWBVH;
// binary: the two-float4 nodes of the binary TLAS and BVH), so lanes at either level do the
// same work and differ only in the ray's frame and the node array.  Entering an instance and
// leaving its BLAS are done on the way to the next node.  Hits and ties are those of the
// nested walks.  ANY: stop at the first triangle hit.
//
// The walk is resumable: init() for one ray, then step() until it reports the end.
// h takes every nearer hit at once; h.element is the placement's index in the order hit
// queries report (the binary TLAS leaf order unless the program walks the wide TLAS).
struct FlatScene {                         // what a walk reads of its batch and prototype
    const void* tlas;
    const void* blas;
    const float4* place;
    const float4* tri;
    const int* id;                         // caller's index of each placement of this walk's order
    const int* element;                    // reported index of each placement (NULL: its own)
    const int* element_id;                 // caller's index of a reported element
};
template <bool WIDE>
__device__ __forceinline__ FlatScene flat_scene(const DevScene& S, const DevBatch& b) {
    const DevMesh& m = S.meshes[b.proto_mesh];
    if (!WIDE) return FlatScene{b.tlas, m.bvh, b.place, m.tri, b.inst_id, nullptr, b.inst_id};
    const bool wide_ids = S.inst_accel == PTR_ACCEL_CWBVH;
    return FlatScene{b.tlas_w, m.cwbvh, b.place_w, m.tri_w, b.inst_id_w, wide_ids ? nullptr : b.slot_of_w,
                     wide_ids ? b.inst_id_w : b.inst_id};
}
template <bool WIDE> struct FlatStack { using Entry = uint2; static constexpr int kSize = 2 * kCwStack; };
template <> struct FlatStack<false> { using Entry = int; static constexpr int kSize = 2 * kBvhStack; };
template <bool WIDE>
struct FlatWalk {
    using Entry = typename FlatStack<WIDE>::Entry;
    Entry stack[FlatStack<WIDE>::kSize];   // both levels share it
    f3 ro, rd;                             // the ray in the frame of the level walked last
    CwRay cr;                              // its reciprocal (wide: and octant)
    int ptr, bottom;                       // stack top; the top when the current instance was entered
    unsigned g_base, g_hits, g_imask;      // wide: the node group under way
    float A, B;                            // binary: words of the node to expand, g_base, when g_hits != 0
    unsigned leaf_base, leaf_left;         // the TLAS leaf's placements still to enter (wide: bits, binary: count)
    int inst;
    bool blas, world, found;               // level; the frame is the world's; this instance holds the hit
    __device__ __forceinline__ void frame(const f3 o, const f3 d) {
        ro = o;
        rd = d;
        if (WIDE) cr = cw_ray(d);
        else cr.inv = f3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    }
    __device__ __forceinline__ void root(const FlatScene& fs, float tmax, Work* w) {
        if constexpr (WIDE) {
            g_base = 0u;
            g_hits = 1u << (cr.octinv & 7u);
            g_imask = 1u;
        } else {
            load(fs, 0, tmax, w);
        }
    }
    __device__ __forceinline__ void push(const DevScene& S, Entry e) {
        if (ptr + 1 < FlatStack<WIDE>::kSize) stack[++ptr] = e;
        else flag_error(S, WIDE ? kErrCwStack : kErrBvhStack);
    }
    __device__ __forceinline__ void push_group(const DevScene& S) {
        if constexpr (WIDE) push(S, make_uint2(g_base, g_hits | (g_imask << 8)));
    }
    // Binary: node ni becomes the one to expand if the ray meets its box.
    __device__ __forceinline__ void load(const FlatScene& fs, int ni, float tmax, Work* w) {
        const float4* nodes = (const float4*)(blas ? fs.blas : fs.tlas);
        const float4 n0 = __ldg(nodes + 2 * (size_t)ni), n1 = __ldg(nodes + 2 * (size_t)ni + 1);
        if (w) { if (blas) w->nodes++; else w->tlas++; }
        g_hits = aabb_hit(n0, n1, ro, cr.inv, tmax) ? 1u : 0u;
        g_base = (unsigned)ni;
        A = n0.w;
        B = n1.w;
    }
    // Binary: both children of an inner node are met here, the nearer along the split axis
    // goes on and the other waits, so a node the ray misses costs no step of its own.
    __device__ __forceinline__ void expand(const DevScene& S, const FlatScene& fs, float tmax, Work* w) {
        const int axis = (int)(-A - 1.0f);
        const bool nf = (axis == 0 ? rd.x : (axis == 1 ? rd.y : rd.z)) >= 0.0f;
        const int L = (int)g_base + 1, R = (int)B, near = nf ? L : R, far = nf ? R : L;
        const float4* nodes = (const float4*)(blas ? fs.blas : fs.tlas);
        const float4 a0 = __ldg(nodes + 2 * (size_t)near), a1 = __ldg(nodes + 2 * (size_t)near + 1);
        const float4 b0 = __ldg(nodes + 2 * (size_t)far), b1 = __ldg(nodes + 2 * (size_t)far + 1);
        if (w) { if (blas) w->nodes += 2; else w->tlas += 2; }
        const bool ha = aabb_hit(a0, a1, ro, cr.inv, tmax), hb = aabb_hit(b0, b1, ro, cr.inv, tmax);
        g_hits = ha || hb ? 1u : 0u;
        g_base = (unsigned)(ha ? near : far);
        A = ha ? a0.w : b0.w;
        B = ha ? a1.w : b1.w;
        if constexpr (!WIDE) {
            if (ha && hb) push(S, far);
        }
    }
    __device__ __forceinline__ void init(const FlatScene& fs, const Ray& r, float tmax, Work* w) {
        frame(r.o, r.d);
        ptr = bottom = -1;
        leaf_left = 0u;
        blas = found = false;
        world = true;
        root(fs, tmax, w);
    }
    // One node; false once the query is over (any-hit: with found set at the first hit).
    template <bool ANY>
    __device__ __forceinline__ bool step(const DevScene& S, const FlatScene& fs, int region, const Ray& r, HitRec& h, float max_dist, Work* w) {
        if (g_hits == 0u && blas && ptr == bottom) blas = false;   // the instance is done
        if (!blas && leaf_left != 0u) {                            // enter the TLAS leaf's next placement
            if (WIDE) {
                if (g_hits != 0u) push_group(S);
                const int lb = find_msb24(leaf_left);
                leaf_left &= ~(1u << (unsigned)lb);
                inst = (int)leaf_base + lb;
            } else {
                inst = (int)leaf_base++;
                leaf_left--;
            }
            const float4 q = __ldg(fs.place + 2 * (size_t)inst), ts = __ldg(fs.place + 2 * (size_t)inst + 1);
            if (w) w->inst++;
            frame(placement_rigid(q, ts, r.o) / ts.w, qrot(q, r.d) / ts.w);
            blas = true;
            world = found = false;
            bottom = ptr;
            root(fs, ANY ? max_dist : h.t, w);
        } else {
            if (g_hits == 0u && ptr < 0) return false;
            if (!blas && !world) {
                frame(r.o, r.d);
                world = true;
            }
            if (g_hits == 0u) {
                const Entry top = stack[ptr--];
                if constexpr (WIDE) {
                    g_base = top.x;
                    g_hits = top.y & 0xFFu;
                    g_imask = top.y >> 8;
                } else {
                    load(fs, top, ANY ? max_dist : h.t, w);   // against the hit found since it was pushed
                }
            }
        }
        if constexpr (!WIDE) {
            if (g_hits == 0u) return true;
            if (A < 0.0f) {
                expand(S, fs, ANY ? max_dist : h.t, w);
                if (g_hits == 0u || A < 0.0f) return true;
            }
            g_hits = 0u;                                       // a leaf of A items from B
            if (!blas) {
                leaf_base = (unsigned)B;
                leaf_left = (unsigned)A;
                return true;
            }
            for (int i = (int)B; i < (int)B + (int)A; ++i)
                if (triangle<ANY>(fs, i, region, h, max_dist, w)) return false;
        } else {
            const unsigned child = cw_next_child(g_hits, g_base, g_imask, cr.octinv);
            if (g_hits != 0u) push_group(S);
            if (w) { if (blas) w->nodes++; else w->tlas++; }
            const CwNodeHits nh = cw_node((const uint4*)(blas ? fs.blas : fs.tlas) + 5 * (size_t)child, ro, cr, ANY ? max_dist : h.t);
            g_base = nh.child_base;
            g_hits = nh.hits;
            g_imask = nh.imask;
            if (!blas) {
                leaf_base = nh.leaf_base;
                leaf_left = nh.leaf_bits;
                return true;
            }
            for (unsigned bits = nh.leaf_bits; bits != 0u;) {
                const int lb = find_msb24(bits);
                bits &= ~(1u << (unsigned)lb);
                if (triangle<ANY>(fs, (int)nh.leaf_base + lb, region, h, max_dist, w)) return false;
            }
        }
        return true;
    }
    // Leaf triangle i; true ends an any-hit query.
    template <bool ANY>
    __device__ __forceinline__ bool triangle(const FlatScene& fs, int i, int region, HitRec& h, float max_dist, Work* w) {
        f3 a, e1, e2;
        if (w) w->tris++;
        load_tri(fs.tri, i, a, e1, e2);
        float t;
        if (!tri_test(ro, rd, a, e1, e2, t) || !(t > 0.0f)) return false;
        if (ANY) {
            found = t < max_dist;
            return found;
        }
        if (t < h.t || (t == h.t && (found ? tri_orig(fs.tri, i) < tri_orig(fs.tri, h.prim)
                                           : (h.region == region && __ldg(fs.id + inst) < __ldg(fs.element_id + h.element))))) {
            h.t = t;
            h.region = region;
            h.element = fs.element ? __ldg(fs.element + inst) : inst;
            h.prim = i;
            found = true;
        }
        return false;
    }
};
constexpr int kFlatGuard = 1 << 22;        // steps of one query before the walk gives up
template <bool WIDE, bool ANY>
__device__ __forceinline__ bool flat_walk(const DevScene& S, const DevBatch& b, int region, const Ray& r, HitRec& h, float max_dist, Work* w) {
    const FlatScene fs = flat_scene<WIDE>(S, b);
    FlatWalk<WIDE> f;
    f.init(fs, r, ANY ? max_dist : h.t, w);
    for (int guard = 0; guard < kFlatGuard; ++guard)
        if (!f.template step<ANY>(S, fs, region, r, h, max_dist, w)) return ANY && f.found;
    flag_error(S, kErrCwGuard);
    return false;
}
// The flat loops a batch takes: wide for mesh prototypes walked as CWBVH (with the wide TLAS,
// whichever TLAS the program names: hits do not depend on it), binary for prototypes walked
// as binary BVH under the binary TLAS.  The rest keep the nested walks.
__device__ __forceinline__ bool flat_wide_ok(const DevScene& S, const DevBatch& b) {
    return kHasMesh && PTR_SPEC_ACCEL != PTR_ACCEL_BVH && b.proto_shape == PTR_SHAPE_MESH && b.tlas_w &&
           walks_cwbvh(S, S.meshes[b.proto_mesh]);
}
__device__ __forceinline__ bool flat_binary_ok(const DevScene& S, const DevBatch& b) {
    return kHasMesh && PTR_SPEC_ACCEL != PTR_ACCEL_CWBVH && b.proto_shape == PTR_SHAPE_MESH &&
           !walks_cwbvh(S, S.meshes[b.proto_mesh]) && !(S.inst_accel == PTR_ACCEL_CWBVH && b.tlas_w);
}

// ---- region arms ------------------------------------------------------------------------
// Inlined, but for the shadow queries through media (and the point classification) of the
// library's generic kernels, which call them (ptx_rt.cu defines PTR_ACCEL_CALL): inlined next to
// every arm of a media query, the tree walks' registers spilled across the region scans (fog with
// 256 lamps and a mesh, 512 x 384 x 8: 25.3 ms with every arm inlined, 20.7 with every arm called).
// The closest hits and the opaque queries lose more by the call than it saves: k_closest of a
// 512 x 512 x 8 frame around one 320-triangle mesh takes 0.78 ms inlined and 0.99 called, around
// one 327,680-triangle mesh at 640 x 360 x 4 1.63 and 1.97; the kernels of the lamps in fog 17.9
// and 19.6 ms.
#ifndef PTR_ACCEL_CALL
#define PTR_ACCEL_CALL __forceinline__
#endif
__device__ __forceinline__ HitRec accel_closest(const DevScene& S, const ptr_region& g, int region, Ray r, HitRec h,
                                               Work* w = nullptr) {
    if (kHasMesh && g.shape == PTR_SHAPE_MESH) {
        const DevMesh& m = S.meshes[g.ref];
        int prim = -1;
        float t = h.t;
        if (mesh_nearest(S, m, r.o, r.d, t, prim, w)) {
            h.t = t;
            h.region = region;
            h.element = 0;
            h.prim = prim;
        }
        return h;
    }
    const DevBatch& b = S.batches[g.ref];
    if (flat_wide_ok(S, b)) { flat_walk<true, false>(S, b, region, r, h, 0.0f, w); return h; }
    if (flat_binary_ok(S, b)) { flat_walk<false, false>(S, b, region, r, h, 0.0f, w); return h; }
    float t_near = h.t;
    const bool wide = S.inst_accel == PTR_ACCEL_CWBVH && b.tlas_w;
    const float4* place = wide ? b.place_w : b.place;
    const int* inst_id = wide ? b.inst_id_w : b.inst_id;
    // an instance wins a tie with the current hit when that hit is an instance of this
    // batch with a higher placement index
    auto wins_tie = [&](int i) { return h.region == region && __ldg(inst_id + i) < __ldg(inst_id + h.element); };
    // one instance: the params-tier sphere, or the mesh prototype in the placement's frame
    auto instance = [&](int i) {
        if (!kHasMesh || b.proto_shape == PTR_SHAPE_SPHERE) {
            float4 rec = __ldg(place + 2 * i);
            float t;
            if (sphere_intersect(r, xyz(rec), rec.w, t) && (t < t_near || (t == t_near && wins_tie(i)))) {
                t_near = t; h.t = t; h.region = region; h.element = i; h.prim = -1;
            }
        } else {
            float4 q = __ldg(place + 2 * i), ts = __ldg(place + 2 * i + 1);
            float s = ts.w;
            if (w) w->inst++;
            f3 ro = placement_rigid(q, ts, r.o) / s;
            f3 rd = qrot(q, r.d) / s;
            int prim = -1;
            float t = t_near;
            if (mesh_nearest(S, S.meshes[b.proto_mesh], ro, rd, t, prim, w, [&] { return wins_tie(i); })) {
                t_near = t; h.t = t; h.region = region; h.element = i; h.prim = prim;
            }
        }
    };
    if (wide) {   // the reference's CWBVH instance accel (intersection/index.ts:99-158)
        walk_wide(S, b.tlas_w, r.o, r.d, t_near, [&](int i) { instance(i); return false; }, w ? &w->tlas : nullptr);
        return h;
    }
    walk_binary(S, b.tlas, r.o, r.d, t_near, [&](int off, int cnt) {
        for (int i = off; i < off + cnt; ++i) instance(i);
        return false;
    }, w ? &w->tlas : nullptr);
    return h;
}

__device__ __forceinline__ bool accel_any(const DevScene& S, const ptr_region& g, Ray r, float max_dist,
                                          Work* w = nullptr) {
    if (kHasMesh && g.shape == PTR_SHAPE_MESH) return mesh_any(S, S.meshes[g.ref], r.o, r.d, max_dist, w);
    const DevBatch& b = S.batches[g.ref];
    HitRec unused;
    if (flat_wide_ok(S, b)) return flat_walk<true, true>(S, b, 0, r, unused, max_dist, w);
    if (flat_binary_ok(S, b)) return flat_walk<false, true>(S, b, 0, r, unused, max_dist, w);
    const bool wide = S.inst_accel == PTR_ACCEL_CWBVH && b.tlas_w;
    const float4* place = wide ? b.place_w : b.place;
    auto instance = [&](int i) -> bool {
        if (!kHasMesh || b.proto_shape == PTR_SHAPE_SPHERE) {
            float4 rec = __ldg(place + 2 * i);
            float t;
            return sphere_intersect(r, xyz(rec), rec.w, t) && t < max_dist;
        }
        float4 q = __ldg(place + 2 * i), ts = __ldg(place + 2 * i + 1);
        float s = ts.w;
        if (w) w->inst++;
        f3 ro = placement_rigid(q, ts, r.o) / s;
        f3 rd = qrot(q, r.d) / s;
        return mesh_any(S, S.meshes[b.proto_mesh], ro, rd, max_dist, w);
    };
    if (wide) return walk_wide(S, b.tlas_w, r.o, r.d, max_dist, instance, w ? &w->tlas : nullptr);
    return walk_binary(S, b.tlas, r.o, r.d, max_dist, [&](int off, int cnt) {
        for (int i = off; i < off + cnt; ++i)
            if (instance(i)) return true;
        return false;
    }, w ? &w->tlas : nullptr);
}

// The same arms as calls.
__device__ PTR_ACCEL_CALL HitRec accel_closest_call(const DevScene& S, const ptr_region& g, int region, Ray r, HitRec h, Work* w) {
    return accel_closest(S, g, region, r, h, w);
}
__device__ PTR_ACCEL_CALL bool accel_any_call(const DevScene& S, const ptr_region& g, Ray r, float max_dist, Work* w) {
    return accel_any(S, g, r, max_dist, w);
}

// Containment of an instanced SPHERE batch (the TLAS point descent of scene_region_at):
// the least-negative signed distance among the instances that contain p, else 1e20.
// Mesh batches are thin (no containment).
__device__ PTR_ACCEL_CALL float accel_region_sdf(const DevScene& S, const ptr_region& g, f3 p) {
    const DevBatch& b = S.batches[g.ref];
    if (b.proto_shape != PTR_SHAPE_SPHERE) return 1.0e20f;
    float best = -1.0e20f;
    bool any = false;
    int stack[kBvhStack];
    int ptr = 0;
    stack[0] = 0;
    while (ptr >= 0) {
        int ni = stack[ptr];
        ptr--;
        float4 n0 = __ldg(b.tlas + 2 * ni), n1 = __ldg(b.tlas + 2 * ni + 1);
        if (!(p.x >= n0.x && p.y >= n0.y && p.z >= n0.z && p.x <= n1.x && p.y <= n1.y && p.z <= n1.z)) continue;
        if (n0.w >= 0.0f) {
            int off = (int)n1.w, cnt = (int)n0.w;
            for (int i = off; i < off + cnt; ++i) {
                float4 rec = __ldg(b.place + 2 * i);
                float ds = length(p - xyz(rec)) - rec.w;
                if (ds < 0.0f && ds > best) { best = ds; any = true; }
            }
        } else {
            int L = ni + 1, R = (int)n1.w;
            if (ptr + 2 < kBvhStack) { stack[++ptr] = L; stack[++ptr] = R; }
            else flag_error(S, kErrBvhStack);
        }
    }
    return any ? best : 1.0e20f;
}

// Hit normals of an acceleration-structure hit (world space): shading normal (returned)
// and the geometric normal (h.ng), plus eps and the per-triangle alpha.
__device__ __forceinline__ f3 accel_hit_normal(const DevScene& S, const ptr_region& g, const HitRec& hr, const Ray&, Hit& h, f3& ng) {
    h.eps = fp_uncertainty(h.p);
    if (g.shape == PTR_SHAPE_INSTANCES) {
        const DevBatch& b = S.batches[g.ref];
        // hr.element indexes the placements of the TLAS the hit was found with
        const float4* place = (S.inst_accel == PTR_ACCEL_CWBVH && b.tlas_w) ? b.place_w : b.place;
        if (!kHasMesh || b.proto_shape == PTR_SHAPE_SPHERE) {
            float4 rec = __ldg(place + 2 * hr.element);
            f3 n = normalize(h.p - xyz(rec));
            ng = n;   // a primitive's normal is its true surface normal (set from frame.n)
            return n;
        }
        const DevMesh& m = S.meshes[b.proto_mesh];
        float4 q = __ldg(place + 2 * hr.element);
        const float4* tri = walks_cwbvh(S, m) ? m.tri_w : m.tri;
        f3 a, e1, e2;
        load_tri(tri, hr.prim, a, e1, e2);
        f3 gl = cross(e1, e2);
        float al = __ldg(&tri[3 * hr.prim + 1].w);
        if (al >= 0.0f) h.alpha = al;
        ng = normalize(placement_normal(q, gl));
        return normalize(placement_normal(q, gl));
    }
    const DevMesh& m = S.meshes[g.ref];
    const float4* tri = walks_cwbvh(S, m) ? m.tri_w : m.tri;
    f3 a, e1, e2;
    load_tri(tri, hr.prim, a, e1, e2);
    f3 gl = cross(e1, e2);
    float al = __ldg(&tri[3 * hr.prim + 1].w);
    if (al >= 0.0f) h.alpha = al;
    ng = normalize(gl);
    return normalize(gl);
}

}  // namespace ptx
