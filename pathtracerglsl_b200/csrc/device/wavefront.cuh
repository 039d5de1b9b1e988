// wavefront.cuh — the transport loop, as a wavefront of kernels over a path pool and as one
// kernel per wave.
//
// The reference runs the whole walk (transport/integrators/pt/pt.ts:299-464) as one
// fragment per pixel.  Scenes without triangle meshes do so here too: k_walk runs a path in
// one thread, its state in registers, and k_film_walk / k_film_batch_walk fold the wave into
// the film.  With meshes (and for large spectral frames) each path lives in struct-of-arrays
// state in HBM and the walk is split at its two traversals:
//
//   k_generate  camera rays + path_state_init for one wave of (pixel, sample) paths
//   k_closest   nearest hit of every live path (the scene_intersect traversal)
//   k_shade     one walk iteration: medium segment, null pass-through, emitter scoring,
//               NEE sampling (emits a shadow query), BSDF continuation, roulette, spawn;
//               live paths are compacted into the next queue with warp ballots
//   k_shadow    visibility / transmittance of the queued shadow queries, folded into
//               the owning path's radiance
//   k_film      per-pixel FP64 sum and sum of squares over the wave's samples
//
// Both forms share one iteration (walk_iteration) and one shadow query (shadow_visibility).
// Every path draws its random numbers in exactly the order of the reference's walk
// (the sampler is counter-based, so a path's stream does not depend on scheduling), and
// its radiance is accumulated in the same order: emission, then the vertex's NEE term,
// then the next vertex's emission.
#pragma once
#include "occupants.cuh"
#include "bvh.cuh"
#include "adjoint.cuh"
#include "materials/registry.cuh"

namespace ptx {

// Path pool (indexed by path slot).
// One field of a two-field path record: path i's value at p[2 i] and the partner field's
// at p[2 i + 1], so the two 16-byte fields a kernel reads and writes together fill one
// 32-byte sector (a surviving path's store never half-fills a sector that the L2 would
// first have to read back from DRAM).
template <class T> struct Pair {
    T* p;
    __host__ __device__ __forceinline__ T& operator[](long long i) const { return p[2 * i]; }
    __host__ __device__ __forceinline__ explicit operator bool() const { return p != nullptr; }
};

struct PathPool {
    Pair<float4> ray_o;  // origin.xyz, prev_bsdf_pdf          } one record
    Pair<float4> ray_d;  // direction.xyz, eta_scale           }
    Pair<float4> thr;    // throughput.xyz, -                  } one record
    Pair<float4> rad;    // radiance.xyz, -                    }
    Pair<float4> prev_q; // stored light-query point (prev_query.p)  } one record, with st
    float4* prev_n;    // stored light-query normal and two-sidedness (light-tree selection)
    unsigned* sh_seed; // the shadow query's sampler dimension at its NEE site (heterogeneous media)
    // first-hit pictures (programs with measurement.aovs; NULL otherwise): per path its
    // albedo and normal samples (2 float4), per pixel their FP64 sums (albedo block of 3
    // doubles per pixel, then the normal block)
    float4* aov;
    double* aov_sum;
    Pair<int4> st;       // bounce, current_medium, null_crossings, prev_was_delta
    uint2* rng;        // sampler base, dimension
    Pair<float4> hit;    // t, u, v, - ; (region, element, prim) in hit_i    } one record
    Pair<int4> hit_i;    // region_owner, element, prim, -                   }
    // shadow queries (one per path and iteration at most)
    Pair<float4> sh_o;   // origin.xyz, max distance (opaque form)     } one record
    Pair<float4> sh_d;   // direction.xyz, crossings left (as int)     }
    Pair<float4> sh_lp;  // light point.xyz, MIS weight                } one record
    Pair<float4> sh_c;   // contribution prefix throughput*Le*f*cos (xyz), pdf  }
    // second shadow slot: the per-segment equiangular query of the same iteration (a path
    // may issue it and a surface NEE query in one walk iteration); NULL when unused
    Pair<float4> sh2_o;
    Pair<float4> sh2_d;
    Pair<float4> sh2_lp;
    Pair<float4> sh2_c;
    int* q[2];         // live-path queues (ping-pong)
    int* shq;          // shadow queue
    int* shq2;         // second-slot shadow queue (count in cnt[4])
    unsigned int* cnt; // [0],[1] queue counts, [2] shadow count, [3] error flags, [4] slot-2 shadow count
    unsigned long long* stats; // [0] closest queries, [1] shadow queries, [2] paths
    long long* wave;   // [0] first global path index of the wave, [1] wave size
    // adjoint replay only (NULL otherwise)
    float4* l_rem;     // radiance the path has still to gather (forward total minus what it gathered)
    float4* dl;        // adjoint radiance of the path: dLoss/dI of its pixel / spp
    float4* sh_g;      // shadow query: lobe derivative D = dlog f(wi_light) - dlog w_cont (xyz)
    int* sh_gm;        // shadow query: vertex material | kind << 16
    // spectral colour model only (NULL otherwise): the path's four wavelengths and their
    // sampling densities; the shadow queries' pdfs (the colour fills all four lanes)
    float4* wl;
    float4* wl_pdf;
    float* sh_pdf;
    float* sh2_pdf;
    // occupant-sorted shading queue: k_closest keys every live path by the occupant it will
    // shade (material model of the hit, inside a medium or not) and counts the keys; a scan
    // and a scatter rebuild the live queue grouped by key before k_shade (sort_buckets <= 1:
    // off, k_shade reads the compacted queue as it is)
    int sort_buckets;
    int* q_sorted;
    unsigned char* sort_key;  // shading class per path (indexed by path)
    unsigned* sort_hist;      // counting-sort scratch: [key][chunk] counts, then offsets
    // work tickets of the queue kernels ([0] k_closest, [1] / [2] k_shadow slots 0 / 1,
    // [3] k_shade), each cleared by the kernel that runs before its consumer; NULL: the
    // kernels fall back to a static grid-stride loop
    unsigned* fetch;
    // ray-coherence order (tuning ray_sort): k_shade keys every spawned ray and every shadow
    // query by (direction octant, origin octant about the scene centre); counting sorts
    // rebuild the closest-hit and shadow queues grouped by key for the traversal kernels
    // (k_shade itself keeps reading the compacted queue q[in])
    int ray_sort;             // keys and sorted queues are written
    int ray_in;               // this k_closest reads q_ray (set per launch; 0 for camera rays)
    unsigned char* rkey;      // key per position of the next live queue
    unsigned char* skey;      // key per position of the shadow queue
    int* q_ray;
    int* shq_s;
    // the adjoint's walk log (ptr_backward; NULL otherwise): for walk iterations below
    // hit_log_iters the forward walk records, per path, four float4 at
    // [4 * (iter * hit_log_stride + path)]: its closest hit (hit, hit_i), then its slot-0
    // shadow query's visibility and media (ShadowLog).  The replay of the same paths reads
    // them back instead of walking the scene again.  iter and hit_log_mode (1 record,
    // 2 replay) are set per launch.
    float4* hit_log;
    long long hit_log_stride;
    int hit_log_iters, hit_log_mode, iter;
    int lockstep;      // k_shade: a block's warps run each part of an iteration together
};

constexpr int kRayBuckets = 64;   // ray_key values
__device__ __forceinline__ unsigned ray_key(const DevScene& S, f3 o, f3 d) {
    unsigned k = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    k = (k << 3) | (o.x > S.sort_c[0] ? 1u : 0u) | (o.y > S.sort_c[1] ? 2u : 0u) | (o.z > S.sort_c[2] ? 4u : 0u);
    return k;
}
// The adjoint's hit log of this launch's iteration (null where it is not logged).
__device__ __forceinline__ float4* hit_log_slice(const PathPool& pool) {
    return pool.hit_log && pool.iter < pool.hit_log_iters ? pool.hit_log + 4 * (size_t)pool.iter * (size_t)pool.hit_log_stride : nullptr;
}
// The queue a k_closest of iteration `in` reads.
__device__ __forceinline__ const int* closest_queue(const PathPool& pool, int in);

// Warp-uniform cursor over a device-counted queue.  With a ticket counter every warp takes
// the next 32 entries when it is done with its last ones, so warps whose rays are long do
// not hold the others' work back (dynamic balance on a one-wave resident grid); without
// one, a grid-stride loop whose trip count is rounded to whole warps.
struct QueueCursor {
    unsigned n, stride, k;
    unsigned* ticket;
    __device__ __forceinline__ QueueCursor(unsigned n_, unsigned* t) : n(n_), ticket(t) {
        stride = gridDim.x * blockDim.x;
        k = blockIdx.x * blockDim.x + threadIdx.x - stride;
    }
    __device__ __forceinline__ bool next(unsigned& out) {
        if (ticket) {
            unsigned base = 0u;
            if ((threadIdx.x & 31u) == 0u) base = atomicAdd(ticket, 32u);
            base = __shfl_sync(0xffffffffu, base, 0);
            out = base + (threadIdx.x & 31u);
            return base < n;
        }
        k += stride;
        out = k;
        return k < ((n + 31u) & ~31u);
    }
};

// The same cursor with the option of a block's warps starting every round together (lockstep:
// uniform over the grid; needs the ticket counter).
struct ShadeCursor {
    QueueCursor warp;
    bool lockstep;
    __device__ __forceinline__ ShadeCursor(unsigned n, unsigned* t, bool lock) : warp(n, t), lockstep(lock && t) {}
    __device__ __forceinline__ bool next(unsigned& out) {
        if (!lockstep) return warp.next(out);
        __shared__ unsigned base;
        __syncthreads();
        if (threadIdx.x == 0) base = atomicAdd(warp.ticket, blockDim.x);
        __syncthreads();
        out = base + threadIdx.x;
        return base < warp.n;
    }
    __device__ __forceinline__ void phase() const {
        if (lockstep) __syncthreads();
    }
};

// Adjoint replay tables: the adjoint image (3 floats per pixel, row 0 at the bottom), the
// per-sample scale and the float64 gradient buffer (PTR_GRAD_SLOTS per material).
struct AdjParams {
    const float* dl_image;
    float inv_spp;
    double* grads;
};

struct FrameParams {
    int width, height, spp, first_sample;
    uint32_t salt;
    int px_off, py_off;
    int img_w, img_h;  // the full image the camera maps film points through
    long long total;   // width*height*spp
    int capacity;
    ptr_camera cam;
    int wavelengths;   // PTR_WAVELENGTHS_* (spectral programs)
    float lambda_min, lambda_max;
    int fresh;         // 1: the film starts from zero at each pixel's first sample of this frame
};

struct ProgParams {
    int max_bounces, direct, rr_start, max_null;
    float rr_max_survival;
    int scattering;
    int equiangular;   // PTR_EQUIANGULAR_*: per-segment medium NEE replaces the at-vertex site
    int light_tree;    // light-tree selection (the scene carries the tree)
};

// Batched renders: per job its scene, program knobs, frame and film; offsets[j] is the
// first global path index of job j (offsets[n_jobs] = total paths).
struct BatchJob {
    FrameParams frame;
    double* sum;
    double* sumsq;
};
struct BatchTables {
    const DevScene* scenes;
    const ProgParams* progs;
    const BatchJob* jobs;
    const long long* offsets;
    int n_jobs;
    long long total;
    int capacity;
};

// The job of global path index g: the last j with offsets[j] <= g.  A batched wave's pool
// slot i holds path base + i for the whole wave (base = pool.wave[0]), so the kernels find a
// path's job from its slot by this search over the small, cached offsets table instead of
// a per-path load from HBM that every scene-table read would wait for.
__device__ __forceinline__ int job_of(const BatchTables& bt, long long g) {
    int lo = 0, hi = bt.n_jobs - 1;   // last j with offsets[j] <= g
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (bt.offsets[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The jobs of a batched wave's slots.  A wave that lies inside one job (every wave of a
// large job but its last) needs no search at all: its job is found once per thread.
struct WaveJobs {
    long long base = 0;
    int single = 0;   // >= 0: every slot of the wave belongs to this job
    WaveJobs() = default;
    __device__ __forceinline__ WaveJobs(const PathPool& pool, const BatchTables& bt) : WaveJobs(pool.wave[0], pool.wave[1], bt) {}
    __device__ __forceinline__ WaveJobs(long long base_, long long n, const BatchTables& bt) : base(base_) {
        const int j = job_of(bt, base);
        single = bt.offsets[j + 1] >= base + n ? j : -1;
    }
    __device__ __forceinline__ int of(const BatchTables& bt, int slot) const {
        return single >= 0 ? single : job_of(bt, base + slot);
    }
};

constexpr unsigned kErrStack = 1u;

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Warp-aggregated append: one atomic per warp, slots in lane order.
__device__ __forceinline__ int warp_append(unsigned* counter, bool pred) {
    unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0u) return -1;
    int lane = threadIdx.x & 31;
    int leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(counter, (unsigned)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    return pred ? (int)(base + __popc(mask & lanemask_lt())) : -1;
}

// ---- scene queries -------------------------------------------------------------------
// Nearest hit over every arm; returns region (or -1), element, primitive and t.  CALL (here and in
// scene_any): the library's generic kernels call the acceleration arms instead of inlining them
// (bvh.cuh).

__device__ __forceinline__ float4 int4_as_float4(int4 v) {
    return make_float4(__int_as_float(v.x), __int_as_float(v.y), __int_as_float(v.z), __int_as_float(v.w));
}
__device__ __forceinline__ int4 float4_as_int4(float4 v) {
    return make_int4(__float_as_int(v.x), __float_as_int(v.y), __float_as_int(v.z), __float_as_int(v.w));
}
template <int V> struct ShapeC { static constexpr int value = V; };
// Calls f(ShapeC<shape>{}, first, end) for each same-shape run of the region list, the
// shape a compile-time constant for the analytic shapes the build holds (one dispatch per
// run instead of one per region); other runs get f(ShapeC<-1>{}, ...).
template <class F>
__device__ __forceinline__ void for_region_runs(const DevScene& S, F&& f) {
    for (int q = 0; q < S.n_runs; ++q) {
        const int4 run = __ldg(S.region_runs + q);
        const int a = run.y, b = run.y + run.z;
        if (has_shape(PTR_SHAPE_SPHERE) && run.x == PTR_SHAPE_SPHERE) f(ShapeC<PTR_SHAPE_SPHERE>{}, a, b);
        else if (has_shape(PTR_SHAPE_QUAD) && run.x == PTR_SHAPE_QUAD) f(ShapeC<PTR_SHAPE_QUAD>{}, a, b);
        else f(ShapeC<-1>{}, a, b);
    }
}

// The root of region i of one analytic shape below limit, its parameters fetched as aligned
// float4s: an uploaded region table is 256-byte aligned and its records 80 bytes, so a
// record's bytes 16..79 are four float4s (ior, p[0..2]), (p[3..6]), (p[7..10]), (p[11..14]).
// Same operands as analytic_root_shape, fewer load instructions.
template <int SH>
__device__ __forceinline__ bool run_root(const DevScene& S, int i, const Ray& r, float limit, float& t) {
    const float4* g4 = reinterpret_cast<const float4*>(S.regions + i);
    if constexpr (SH == PTR_SHAPE_SPHERE) {
        const float4 a = __ldg(g4 + 1), b = __ldg(g4 + 2);
        return sphere_intersect(r, f3(a.y, a.z, a.w), b.x, t) && t < limit;
    } else {
        static_assert(SH == PTR_SHAPE_QUAD, "a run of spheres or quads");
        const float4 a = __ldg(g4 + 1), b = __ldg(g4 + 2), c = __ldg(g4 + 3), d = __ldg(g4 + 4);
        return quad_intersect_scan(r, f3(a.y, a.z, a.w), f3(b.x, b.y, b.z), f3(b.w, c.x, c.y), f3(c.z, c.w, d.x),
                                   __ldg(S.region_scan + i), limit, t);
    }
}
#ifndef __CUDACC_RTC__   // (NVRTC has no offsetof; the library build checks the layout)
static_assert(sizeof(ptr_region) == 80 && __builtin_offsetof(ptr_region, p) == 20, "run_root's float4 view of a region record");
#endif

// Calls hit(i) for the spheres [a, b) that may meet the ray, in ascending order, until it
// returns true.  A run is scanned 32 spheres at a time in two passes: the cheap condition
// marks the candidates of every lane (all lanes busy), then each lane runs the exact test of
// its own few.  In one pass a warp runs the root's square root and division at almost every
// sphere, for the one or two lanes that need it.
template <class F>
__device__ __forceinline__ bool for_sphere_candidates(const DevScene& S, const Ray& r, int a, int b, F&& hit) {
    const RayScan scan(r);
    for (int base = a; base < b; base += 32) {
        const int cnt = min(32, b - base);
        unsigned mask = 0u;
#pragma unroll 4
        for (int k = 0; k < cnt; ++k)
            if (scan.sphere(r, __ldg(S.region_scan + base + k))) mask |= 1u << k;
        while (mask) {
            const int k = __ffs(mask) - 1;
            mask &= mask - 1u;
            if (hit(base + k)) return true;
        }
    }
    return false;
}

template <bool CALL = true>
__device__ __forceinline__ HitRec scene_closest(const DevScene& S, const Ray& r, Work* w = nullptr) {
    HitRec h;
    h.t = kMaxDist;
    h.u = h.v = 0.f;
    h.region = -1;
    h.element = 0;
    h.prim = -1;
    auto take = [&](int i, float t) {
        h.t = t;
        h.region = i;
        h.element = 0;
        h.prim = -1;
    };
    auto arm = [&](int i, const ptr_region& g, int shape) {
        if (has_accel() && shape >= PTR_SHAPE_MESH) {
            h = CALL ? accel_closest_call(S, g, i, r, h, w) : accel_closest(S, g, i, r, h, w);
            return;
        }
        float t;
        if (analytic_root_shape(shape, g, r, t) && t < h.t) take(i, t);
    };
#if PTR_SPEC_NREGIONS > 0
    constexpr bool tabled = false;
#pragma unroll
    for (int k = 0; k < PTR_SPEC_NREGIONS; ++k) {
        const int sh = spec_shape(k);   // folds to a constant in each unrolled arm
        float t;
        bool hit = false;
        if (sh == PTR_SHAPE_SPHERE) hit = run_root<PTR_SHAPE_SPHERE>(S, k, r, h.t, t);
        else if (sh == PTR_SHAPE_QUAD) hit = run_root<PTR_SHAPE_QUAD>(S, k, r, h.t, t);
        else arm(k, S.regions[k], sh);
        if (hit) take(k, t);
    }
#else
    const bool tabled = PTR_SPEC_BVH && S.region_bvh != nullptr;
    if (!tabled && S.region_runs) {
        for_region_runs(S, [&](auto sc, int a, int b) {
            constexpr int SH = decltype(sc)::value;
            float t;
            if constexpr (SH == PTR_SHAPE_SPHERE) {
                for_sphere_candidates(S, r, a, b, [&](int i) {
                    if (run_root<SH>(S, i, r, h.t, t)) take(i, t);
                    return false;
                });
            } else {
                for (int i = a; i < b; ++i) {
                    if constexpr (SH == PTR_SHAPE_QUAD) {
                        if (run_root<SH>(S, i, r, h.t, t)) take(i, t);
                    } else {
                        arm(i, S.regions[i], S.regions[i].shape);
                    }
                }
            }
        });
    } else {
        const int n = tabled ? S.n_linear : S.n_regions;
        for (int k = 0; k < n; ++k) {
            const int i = tabled ? S.linear_regions[k] : k;
            arm(i, S.regions[i], S.regions[i].shape);
        }
    }
#endif
    if (tabled) {
        float tb = h.t;
        walk_binary(S, S.region_bvh, r.o, r.d, tb, [&](int off, int cnt) {
            for (int j = off; j < off + cnt; ++j) {
                const int i = S.region_items[j];
                float t;
                // strict '<', and on an exact tie the lower region index (the order of the
                // unrolled arms) keeps the hit
                if (analytic_root(S.regions[i], r, t) && (t < tb || (t == tb && h.region > i))) {
                    tb = t;
                    take(i, t);
                }
            }
            return false;
        });
    }
    return h;
}

template <bool CALL = true>
__device__ __forceinline__ bool scene_any(const DevScene& S, const Ray& r, float max_dist, Work* w = nullptr) {
    auto arm = [&](const ptr_region& g, int shape) -> bool {
        if (has_accel() && shape >= PTR_SHAPE_MESH) return CALL ? accel_any_call(S, g, r, max_dist, w) : accel_any(S, g, r, max_dist, w);
        float t;
        return analytic_root_shape(shape, g, r, t) && t < max_dist;
    };
#if PTR_SPEC_NREGIONS > 0
    constexpr bool tabled = false;
#pragma unroll
    for (int k = 0; k < PTR_SPEC_NREGIONS; ++k) {
        const int sh = spec_shape(k);   // folds to a constant in each unrolled arm
        float t;
        if (sh == PTR_SHAPE_SPHERE) {
            if (run_root<PTR_SHAPE_SPHERE>(S, k, r, max_dist, t)) return true;
        } else if (sh == PTR_SHAPE_QUAD) {
            if (run_root<PTR_SHAPE_QUAD>(S, k, r, max_dist, t)) return true;
        } else if (arm(S.regions[k], sh)) {
            return true;
        }
    }
#else
    const bool tabled = PTR_SPEC_BVH && S.region_bvh != nullptr;
    if (!tabled && S.region_runs) {
        bool hit = false;
        for (int q = 0; q < S.n_runs && !hit; ++q) {
            const int4 run = __ldg(S.region_runs + q);
            const int a = run.y, b = run.y + run.z;
            float t;
            if (has_shape(PTR_SHAPE_SPHERE) && run.x == PTR_SHAPE_SPHERE) {
                hit = for_sphere_candidates(S, r, a, b, [&](int i) { return run_root<PTR_SHAPE_SPHERE>(S, i, r, max_dist, t); });
            } else if (has_shape(PTR_SHAPE_QUAD) && run.x == PTR_SHAPE_QUAD) {
                for (int i = a; i < b && !hit; ++i) hit = run_root<PTR_SHAPE_QUAD>(S, i, r, max_dist, t);
            } else {
                for (int i = a; i < b && !hit; ++i) hit = arm(S.regions[i], S.regions[i].shape);
            }
        }
        if (hit) return true;
    } else {
        const int n = tabled ? S.n_linear : S.n_regions;
        for (int k = 0; k < n; ++k) {
            const int i = tabled ? S.linear_regions[k] : k;
            if (arm(S.regions[i], S.regions[i].shape)) return true;
        }
    }
#endif
    if (tabled) {
        return walk_binary(S, S.region_bvh, r.o, r.d, max_dist, [&](int off, int cnt) {
            for (int j = off; j < off + cnt; ++j) {
                float t;
                if (analytic_root(S.regions[S.region_items[j]], r, t) && t < max_dist) return true;
            }
            return false;
        });
    }
    return false;
}

// Innermost-wins point classification (features/intersection.ts:1121-1225); with a region
// BVH the bounded solids are found by the containment descent (bvh.ts bvhPointWalkLines).
__device__ __forceinline__ int scene_region_at(const DevScene& S, f3 p) {
    int region = -1;
    float best = -1.0e20f;
    auto arm = [&](int i, const ptr_region& g, int shape) {
        float d = has_shape(PTR_SHAPE_INSTANCES) && shape == PTR_SHAPE_INSTANCES ? accel_region_sdf(S, g, p) : analytic_sdf_shape(shape, g, p);
        if (d < 0.0f && (d > best || (d == best && i < region))) { best = d; region = i; }
    };
#if PTR_SPEC_NREGIONS > 0
    constexpr bool tabled = false;
#pragma unroll
    for (int k = 0; k < PTR_SPEC_NREGIONS; ++k) arm(k, S.regions[k], spec_shape(k));
#else
    const bool tabled = PTR_SPEC_BVH && S.region_bvh != nullptr;
    if (!tabled && S.region_runs) {
        for_region_runs(S, [&](auto sc, int a, int b) {
            constexpr int SH = decltype(sc)::value;
            for (int i = a; i < b; ++i) {
                if constexpr (SH == PTR_SHAPE_SPHERE) {
                    // inside only if |p - c|^2 is below the widened radius^2: the exact distance
                    // (a square root) is taken for the few that pass
                    const float4 scan = __ldg(S.region_scan + i);
                    const float x = p.x - scan.x, y = p.y - scan.y, z = p.z - scan.z;
                    if (!(__fmaf_rn(z, z, __fmaf_rn(y, y, x * x)) < scan.w)) continue;
                    const float4* g4 = reinterpret_cast<const float4*>(S.regions + i);
                    const float4 c = __ldg(g4 + 1), rr = __ldg(g4 + 2);
                    const float d = length(p - f3(c.y, c.z, c.w)) - rr.x;
                    if (d < 0.0f && (d > best || (d == best && i < region))) { best = d; region = i; }
                } else {
                    arm(i, S.regions[i], SH >= 0 ? SH : S.regions[i].shape);
                }
            }
        });
    } else {
        const int n = tabled ? S.n_linear : S.n_regions;
        for (int k = 0; k < n; ++k) {
            const int i = tabled ? S.linear_regions[k] : k;
            arm(i, S.regions[i], S.regions[i].shape);
        }
    }
#endif
    if (tabled) {
        int stack[kBvhStack];
        int ptr = 0;
        stack[0] = 0;
        while (ptr >= 0) {
            int ni = stack[ptr];
            ptr--;
            float4 n0 = __ldg(S.region_bvh + 2 * ni), n1 = __ldg(S.region_bvh + 2 * ni + 1);
            if (!(p.x >= n0.x && p.y >= n0.y && p.z >= n0.z && p.x <= n1.x && p.y <= n1.y && p.z <= n1.z)) continue;
            if (n0.w >= 0.0f) {
                for (int j = (int)n1.w; j < (int)n1.w + (int)n0.w; ++j) {
                    const int i = S.region_items[j];
                    float d = analytic_sdf(S.regions[i], p);
                    if (d < 0.0f && (d > best || (d == best && i < region))) { best = d; region = i; }
                }
            } else {
                int L = ni + 1, R = (int)n1.w;
                if (ptr + 2 < kBvhStack) { stack[++ptr] = L; stack[++ptr] = R; }
                else flag_error(S, kErrBvhStack);
            }
        }
    }
    return region;
}

// Complete the hit record: point, uncertainty, frame, and the region classification of
// scene_intersect (intersection.ts:1665-1713).
// need_from / need_to: whether the caller reads region_from / region_to; a side nobody reads is
// not classified (its point scan over every region is the costliest part) and holds -1 or the
// hit region.
__device__ __forceinline__ void fill_hit(const DevScene& S, const Ray& r, const HitRec& hr, Hit& h, bool need_from, bool need_to) {
    h.t = hr.t;
    h.p = r.o + r.d * hr.t;
    h.region_owner = hr.region;
    h.element = hr.element;
    h.alpha = -1.0f;
    const ptr_region& g = S.regions[hr.region];
    f3 n;
    bool mesh = false;
    if (kHasMesh && (g.shape == PTR_SHAPE_MESH || (g.shape == PTR_SHAPE_INSTANCES && S.batches[g.ref].proto_shape == PTR_SHAPE_MESH))) {
        // mesh hits: frame from the (normalised) shading normal, ng the triangle's plane normal
        n = accel_hit_normal(S, g, hr, r, h, h.ng);
        mesh = true;
    } else if (has_shape(PTR_SHAPE_INSTANCES) && g.shape == PTR_SHAPE_INSTANCES) {
        f3 unused;
        n = accel_hit_normal(S, g, hr, r, h, unused);
    } else {
        n = analytic_normal(g, h.p);
        h.eps = fp_uncertainty(h.p);
    }
    n = normalize(n);
    if (!mesh) h.ng = n;   // a primitive's normal is its true surface normal
    // the classification probes a caller needs: the outer side, and for a thin owner met from
    // behind its inner side too (one scan's code for both)
    const bool front = dot(r.d, h.ng) < 0.0f;
    int inside = hr.region, outside = -1;
    const int first = (front ? need_from : need_to) ? 0 : 1, last = !front && g.thin && need_from ? 2 : 1;
#pragma unroll 1
    for (int k = first; k < last; ++k) {
        const int at = scene_region_at(S, h.p + h.ng * (k == 0 ? kEpsInterface : -kEpsInterface));
        if (k == 0) outside = at; else inside = at;
    }
    h.region_from = front ? outside : inside;
    h.region_to = front ? hr.region : outside;
    if (!front) {
        n = -n;
        h.ng = -h.ng;
        n = normalize(n);
    }
    h.frame = unit_frame(n);
}

__device__ __forceinline__ int material_of(const DevScene& S, int region) {
    return region < 0 ? S.ambient_material : S.regions[region].material;
}
__device__ __forceinline__ float ior_of(const DevScene& S, int region) {
    return region < 0 ? 1.0f : S.regions[region].ior;
}
__device__ __forceinline__ bool mat_has_medium(const DevScene& S, int m) {
    return m >= 0 && (S.materials[m].flags & PTR_MATF_MEDIUM);
}
__device__ __forceinline__ bool scatter_live(const DevScene& S, const ProgParams& P, int m) {
    return P.scattering && (S.materials[m].flags & PTR_MATF_SCATTERING);
}
template <class Col>
__device__ __forceinline__ Col medium_transmittance(const DevScene& S, const ProgParams& P, int m, float len, const Wl& wl) {
    Col st = scatter_live(S, P, m) ? Colors<Col>::sigma_a(S, m, wl) + Colors<Col>::sigma_s(S, m, wl)
                                   : Colors<Col>::sigma_a(S, m, wl);
    return vexp(-st * len);
}

// wavelengths_sample (color/spectral/spectral.glsl:1-10): one number, four cyclic
// quarter-interval offsets in CDF space, each lane with its own marginal density; the
// visible density is the normalised sech^2 (visible.glsl:3-13), or uniform (uniform.glsl).
__device__ __forceinline__ float wavelength_pdf(const FrameParams& F, float lambda) {
    if (F.wavelengths == PTR_WAVELENGTHS_UNIFORM) return 1.0f / (F.lambda_max - F.lambda_min);
    float a = m_tanh(0.0072f * (F.lambda_min - 538.0f));
    float b = m_tanh(0.0072f * (F.lambda_max - 538.0f));
    float c = m_cosh(0.0072f * (lambda - 538.0f));
    return 0.0072f / ((b - a) * c * c);
}
__device__ __forceinline__ float4 wavelength_pdfs(const FrameParams& F, float4 l) {
    return make_float4(wavelength_pdf(F, l.x), wavelength_pdf(F, l.y), wavelength_pdf(F, l.z), wavelength_pdf(F, l.w));
}
__device__ __forceinline__ float4 wavelengths_sample(const FrameParams& F, float u) {
    float l[4];
    for (int k = 0; k < 4; ++k) {
        float v = u + 0.25f * (float)k;
        v = v - floorf(v);
        if (F.wavelengths == PTR_WAVELENGTHS_UNIFORM) {
            l[k] = F.lambda_min + (F.lambda_max - F.lambda_min) * v;
        } else {
            float a = m_tanh(0.0072f * (F.lambda_min - 538.0f));
            float b = m_tanh(0.0072f * (F.lambda_max - 538.0f));
            l[k] = 538.0f + m_atanh(a * (1.0f - v) + b * v) / 0.0072f;
        }
    }
    return make_float4(l[0], l[1], l[2], l[3]);
}

// color_to_pixel (spectral.glsl:27-33) with the CIE 1931 sensor (sensor/cie1931/cie1931.glsl:3-5):
// 0.25 * sum_i M xyz(lambda_i) / int(ybar) * (L_i / pdf_i).
__device__ __forceinline__ f3 color_to_pixel(const DevScene& S, float4 L, float4 lam, float4 pdf) {
    const float Ls[4] = {L.x, L.y, L.z, L.w}, ls[4] = {lam.x, lam.y, lam.z, lam.w}, ps[4] = {pdf.x, pdf.y, pdf.z, pdf.w};
    f3 pixel(0.0f);
    for (int k = 0; k < 4; ++k) {
        float4 c = spectral_curves(S.spec_curves, ls[k]);
        f3 rgb(S.spec_m[0] * c.x + S.spec_m[1] * c.y + S.spec_m[2] * c.z,
               S.spec_m[3] * c.x + S.spec_m[4] * c.y + S.spec_m[5] * c.z,
               S.spec_m[6] * c.x + S.spec_m[7] * c.y + S.spec_m[8] * c.z);
        pixel = pixel + rgb / S.spec_y * (Ls[k] / ps[k]);
    }
    return 0.25f * pixel;
}

// ---- kernels ---------------------------------------------------------------------------

// Pixel and sample of a frame's path index (samples are the outer dimension).
__device__ __forceinline__ void split_path(long long g, unsigned npix, int& pix, int& sample) {
    if ((unsigned long long)g >> 32) {
        pix = (int)(g % npix);
        sample = (int)(g / npix);
    } else {   // the 32-bit division is several times cheaper
        const unsigned k = (unsigned)g, q = k / npix;
        pix = (int)(k - q * npix);
        sample = (int)q;
    }
}
// The camera ray of one sample of pixel pix and its random stream (accumulation.ts:14-26
// cameraSample; pinhole.glsl:4-18); spectral programs also draw their wavelengths.
template <bool SPECTRAL>
__device__ __forceinline__ void camera_path(const FrameParams& F, int pix, int sample, Rng& rng, Ray& r, float4& lambda) {
    int x = (int)((unsigned)pix % (unsigned)F.width), y = (int)((unsigned)pix / (unsigned)F.width);
    rng.init((uint32_t)(x + F.px_off), (uint32_t)(y + F.py_off), (uint32_t)(F.first_sample + sample), F.salt);
    float pxf = (float)x + 0.5f + (float)F.px_off;
    float pyf = (float)y + 0.5f + (float)F.py_off;
    float a0 = rng.next();
    float a1 = rng.next();
    float fx = pxf + (a0 - 0.5f), fy = pyf + (a1 - 0.5f);
    if (SPECTRAL) lambda = wavelengths_sample(F, rng.next());   // between the film point and the camera ray
    rng.next();   // the lens draw (a pinhole has no aperture)
    rng.next();
    float ndcx = (2.0f * fx / (float)F.img_w) - 1.0f;
    float ndcy = (2.0f * fy / (float)F.img_h) - 1.0f;
    ndcx *= F.cam.aspect;
    r.d = normalize(ld3(F.cam.forward) + ndcx * F.cam.tan_fov * ld3(F.cam.right) +
                    ndcy * F.cam.tan_fov * ld3(F.cam.up));
    r.o = ld3(F.cam.position);
}
// path_state_init of path slot i.
__device__ __forceinline__ void init_slot(const PathPool& pool, long long i, const Rng& rng, const Ray& r, int medium) {
    pool.ray_o[i] = f4(r.o, 0.0f);
    pool.ray_d[i] = f4(r.d, 1.0f);
    pool.thr[i] = make_float4(1.f, 1.f, 1.f, 1.f);   // the spectral model's fourth lane included
    pool.rad[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    pool.prev_q[i] = f4(r.o, 0.0f);
    pool.st[i] = make_int4(0, medium, 0, 1);
    pool.rng[i] = make_uint2(rng.base, rng.dim);
    pool.q[0][i] = (int)i;
}

// Camera rays for one wave.
template <bool ADJ = false, bool SPECTRAL = false>
__global__ void k_generate(const __grid_constant__ DevScene S, PathPool pool, const FrameParams* fp, AdjParams adj = AdjParams{}) {
    const FrameParams F = *fp;
    long long base = pool.wave[0];
    long long n = F.total - base;
    if (n > F.capacity) n = F.capacity;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        pool.cnt[0] = (unsigned)n;
        pool.wave[1] = n;
        pool.stats[2] += (unsigned long long)n;
        if (pool.fetch) pool.fetch[0] = 0u;
    }
    const unsigned npix = (unsigned)F.width * (unsigned)F.height;
    // every path starts at the pinhole: its region is found once per thread
    const int medium = S.has_media ? scene_region_at(S, ld3(F.cam.position)) : -1;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        int pix, sample;
        split_path(base + i, npix, pix, sample);
        Rng rng;
        Ray r;
        float4 lambda;
        camera_path<SPECTRAL>(F, pix, sample, rng, r, lambda);
        if (SPECTRAL) {
            pool.wl[i] = lambda;
            pool.wl_pdf[i] = wavelength_pdfs(F, lambda);
        }
        if (ADJ) {   // replay: the forward pass left this path's total radiance in rad
            pool.l_rem[i] = pool.rad[i];
            const float* g = adj.dl_image + 3 * (size_t)pix;
            pool.dl[i] = make_float4(g[0] * adj.inv_spp, g[1] * adj.inv_spp, g[2] * adj.inv_spp, 0.f);
        }
        init_slot(pool, i, rng, r, medium);
        if (pool.aov) { pool.aov[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f); pool.aov[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f); }
    }
}

#ifndef PTR_TRACE_MIN_BLOCKS
#define PTR_TRACE_MIN_BLOCKS 4
#endif

// Fold a thread's tally into S.work (one atomic per warp and counter).
__device__ __forceinline__ void flush_work(const DevScene& S, const Work& w) {
    unsigned v[4] = {w.nodes, w.tris, w.tlas, w.inst};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        unsigned x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(&S.work[k], (unsigned long long)x);
    }
}

constexpr int kMaxSortBuckets = 32;
// Shading class of a live path: 0 miss, 1 + the material model of the surface it hit; with
// more than 8 buckets, + 8 when its segment starts inside a medium (the medium arm runs first).
__device__ __forceinline__ unsigned shade_key(const DevScene& S, int region, int cur_med, int buckets) {
    unsigned k = 0u;
    if (region >= 0) {
        const int m = S.regions[region].material;
        k = 1u + (unsigned)(m >= 0 ? S.materials[m].model : 0);
    }
    if (buckets > 8) {
        const int mm = cur_med < 0 ? S.ambient_material : S.regions[cur_med].material;
        if (mm >= 0 && (S.materials[mm].flags & PTR_MATF_MEDIUM)) k += 8u;
    }
    return k < (unsigned)buckets ? k : (unsigned)buckets - 1u;
}

// Nearest hit of every live path (and, for the sorted queue, its shading key).
// Closest hits of a queue whose scene is analytic regions plus one instanced mesh batch
// walked by the flat two-level loop: a lane whose query ends takes the next ray at once
// (warp-aggregated tickets whenever at least kRefillMin lanes are idle) instead of idling
// until the warp's slowest ray is done.  The regions before and after the instanced one
// are tested in region order around the walk, as in scene_closest, so hits are identical.
// (PTR_REFILL=0 builds keep the per-warp queue cursor everywhere.)
#ifndef PTR_REFILL
#define PTR_REFILL 1
#endif
#ifndef PTR_REFILL_MIN
#define PTR_REFILL_MIN 8
#endif
constexpr int kRefillMin = PTR_REFILL_MIN;
template <bool COUNT, bool WIDE>
__device__ __forceinline__ void closest_refill(const DevScene& S, const PathPool& pool, const int* q, unsigned n, int buckets,
                                               unsigned* ticket, Work* w) {
    const int fr = S.flat_region;
    const FlatScene fs = flat_scene<WIDE>(S, S.batches[S.regions[fr].ref]);
    const unsigned lane = threadIdx.x & 31u;
    FlatWalk<WIDE> f;
    Ray r;
    HitRec h;
    int i = -1, steps = 0;
    bool active = false, exhausted = false;
    for (;;) {
        if (!exhausted) {
            const unsigned need = __ballot_sync(0xffffffffu, !active);
            if (__popc(need) >= kRefillMin) {
                const int leader = __ffs(need) - 1;
                unsigned base = 0u;
                if ((int)lane == leader) base = atomicAdd(ticket, (unsigned)__popc(need));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (base + (unsigned)__popc(need) >= n) exhausted = true;
                if (!active) {
                    const unsigned k = base + __popc(need & lanemask_lt());
                    if (k < n) {
                        i = q[k];
                        r.o = xyz(pool.ray_o[i]);
                        r.d = xyz(pool.ray_d[i]);
                        h.t = kMaxDist;
                        h.u = h.v = 0.f;
                        h.region = -1;
                        h.element = 0;
                        h.prim = -1;
                        for (int g = 0; g < fr; ++g) {
                            float t;
                            if (analytic_root(S.regions[g], r, t) && t < h.t) { h.t = t; h.region = g; h.element = 0; h.prim = -1; }
                        }
                        f.init(fs, r, h.t, COUNT ? w : nullptr);
                        steps = 0;
                        active = true;
                    }
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) break;
        if (!active) continue;
        bool more = f.template step<false>(S, fs, fr, r, h, 0.0f, COUNT ? w : nullptr);
        if (more && ++steps >= kFlatGuard) {
            flag_error(S, kErrCwGuard);
            more = false;
        }
        if (!more) {
            for (int g = fr + 1; g < S.n_regions; ++g) {
                float t;
                if (analytic_root(S.regions[g], r, t) && t < h.t) { h.t = t; h.region = g; h.element = 0; h.prim = -1; }
            }
            const float4 hf = make_float4(h.t, h.u, h.v, 0.f);
            const int4 hi = make_int4(h.region, h.element, h.prim, 0);
            pool.hit[i] = hf;
            pool.hit_i[i] = hi;
            if (float4* log = pool.hit_log_mode == 1 ? hit_log_slice(pool) : nullptr) {
                log[4 * (size_t)i] = hf;
                log[4 * (size_t)i + 1] = int4_as_float4(hi);
            }
            if (buckets > 1) pool.sort_key[i] = (unsigned char)shade_key(S, h.region, pool.st[i].y, buckets);
            active = false;
        }
    }
}

template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256, PTR_TRACE_MIN_BLOCKS) k_closest(const __grid_constant__ DevScene S0, PathPool pool, int in, BatchTables bt) {
    const int buckets = pool.sort_buckets;
    unsigned n = pool.cnt[in];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        pool.cnt[in ^ 1] = 0u;
        pool.cnt[2] = 0u;
        pool.cnt[4] = 0u;
        pool.stats[0] += n;
        if (pool.fetch) { pool.fetch[1] = 0u; pool.fetch[2] = 0u; pool.fetch[3] = 0u; }
    }
    const int* q = closest_queue(pool, in);
    Work w{0u, 0u, 0u, 0u};
    float4* log = BATCH ? nullptr : hit_log_slice(pool);
    // (a logged iteration of the replay walks nothing: it reads the log in the loop below)
    if (PTR_REFILL && kHasMesh && !BATCH && pool.fetch && S0.flat_region >= 0 && !(log && pool.hit_log_mode == 2)) {
        const DevBatch& b = S0.batches[S0.regions[S0.flat_region].ref];
        const bool wide = flat_wide_ok(S0, b), binary = flat_binary_ok(S0, b);
        if (wide) closest_refill<COUNT, true>(S0, pool, q, n, buckets, pool.fetch + 0, &w);
        else if (binary) closest_refill<COUNT, false>(S0, pool, q, n, buckets, pool.fetch + 0, &w);
        if (wide || binary) {
            if (COUNT) flush_work(S0, w);
            return;
        }
    }
    const WaveJobs wj = BATCH ? WaveJobs(pool, bt) : WaveJobs{};
    QueueCursor cur(n, pool.fetch ? pool.fetch + 0 : nullptr);
    unsigned k;
    while (cur.next(k)) {
        if (k >= n) continue;
        int i = q[k];
        const DevScene& S = BATCH ? bt.scenes[wj.of(bt, i)] : S0;
        float4 hf;
        int4 hi;
        if (log && pool.hit_log_mode == 2) {   // the replay: the forward walk's hit of this path
            hf = log[4 * (size_t)i];
            hi = float4_as_int4(log[4 * (size_t)i + 1]);
        } else {
            Ray r;
            r.o = xyz(pool.ray_o[i]);
            r.d = xyz(pool.ray_d[i]);
            HitRec h = scene_closest<false>(S, r, COUNT ? &w : nullptr);
            hf = make_float4(h.t, h.u, h.v, 0.f);
            hi = make_int4(h.region, h.element, h.prim, 0);
            if (log && pool.hit_log_mode == 1) {
                log[4 * (size_t)i] = hf;
                log[4 * (size_t)i + 1] = int4_as_float4(hi);
            }
        }
        pool.hit[i] = hf;
        pool.hit_i[i] = hi;
        if (buckets > 1) pool.sort_key[i] = (unsigned char)shade_key(S, hi.x, pool.st[i].y, buckets);
    }
    if (COUNT) flush_work(S0, w);
}

// Counting sort of a device-counted queue by 1-byte keys (< kMaxKeys), in three launches
// on fixed grids: per-chunk key counts, one scan into per-(key, chunk) offsets, and a
// scatter that reserves slots from shared-memory offsets.  Each of kSortChunks blocks owns
// one contiguous chunk of the queue (a multiple of kSortVec entries), so global traffic is
// the keys twice, the source once and the destination once, and no global atomics are
// taken.  Each thread reads kSortVec consecutive keys with one 16-byte load (and their
// sources with four), and lanes with equal keys find each other with seven ballots (a
// warp multi-split).  The consumers are order-independent; the order within a key only
// matters for their memory coalescing.
// GATHER: the keys are indexed by path (keys[src[k]]) rather than by queue position.
// Queues shorter than kSortMin are not sorted: every consumer reads the unsorted queue
// then (sorted_queue), deciding from the same device count as the sort kernels.
constexpr int kSortChunks = 512;
constexpr int kMaxKeys = 64;
constexpr int kSortThreads = 256;
constexpr int kSortVec = 16;
constexpr int kSortScanThreads = 1024;
constexpr int kSortEntries = kMaxKeys * kSortChunks;
constexpr int kSortScanPer = kSortEntries / kSortScanThreads;   // 32: one padded smem row per thread
static_assert(kSortScanPer == 32, "the scan's padded layout assumes 32 entries per thread");
constexpr size_t kSortScanSmem = (size_t)(kSortEntries + kSortEntries / 32) * sizeof(unsigned);
constexpr unsigned kSortMin = 65536u;
constexpr unsigned kNoKey = (unsigned)kMaxKeys;   // 7-bit key of an idle lane
__device__ __forceinline__ const int* sorted_queue(const int* sorted, const int* plain, unsigned n) {
    return n >= kSortMin ? sorted : plain;
}
__device__ __forceinline__ void sort_chunk(unsigned n, unsigned& lo, unsigned& hi) {
    unsigned chunk = (n + kSortChunks - 1) / kSortChunks;
    chunk = (chunk + kSortVec - 1) & ~(unsigned)(kSortVec - 1);
    lo = min(n, blockIdx.x * chunk);
    hi = min(n, lo + chunk);
}
// Lanes of the warp whose 7-bit key equals this lane's (all lanes take part).
__device__ __forceinline__ unsigned warp_peers(unsigned key) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 7; ++b) {
        const unsigned m = __ballot_sync(0xffffffffu, (key >> b) & 1u);
        peers &= ((key >> b) & 1u) ? m : ~m;
    }
    return peers;
}
// Keys (and, if asked or gathering, sources) of entries [base, base + kSortVec) below hi;
// base is a multiple of kSortVec, so the full-width loads are 16-byte aligned.
template <bool GATHER>
__device__ __forceinline__ void sort_load(const int* src, const unsigned char* keys, unsigned base, unsigned hi,
                                          unsigned (&key)[kSortVec], int (&val)[kSortVec], bool want_val) {
    if (base + kSortVec <= hi) {
        if (GATHER || want_val) {
#pragma unroll
            for (int v = 0; v < kSortVec / 4; ++v) {
                const int4 x = *reinterpret_cast<const int4*>(src + base + 4 * v);
                val[4 * v] = x.x; val[4 * v + 1] = x.y; val[4 * v + 2] = x.z; val[4 * v + 3] = x.w;
            }
        }
        if (GATHER) {
#pragma unroll
            for (int j = 0; j < kSortVec; ++j) key[j] = keys[(unsigned)val[j]];
        } else {
            const uint4 x = *reinterpret_cast<const uint4*>(keys + base);
            const unsigned w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < kSortVec; ++j) key[j] = (w[j >> 2] >> (8 * (j & 3))) & 0xffu;
        }
    } else {
#pragma unroll
        for (int j = 0; j < kSortVec; ++j) {
            const unsigned k = base + j;
            const bool v = k < hi;
            val[j] = (v && (GATHER || want_val)) ? src[k] : 0;
            key[j] = v ? (unsigned)keys[GATHER ? (unsigned)val[j] : k] : kNoKey;
        }
    }
}
// Counts of every key (all kMaxKeys rows are written, unused ones zero).
template <bool GATHER>
__global__ void __launch_bounds__(kSortThreads) k_sort_hist(const int* src, const unsigned char* keys, const unsigned* count, unsigned* hist) {
    const unsigned n = *count;
    if (n < kSortMin) return;
    __shared__ unsigned h[kMaxKeys];
    if (threadIdx.x < kMaxKeys) h[threadIdx.x] = 0u;
    __syncthreads();
    unsigned lo, hi;
    sort_chunk(n, lo, hi);
    for (unsigned k0 = lo; k0 < hi; k0 += kSortThreads * kSortVec) {   // block-uniform trip count
        unsigned key[kSortVec];
        int val[kSortVec];
        sort_load<GATHER>(src, keys, k0 + threadIdx.x * kSortVec, hi, key, val, false);
#pragma unroll
        for (int j = 0; j < kSortVec; ++j) {
            const unsigned peers = warp_peers(key[j]);
            if (key[j] != kNoKey && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[key[j]], (unsigned)__popc(peers));
        }
    }
    __syncthreads();
    if (threadIdx.x < kMaxKeys) hist[threadIdx.x * kSortChunks + blockIdx.x] = h[threadIdx.x];
}
// Exclusive scan, in place, of the key-major [kMaxKeys][kSortChunks] counts: one block
// stages them in shared memory with coalesced loads (one padding word per 32 entries, so
// the per-thread rows below are bank-conflict free), scans, and writes them back.
__global__ void __launch_bounds__(kSortScanThreads) k_sort_scan(const unsigned* count, unsigned* hist) {
    if (*count < kSortMin) return;
    extern __shared__ unsigned sm[];
    __shared__ unsigned warp_sum[kSortScanThreads / 32];
    for (int e = threadIdx.x; e < kSortEntries; e += kSortScanThreads) sm[e + (e >> 5)] = hist[e];
    __syncthreads();
    const int row = threadIdx.x * (kSortScanPer + 1);   // entries [32 t, 32 t + 32) of the padded layout
    unsigned s = 0u;
#pragma unroll
    for (int j = 0; j < kSortScanPer; ++j) s += sm[row + j];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = s;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned w = warp_sum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sum[lane] = w;
    }
    __syncthreads();
    unsigned run = incl - s + (warp ? warp_sum[warp - 1] : 0u);
#pragma unroll
    for (int j = 0; j < kSortScanPer; ++j) {
        const unsigned c = sm[row + j];
        sm[row + j] = run;
        run += c;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kSortEntries; e += kSortScanThreads) hist[e] = sm[e + (e >> 5)];
}
// The scatter stages each warp's 32 * kSortVec entries in shared memory (16-byte loads),
// then places them in rounds of 32 consecutive entries: peers of one round land in one
// contiguous run, so a sorted queue keeps the compaction's ascending path order within
// its runs (the pool's SoA reads of its consumers stay coalesced).
template <bool GATHER>
__global__ void __launch_bounds__(kSortThreads) k_sort_scatter(const int* src, const unsigned char* keys, const unsigned* count,
                                                               const unsigned* offsets, int* dst) {
    const unsigned n = *count;
    if (n < kSortMin) return;
    constexpr int kSpan = 32 * kSortVec;   // entries one warp stages per round
    __shared__ unsigned base[kMaxKeys];
    __shared__ __align__(16) int s_val[kSortThreads / 32][kSpan];
    __shared__ __align__(16) unsigned char s_key[kSortThreads / 32][kSpan];
    if (threadIdx.x < kMaxKeys) base[threadIdx.x] = offsets[threadIdx.x * kSortChunks + blockIdx.x];
    __syncthreads();
    unsigned lo, hi;
    sort_chunk(n, lo, hi);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* sv = s_val[warp];
    unsigned char* sk = s_key[warp];
    for (unsigned k0 = lo; k0 < hi; k0 += kSortThreads * kSortVec) {   // block-uniform trip count
        const unsigned ws = k0 + warp * kSpan;
        const unsigned b = ws + lane * kSortVec;
        if (b + kSortVec <= hi) {
#pragma unroll
            for (int v = 0; v < kSortVec / 4; ++v)
                *reinterpret_cast<int4*>(sv + lane * kSortVec + 4 * v) = *reinterpret_cast<const int4*>(src + b + 4 * v);
            if (!GATHER) *reinterpret_cast<uint4*>(sk + lane * kSortVec) = *reinterpret_cast<const uint4*>(keys + b);
        } else {
            for (int j = 0; j < kSortVec; ++j) {
                if (b + j < hi) {
                    sv[lane * kSortVec + j] = src[b + j];
                    if (!GATHER) sk[lane * kSortVec + j] = keys[b + j];
                }
            }
        }
        __syncwarp();
#pragma unroll 4
        for (int j = 0; j < kSortVec; ++j) {
            const int e = j * 32 + lane;
            const bool valid = ws + e < hi;
            const int val = valid ? sv[e] : 0;
            const unsigned key = valid ? (unsigned)(GATHER ? keys[(unsigned)val] : sk[e]) : kNoKey;
            const unsigned peers = warp_peers(key);
            const int leader = __ffs(peers) - 1;
            unsigned o = 0u;
            if (valid && lane == leader) o = atomicAdd(&base[key], (unsigned)__popc(peers));
            o = __shfl_sync(0xffffffffu, o, leader);
            if (valid) dst[o + __popc(peers & lanemask_lt())] = val;
        }
        __syncwarp();
    }
}

__device__ __forceinline__ const int* closest_queue(const PathPool& pool, int in) {
    return pool.ray_in ? sorted_queue(pool.q_ray, pool.q[in], pool.cnt[in]) : pool.q[in];
}

// What one walk iteration carries of a path: k_shade loads it from the pool and stores it
// back, k_walk keeps it in registers for the whole walk.
template <class Col>
struct WalkState {
    Ray r;
    float prev_bsdf_pdf, eta_scale;
    Col thr, rad;
    f3 prev_qp;              // the stored light-query point
    Wl wl;                   // spectral only
    int bounce, cur_med, nulls;
    bool prev_delta;
    Rng rng;
    Col lrem;                // adjoint replay only: the radiance still to come
};

// One walk iteration of a path whose segment's closest hit is hr: the medium segment, null
// pass-through, emitter scoring, NEE sampling (its queries go to the sink), the
// continuation lobe and roulette.  Returns true while the path goes on.
// Sink: segment_query / vertex_query take the iteration's shadow queries (slots 1 and 0),
// seed() the sampler dimension of a heterogeneous medium's query, put_prev_n / get_prev_n
// the stored query normal of light-tree programs, aov() the path's two first-hit samples
// (null when the program has none).
// ADJ: also scatters the gradient terms through ga and leaves the slot-0 query's vertex
// material and lobe derivative in sh_mat / sg.
// live: this lane has a path; phase() is called by every lane between the parts of the iteration.
// tracked: the outcome of the segment's delta tracking where the caller ran it (TRACKED; the
// site's two numbers are drawn then).
template <class Col, int DIRECT, bool MEDIA, bool ADJ, bool TRACKED = false, class Sink, class Phase>
__device__ __forceinline__ bool walk_iteration(const DevScene& S, const ProgParams& P, WalkState<Col>& ws, const HitRec& hr,
                                               Sink& sink, const GradAcc& ga, int& sh_mat, NeeGrad& sg, bool live, Phase phase,
                                               const MediumSample<f3>* tracked = nullptr) {
    constexpr bool SPECTRAL = sizeof(Col) == sizeof(s4);
    using CM = Colors<Col>;
    const bool nee = DIRECT != PTR_DIRECT_NONE;
    const bool mis = DIRECT == PTR_DIRECT_MIS;
    const bool tree = PTR_SPEC_TREE && P.light_tree;
    Ray& r = ws.r;
    float& prev_bsdf_pdf = ws.prev_bsdf_pdf;
    float& eta_scale = ws.eta_scale;
    Col& thr = ws.thr;
    Col& rad = ws.rad;
    f3& prev_qp = ws.prev_qp;
    const Wl& wl = ws.wl;
    int &bounce = ws.bounce, &cur_med = ws.cur_med, &nulls = ws.nulls;
    bool& prev_delta = ws.prev_delta;
    Rng& rng = ws.rng;
    Col& lrem = ws.lrem;
    bool alive = false, shadow = false;
    const bool boundary = hr.region >= 0;
    const int N = P.max_bounces;

    // -- the volumetric call site: one segment (features/materials.ts:675-746).  event: the
    // segment scattered at p_evt in the medium of material mat
    bool event = false, het = false;
    int mat = 0;
    f3 p_evt;
    // The medium's coefficients. In the spectral model each is four evaluations of a lifted
    // spectrum, so the segment makes them once and its users share them (a 1024 x 1024 frame at
    // 16 spp in spectral fogs: k_shade 14.1 -> 13.2 ms, the frame 20.7 -> 19.8); in RGB each is
    // one load, made where it is used.
    Col lane_a(0.0f), lane_s(0.0f);
    auto sigma_a = [&](int m) { return SPECTRAL ? lane_a : CM::sigma_a(S, m, wl); };
    auto sigma_s = [&](int m) { return SPECTRAL ? lane_s : CM::sigma_s(S, m, wl); };
    if (MEDIA && live) {
        const int med_mat = material_of(S, cur_med);
        if (mat_has_medium(S, med_mat)) {
            const ptr_material& mm = S.materials[med_mat];
            if constexpr (SPECTRAL) {
                lane_a = CM::sigma_a(S, med_mat, wl);
                lane_s = CM::sigma_s(S, med_mat, wl);
            }
            // the per-segment equiangular site precedes the transmittance sample
            // (pt.ts:322-328) and rides the second shadow slot
            if (P.equiangular && bounce < N) {
                EquiangularQuery<Col> eq;
                if (equiangular_site<Col>(S, med_mat, sigma_a, sigma_s, r, boundary ? hr.t : kMaxDist, rng, thr, wl, eq))
                    sink.segment_query(eq.p_evt, eq.wi, P.max_null - nulls, eq.light_pos, eq.contrib, eq.denom);
            }
            // heterogeneous media take the tracking arms (delta_tracking.glsl)
            het = !SPECTRAL && PTR_SPEC_HET && S.has_het && mat_is_het(mm);
            float x0 = 0.0f, x1 = 0.0f;
            if (!(TRACKED && het && scatter_live(S, P, med_mat))) {
                x0 = rng.next();
                x1 = rng.next();
            }
            float t_max = boundary ? hr.t : kMaxDist;
            if (!scatter_live(S, P, med_mat) && !het) {
                thr = thr * vexp(-sigma_a(med_mat) * t_max);
                if constexpr (ADJ) {   // w = exp(-(1-a) st t)
                    GreyMedium gm = grey_medium(mm);
                    ga.scl(med_mat, PTR_GRAD_SIGMA_T, lrem, -(1.0f - gm.a) * t_max);
                    ga.scl(med_mat, PTR_GRAD_MEDIUM_ALBEDO, lrem, gm.st * t_max);
                }
            } else {
                MediumSample<Col> ms;
                bool done = false;
                if constexpr (!SPECTRAL && PTR_SPEC_HET) {
                    if (het && scatter_live(S, P, med_mat)) {
                        if constexpr (TRACKED) {
                            ms = *tracked;
                        } else {
                            DeltaTrack track;
                            track.begin(mm, t_max, x0, x1);
                            track.advance(S, mm, r, t_max, rng, track.left);
                            ms = track.ms;
                        }
                        done = true;
                    } else if (het) {   // absorbing only: the ratio-tracked pass-through
                        ms.scattered = false;
                        ms.weight = medium_ratio_track(S, mm, r, t_max, rng, false);
                        done = true;
                    }
                }
                if (!done)
                    ms = medium_sample_analytic<Col>(sigma_a(med_mat), sigma_s(med_mat), r, t_max, x0, x1);
                thr = thr * ms.weight;
                if constexpr (ADJ) {   // scattered at t: w = a st exp(-st t)/pdf; passed: exp(-st t_max)/P
                    GreyMedium gm = grey_medium(mm);
                    if (ms.scattered) {
                        float t_evt = dot(ms.exit_p - r.o, r.d);
                        ga.scl(med_mat, PTR_GRAD_SIGMA_T, lrem, 1.0f / gm.st - t_evt);
                        ga.scl(med_mat, PTR_GRAD_MEDIUM_ALBEDO, lrem, 1.0f / gm.a);
                    } else {
                        ga.scl(med_mat, PTR_GRAD_SIGMA_T, lrem, -t_max);
                    }
                }
                event = ms.scattered;
                p_evt = ms.exit_p;
                mat = med_mat;
            }
        }
    }

    // -- the segment's end: a miss, a null interface, or a surface vertex.  vertex: the walk
    // scatters here (medium event or surface) and the bounce budget allows it
    bool vertex = event && bounce != N;
    Hit hit;
    if (MEDIA) phase();
    if (!live) {
    } else if (!event && !boundary) {   // kernel_score_miss (kernel.glsl:11-14)
        float w = 1.0f;
        if (nee && S.env_samplable && !prev_delta) {
            if (!mis) w = 0.0f;
            else {
                float pe = S.env_select_live ? S.env_select_prob : 1.0f;
                w = power_heuristic(prev_bsdf_pdf, pe * env_pdf(S, r.d));
            }
        }
        Col e = thr * w * env_radiance<Col>(S, r.d, wl);
        rad = rad + e;
        if constexpr (ADJ) lrem = lrem - e;
    } else if (!event) {
        mat = material_of(S, hr.region);
        // the incident side: the current medium, or the IOR of a model that refracts
        fill_hit(S, r, hr, hit, MEDIA || material_in<MatUsesIor>(S.materials[mat].model), true);
        if (MEDIA && hit.region_from != cur_med) cur_med = hit.region_from;
        const ptr_material& m = S.materials[mat];
        if (MEDIA && m.model == PTR_MAT_NONE) {   // null pass-through (pt.ts:404-417)
            cur_med = hit.region_to;
            r = ray_spawn(hit, r.d);
            nulls += 1;
            alive = nulls <= P.max_null;
        } else {
            const f3 wo = -r.d;
            // the AOV capture (pt.ts:422-433): the first non-null surface before
            // any event, weighted by the arrival throughput
            if constexpr (!SPECTRAL) {
                if (bounce == 0 && sink.aov()) {
                    f3 fact = ld3(m.transmittance);
                    auto aov = [&](auto M) { fact = decltype(M)::aov(m); };
                    dispatch_material<MatPresent>(m.model, aov);
                    fact = vmin(vmax(fact, f3(0.0f)), f3(1.0f));
                    f3 nf = dot(hit.frame.n, wo) < 0.0f ? -hit.frame.n : hit.frame.n;
                    sink.aov()[0] = f4(fact * thr, 0.0f);
                    sink.aov()[1] = f4(nf * spectrum_average(thr), 0.0f);
                }
            }
            // kernel_score_emitter_hit (kernel.glsl:16-25; combiner.ts:27-46)
            int mat_emit = material_of(S, hit.region_to);
            if (mat_emit >= 0 && (S.materials[mat_emit].flags & PTR_MATF_EMISSIVE)) {
                float w = 1.0f;
                if (nee) {
                    int lid = hit.region_to >= 0 ? emitter_light(S, hit) : -1;
                    if (lid >= 0 && !prev_delta) {
                        if (!mis) w = 0.0f;
                        else {
                            // the stored selection context (its normal and sidedness
                            // only under light-tree selection)
                            LightQuery pq{prev_qp, f3(0.0f), false};
                            if (tree) {
                                float4 pqn = sink.get_prev_n();
                                pq.n = xyz(pqn);
                                pq.two_sided = pqn.w != 0.0f;
                            }
                            w = power_heuristic(prev_bsdf_pdf, lighting_pdf(S, pq, r.d, lid, hit.p, hit.ng, tree));
                        }
                    }
                }
                Col e = thr * w * CM::emission(S, mat_emit, wl);
                rad = rad + e;
                if constexpr (ADJ) lrem = lrem - e;
            }
            vertex = bounce != N;
        }
    }
    phase();

    // -- the vertex: next-event estimation, then the continuation.  Medium events and
    // surfaces meet one light-sampling site (one copy of its code, their lanes together).
    const ptr_material& m = S.materials[mat];
    const f3 wo = -r.d;
    const float alpha = !event && hit.alpha >= 0.0f ? hit.alpha : m.alpha;
    // light queries with sphere support (a transmissive non-delta lobe)
    const bool rough = vertex && !event && material_in<MatSphereQuery>(m.model);
    const bool surface = vertex && !event;
    const float n_from = surface ? ior_of(S, hit.region_from) : 1.0f, n_to = surface ? ior_of(S, hit.region_to) : 1.0f;
    const MatSite<Col> site{S, mat, m, hit, wl, alpha, n_from, n_to};
    const f3 vp = event ? p_evt : hit.p;
    if (vertex && nee && (event ? !P.equiangular : material_in<MatNonDelta>(m.model))) {
        // light_sample_direct (light.glsl:8-28), light_sample_direct_medium (light_medium.glsl:7-18)
        float y0 = rng.next();
        float y1 = rng.next();
        // no orientation at a medium event; rough glass: sphere support
        LightQuery lq{vp, event ? f3(0.0f) : hit.frame.n, rough};
        LightSample<Col> ls = lighting_sample<Col>(S, lq, y0, y1, rng, tree, wl);
        if (MEDIA && PTR_SPEC_HET && S.has_het) sink.seed(rng.dim);
        if (ls.pdf > 0.0f) {
            const f3 light_p = vp + ls.wi * ls.distance;
            const bool want_pdf = mis && !(ls.flags & kLightDelta);
            Ray sr{vp, ls.wi};
            float maxd = 0.0f, bp = 0.0f;
            Col contrib;
            if (event) {
                const float ph = hg_eval(ls.wi, wo, m.phase_g);
                contrib = thr * ls.radiance * Col(ph);
                if (want_pdf) bp = spectrum_average(Col(ph));
                if constexpr (ADJ) {
                    sg.kind = kGradKindPhase;
                    sg.dnee = f3(hg_dlog_g(ls.wi, wo, m.phase_g), 0.0f, 0.0f);
                }
            } else {
                sr = ray_spawn(hit, ls.wi);
                sr.d = normalize(light_p - sr.o);
                Col f(0.0f);
                auto lobe = [&](auto M) {
                    f = decltype(M)::eval(site, ls.wi, wo);
                    if (want_pdf) bp = decltype(M)::pdf(site, ls.wi, wo);
                };
                dispatch_material<MatNonDelta, true>(m.model, lobe);   // the model has a non-delta lobe here
                const float cos_i = fabsf(dot(ls.wi, hit.frame.n));
                maxd = length(light_p - sr.o) - kShadowBackoff;
                contrib = thr * ls.radiance * f * cos_i;
                if constexpr (ADJ) {
                    auto ng = [&](auto M) { decltype(M)::nee_grad(site, ls.wi, wo, sg); };
                    dispatch_material<MatNonDelta, true>(m.model, ng);
                }
            }
            sh_mat = mat;
            const float w = want_pdf ? power_heuristic(ls.pdf, bp) : 1.0f;
            sink.vertex_query(sr.o, maxd, sr.d, P.max_null - nulls, light_p, w, contrib, ls.pdf);
            shadow = true;
        }
    }
    phase();
    if (!vertex) return alive;
    bool survive = true;
    if (event) {
        float z0 = rng.next();
        float z1 = rng.next();
        ISample<Col> ps = hg_sample<Col>(wo, m.phase_g, z0, z1);
        thr = thr * ps.weight;
        if constexpr (ADJ) {   // phase continuation: w = p_HG / pdf_detached
            float dg = hg_dlog_g(ps.wi, wo, m.phase_g);
            ga.scl(mat, PTR_GRAD_HG_G, lrem, dg);
            if (shadow) sg.dnee.x -= dg;
        }
        prev_delta = false;
        prev_bsdf_pdf = ps.pdf;
        prev_qp = p_evt;
        if (tree) sink.put_prev_n(make_float4(0.f, 0.f, 0.f, 0.f));   // no orientation
        r.o = p_evt;
        r.d = ps.wi;
        // roulette_interior (pt.ts:230-283); nothing is owed after a
        // tracking arm, whose lottery settled absorption already
        if (P.rr_start >= 0 && bounce >= P.rr_start && !het) {
            Col ss = sigma_s(mat), sa = sigma_a(mat);
            Col surv = ss / vmax(ss + sa, Col(1e-9f));
            float p_survive = spectrum_max(surv);
            if (p_survive <= 0.0f) survive = false;
            else if (rng.next() > p_survive) survive = false;
            else thr = thr / p_survive;
        }
    } else {
        // kernel_sample_continuation (kernel.glsl:27-34)
        float uc = rng.next();
        float u0 = rng.next();
        float u1 = rng.next();
        ISample<Col> bs;
        bs.weight = Col(0.0f);   // stays black only in a build without the scene's models
        auto cont = [&](auto M) { bs = decltype(M)::sample(site, wo, uc, u0, u1); };
        dispatch_material<MatPresent>(m.model, cont);
        if (spectrum_is_black(bs.weight)) return false;
        thr = thr * bs.weight;
        if constexpr (ADJ) {   // the continuation lobe: d log w_cont
            auto cg = [&](auto M) { decltype(M)::cont_grad(site, bs, wo, ga, lrem, shadow, sg); };
            dispatch_material<MatPresent>(m.model, cg);
        }
        prev_delta = (bs.flags & kLobeDelta) != 0u;
        prev_bsdf_pdf = bs.pdf;
        prev_qp = hit.p;
        if (tree) sink.put_prev_n(f4(hit.frame.n, rough ? 1.0f : 0.0f));
        if (bs.flags & kLobeTransmission) {
            if (MEDIA) cur_med = hit.region_to;
            float rr = n_to / n_from;
            eta_scale *= rr * rr;
        }
        // roulette (pt.ts:204-222)
        if (P.rr_start >= 0 && bounce >= P.rr_start) {
            float p_survive = gmin(P.rr_max_survival, spectrum_max(thr) * eta_scale);
            if (p_survive <= 0.0f) survive = false;
            else if (rng.next() > p_survive) survive = false;
            else thr = thr / p_survive;
        }
        if (survive) r = ray_spawn(hit, bs.wi);
    }
    if (survive) bounce += 1;
    return survive;
}

// k_shade's sink: queries and stored normals go to the path's pool records at once.
template <class Col>
struct PoolSink {
    const PathPool& pool;
    const int i;
    bool shadow = false, shadow2 = false;
    __device__ __forceinline__ PoolSink(const PathPool& p, int slot) : pool(p), i(slot) {}
    __device__ __forceinline__ void segment_query(f3 o, f3 d, int crossings, f3 light_p, Col contrib, float pdf) {
        pool.sh2_o[i] = f4(o, 0.0f);
        pool.sh2_d[i] = f4(d, __int_as_float(crossings));
        pool.sh2_lp[i] = f4(light_p, 1.0f);
        pool.sh2_c[i] = col_st(contrib, pdf);
        if constexpr (sizeof(Col) == sizeof(s4)) pool.sh2_pdf[i] = pdf;
        shadow2 = true;
    }
    __device__ __forceinline__ void vertex_query(f3 o, float max_dist, f3 d, int crossings, f3 light_p, float w, Col contrib, float pdf) {
        pool.sh_o[i] = f4(o, max_dist);
        pool.sh_d[i] = f4(d, __int_as_float(crossings));
        pool.sh_lp[i] = f4(light_p, w);
        pool.sh_c[i] = col_st(contrib, pdf);
        if constexpr (sizeof(Col) == sizeof(s4)) pool.sh_pdf[i] = pdf;
        shadow = true;
    }
    __device__ __forceinline__ void seed(unsigned dim) { pool.sh_seed[i] = dim; }
    __device__ __forceinline__ void put_prev_n(float4 n) { pool.prev_n[i] = n; }
    __device__ __forceinline__ float4 get_prev_n() const { return pool.prev_n[i]; }
    __device__ __forceinline__ float4* aov() const { return pool.aov ? pool.aov + 2 * i : nullptr; }
};

// One walk iteration for every live path.
#ifndef PTR_SHADE_MIN_BLOCKS
#define PTR_SHADE_MIN_BLOCKS 3
#endif
// ADJ: the replay pass of the adjoint — the same walk on the same random numbers, which
// also scatters d Loss / d theta into per-block float64 accumulators (dynamic shared
// memory: PTR_GRAD_SLOTS doubles per material).
// Col: f3 (RGB) or s4 (spectral, four wavelength lanes; the adjoint is RGB only).
template <class Col, int DIRECT, bool MEDIA, bool BATCH, bool ADJ = false>
__global__ void __launch_bounds__(256, PTR_SHADE_MIN_BLOCKS) k_shade(const __grid_constant__ DevScene S0, PathPool pool, ProgParams P0, int in, BatchTables bt,
                                                                     AdjParams adj = AdjParams{}) {
    constexpr bool SPECTRAL = sizeof(Col) == sizeof(s4);
    static_assert(!(ADJ && SPECTRAL), "the adjoint replay is RGB only");
    extern __shared__ double s_grad[];
    if constexpr (ADJ) grad_block_init(s_grad, PTR_GRAD_SLOTS * S0.n_materials);
    const unsigned n = pool.cnt[in];
    // the compacted queue, not the ray-coherence one: compaction keeps path indices nearly
    // ascending, so the pool's SoA reads and writes stay coalesced
    const int* q = pool.sort_buckets > 1 ? sorted_queue(pool.q_sorted, pool.q[in], n) : pool.q[in];
    int* qout = pool.q[in ^ 1];
    if (blockIdx.x == 0 && threadIdx.x == 0 && pool.fetch) pool.fetch[0] = 0u;   // the next k_closest's ticket
    const WaveJobs wj = BATCH ? WaveJobs(pool, bt) : WaveJobs{};
    ShadeCursor cur(n, pool.fetch ? pool.fetch + 3 : nullptr, pool.lockstep != 0);
    unsigned k;
    while (cur.next(k)) {
        bool alive = false, shadow = false, shadow2 = false;
        int i = -1;
        unsigned rk = 0u, sk = 0u;   // ray-coherence keys of the spawned ray / shadow query
        const bool live = k < n;
        if (live || cur.lockstep) {   // a lane past the end reads the last path and stores nothing
            i = q[live ? k : n - 1u];
            const int job = BATCH ? wj.of(bt, i) : 0;
            const DevScene& S = BATCH ? bt.scenes[job] : S0;
            const ProgParams& P = BATCH ? bt.progs[job] : P0;
            float4 ro = pool.ray_o[i], rd = pool.ray_d[i];
            WalkState<Col> ws;
            ws.r.o = xyz(ro);
            ws.r.d = xyz(rd);
            ws.prev_bsdf_pdf = ro.w;
            ws.eta_scale = rd.w;
            ws.thr = col_ld<Col>(pool.thr[i]);
            ws.rad = col_ld<Col>(pool.rad[i]);
            ws.prev_qp = xyz(pool.prev_q[i]);
            if constexpr (SPECTRAL) ws.wl.lambda = pool.wl[i];
            int4 st = pool.st[i];
            ws.bounce = st.x;
            ws.cur_med = st.y;
            ws.nulls = st.z;
            ws.prev_delta = st.w != 0;
            uint2 rs = pool.rng[i];
            ws.rng.base = rs.x;
            ws.rng.dim = rs.y;
            GradAcc ga;
            int sh_mat = 0;
            // the NEE query's lobe derivative: dlog f toward the light (per channel) and its
            // scalar part (GGX alpha beside the per-channel F0 part)
            NeeGrad sg{kGradKindNone, f3(0.0f), 0.0f};
            if constexpr (ADJ) {
                ws.lrem = xyz(pool.l_rem[i]);
                ga.s = s_grad;
                ga.dl = xyz(pool.dl[i]);
            }
            float4 hf = pool.hit[i];
            int4 hi = pool.hit_i[i];
            HitRec hr;
            hr.t = hf.x; hr.u = hf.y; hr.v = hf.z;
            hr.region = hi.x; hr.element = hi.y; hr.prim = hi.z;
            PoolSink<Col> sink(pool, i);
            alive = walk_iteration<Col, DIRECT, MEDIA, ADJ>(S, P, ws, hr, sink, ga, sh_mat, sg, live, [&] { cur.phase(); });
            shadow = sink.shadow;
            shadow2 = sink.shadow2;
            if (pool.ray_sort) {
                if (alive) rk = ray_key(S, ws.r.o, ws.r.d);
                if (shadow) {
                    float4 so = pool.sh_o[i], sd = pool.sh_d[i];
                    sk = ray_key(S, xyz(so), xyz(sd));
                }
            }
            if (live) {
                pool.rad[i] = col_st(ws.rad, 0.0f);
                pool.thr[i] = col_st(ws.thr, 0.0f);   // with rad: the whole record, for a dying path too
            }
            if constexpr (ADJ) {
                if (live) pool.l_rem[i] = f4(ws.lrem, 0.0f);
                if (shadow) {
                    pool.sh_g[i] = f4(sg.dnee, sg.dw);
                    pool.sh_gm[i] = sh_mat | (sg.kind << 16);
                }
            }
            if (alive) {
                pool.ray_o[i] = f4(ws.r.o, ws.prev_bsdf_pdf);
                pool.ray_d[i] = f4(ws.r.d, ws.eta_scale);
                pool.prev_q[i] = f4(ws.prev_qp, 0.0f);
                pool.st[i] = make_int4(ws.bounce, ws.cur_med, ws.nulls, ws.prev_delta ? 1 : 0);
                pool.rng[i] = make_uint2(ws.rng.base, ws.rng.dim);
            }
        }
        int slot = warp_append(&pool.cnt[in ^ 1], alive);
        if (alive) qout[slot] = i;
        int sslot = warp_append(&pool.cnt[2], shadow);
        if (shadow) pool.shq[sslot] = i;
        if (pool.ray_sort) {
            if (alive) pool.rkey[slot] = (unsigned char)rk;
            if (shadow) pool.skey[sslot] = (unsigned char)sk;
        }
        if (MEDIA) {
            int s2 = warp_append(&pool.cnt[4], shadow2);
            if (shadow2) pool.shq2[s2] = i;
        }
    }
    if constexpr (ADJ) grad_block_flush(s_grad, PTR_GRAD_SLOTS * S0.n_materials, adj.grads);
}

// Shadow queries: opaque visibility (shadow/opaque/opaque.glsl:16-19) or the media
// segment walker (shadow/media/media.glsl:29-62); the surviving fraction scales the
// stored contribution prefix into the path's radiance.
// slot 1 reads the second shadow slot (the equiangular segment queries); its launch
// precedes the slot-0 launch of the same iteration, so the two never add to one path's
// radiance concurrently.
// ADJ: the replay pass also folds the query's gradient terms — the lobe derivative D of
// its vertex and d log T / d theta of every medium segment the shadow ray crossed.
constexpr int kAdjMaxMedia = 4;            // distinct media one adjoint shadow query may cross
constexpr unsigned kErrAdjMedia = 8u;      // ... more were crossed (their terms were dropped)
// The distinct media a shadow query crossed and its length in each (the adjoint's terms).
struct ShadowMedia {
    int id[kAdjMaxMedia];
    float len[kAdjMaxMedia];
    int n = 0;
};
// What one shadow query lets through: opaque visibility (shadow/opaque/opaque.glsl:16-19) or
// the media segment walker (shadow/media/media.glsl:29-62).  seed_of() starts the query's own
// stream, called only where a heterogeneous medium asks for it.  collect: note the media
// crossed in mm; flag_more: raise the adjoint's guard where they exceed it (a recording
// walk logs a negative count there instead).
template <class Col, bool MEDIA, class SeedOf>
__device__ __forceinline__ Col shadow_visibility(const DevScene& S, const ProgParams& P, const Ray& sr, float max_dist, f3 light_p,
                                                 int crossings_left, const Wl& wl, SeedOf seed_of, bool collect, bool flag_more,
                                                 ShadowMedia& mm, Work* work) {
    constexpr bool SPECTRAL = sizeof(Col) == sizeof(s4);
    if (!MEDIA) return scene_any<false>(S, sr, max_dist, work) ? Col(0.0f) : Col(1.0f);
    Col T(1.0f);
    Rng srng;
    bool srng_live = false;
    // the medium of a segment attenuates only a query that gets past it: a query that an
    // optical surface blocks is done without its point classification and transmittance
    auto attenuate = [&](const Ray& seg, int medium, float seg_len) {
        const int med_mat = material_of(S, medium);
        if (!mat_has_medium(S, med_mat)) return;
        bool het = false;
        if constexpr (!SPECTRAL) {
            const ptr_material& smm = S.materials[med_mat];
            if (PTR_SPEC_HET && S.has_het && mat_is_het(smm)) {   // ratio tracking on the query's own stream
                het = true;
                if (!srng_live) { srng = seed_of(); srng_live = true; }
                T = T * medium_ratio_track(S, smm, seg, seg_len, srng, scatter_live(S, P, med_mat));
            }
        }
        if (!het) T = T * medium_transmittance<Col>(S, P, med_mat, seg_len, wl);
        if (collect) {
            int e = 0;
            while (e < mm.n && mm.id[e] != med_mat) e++;
            if (e < mm.n) mm.len[e] += seg_len;
            else if (mm.n < kAdjMaxMedia) { mm.id[mm.n] = med_mat; mm.len[mm.n] = seg_len; mm.n++; }
            else if (flag_more) flag_error(S, kErrAdjMedia);
        }
    };
    if (PTR_SPEC_NULL < 0 ? !S.has_null : !PTR_SPEC_NULL) {   // every surface is optical: any hit before the light blocks the query
        const float remaining = length(light_p - sr.o) - kShadowBackoff;
        if (remaining <= 0.0f) return T;
        if (scene_any(S, sr, gmin(remaining, kMaxDist), work)) return Col(0.0f);
        attenuate(sr, scene_region_at(S, sr.o), remaining);
        return T;
    }
    if (PTR_SPEC_NULL == 0) return T;
    int medium = 0;
    Ray seg = sr;
    for (int crossed = 0; crossed <= crossings_left; crossed++) {
        float remaining = length(light_p - seg.o) - kShadowBackoff;
        if (remaining <= 0.0f) return T;
        HitRec hr = scene_closest(S, seg, work);
        bool hit_boundary = hr.region >= 0 && hr.t < remaining;
        // an optical surface blocks the query: decided from the hit region alone
        if (hit_boundary) {
            const int om = material_of(S, hr.region);
            if (!(om >= 0 && S.materials[om].model == PTR_MAT_NONE)) return Col(0.0f);
        }
        if (crossed == 0) medium = scene_region_at(S, sr.o);
        attenuate(seg, medium, hit_boundary ? hr.t : remaining);
        if (!hit_boundary) return T;
        Hit h;
        fill_hit(S, seg, hr, h, false, true);
        medium = h.region_to;
        seg = ray_spawn(h, seg.d);
        seg.d = normalize(light_p - seg.o);
    }
    return Col(0.0f);
}
// The walk log's shadow record (PathPool::hit_log): visibility rgb and the media count, then
// up to two (medium, length) pairs; a count of -1 marks a query the replay walks again.
__device__ __forceinline__ void shadow_log_write(float4* rec, f3 vis, const ShadowMedia& mm) {
    rec[0] = make_float4(vis.x, vis.y, vis.z, __int_as_float(mm.n <= 2 ? mm.n : -1));
    rec[1] = make_float4(__int_as_float(mm.n > 0 ? mm.id[0] : -1), mm.n > 0 ? mm.len[0] : 0.0f,
                         __int_as_float(mm.n > 1 ? mm.id[1] : -1), mm.n > 1 ? mm.len[1] : 0.0f);
}
__device__ __forceinline__ bool shadow_log_read(const float4* rec, f3& vis, ShadowMedia& mm) {
    const float4 a = rec[0], b = rec[1];
    const int n = __float_as_int(a.w);
    if (n < 0) return false;
    vis = f3(a.x, a.y, a.z);
    mm.n = n;
    mm.id[0] = __float_as_int(b.x);
    mm.len[0] = b.y;
    mm.id[1] = __float_as_int(b.z);
    mm.len[1] = b.w;
    return true;
}
// The replay's gradient terms of one shadow query whose contribution is add: its vertex's lobe
// derivative and d log T / d theta of every medium it crossed.
__device__ __forceinline__ void shadow_grads(const DevScene& S, const ProgParams& P, const GradAcc& ga, f3 add, int vmat, int kind,
                                             f3 D, float dw, const ShadowMedia& mm) {
    if (kind == kGradKindAlbedo) ga.vec(vmat, PTR_GRAD_COLOR_R, add, D);
    else if (kind == kGradKindGGX) {
        ga.vec(vmat, PTR_GRAD_COLOR_R, add, D);
        ga.scl(vmat, PTR_GRAD_ALPHA, add, dw);
    }
    else if (kind == kGradKindPhase) ga.scl(vmat, PTR_GRAD_HG_G, add, D.x);
    for (int e = 0; e < mm.n; ++e) {   // T = exp(-st len) (scattering) or exp(-(1-a) st len)
        GreyMedium g = grey_medium(S.materials[mm.id[e]]);
        if (scatter_live(S, P, mm.id[e])) {
            ga.scl(mm.id[e], PTR_GRAD_SIGMA_T, add, -mm.len[e]);
        } else {
            ga.scl(mm.id[e], PTR_GRAD_SIGMA_T, add, -(1.0f - g.a) * mm.len[e]);
            ga.scl(mm.id[e], PTR_GRAD_MEDIUM_ALBEDO, add, g.st * mm.len[e]);
        }
    }
}

// Opaque shadow queries over the same scene form, with the same per-lane refill: the
// regions before the instanced one, the flat any-hit walk, then the regions after it (the
// order of scene_any); an unoccluded query adds its stored contribution as k_shadow does.
template <class Col, bool COUNT, bool WIDE>
__device__ __forceinline__ void shadow_refill(const DevScene& S, const PathPool& pool, const int* shq, unsigned n, int slot,
                                              const Pair<float4> a_o, const Pair<float4> a_d, const Pair<float4> a_lp,
                                              const Pair<float4> a_c, unsigned* ticket, Work* w) {
    constexpr bool SPECTRAL = sizeof(Col) == sizeof(s4);
    const int fr = S.flat_region;
    const FlatScene fs = flat_scene<WIDE>(S, S.batches[S.regions[fr].ref]);
    const unsigned lane = threadIdx.x & 31u;
    FlatWalk<WIDE> f;
    Ray r;
    HitRec unused;
    float max_dist = 0.0f;
    int i = -1, steps = 0;
    bool active = false, exhausted = false;
    for (;;) {
        if (!exhausted) {
            const unsigned need = __ballot_sync(0xffffffffu, !active);
            if (__popc(need) >= kRefillMin) {
                const int leader = __ffs(need) - 1;
                unsigned base = 0u;
                if ((int)lane == leader) base = atomicAdd(ticket, (unsigned)__popc(need));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (base + (unsigned)__popc(need) >= n) exhausted = true;
                if (!active) {
                    const unsigned k = base + __popc(need & lanemask_lt());
                    if (k < n) {
                        i = shq[k];
                        const float4 so = a_o[i], sd = a_d[i];
                        r.o = xyz(so);
                        r.d = xyz(sd);
                        max_dist = so.w;
                        bool blocked = false;
                        for (int g = 0; g < fr && !blocked; ++g) {
                            float t;
                            blocked = analytic_root(S.regions[g], r, t) && t < max_dist;
                        }
                        if (!blocked) {            // an occluded query is finished: nothing to add
                            f.init(fs, r, max_dist, COUNT ? w : nullptr);
                            steps = 0;
                            active = true;
                        }
                    }
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) break;
        if (!active) continue;
        bool more = f.template step<true>(S, fs, fr, r, unused, max_dist, COUNT ? w : nullptr);
        if (more && ++steps >= kFlatGuard) {
            flag_error(S, kErrCwGuard);
            more = false;
        }
        if (!more) {
            bool blocked = f.found;
            for (int g = fr + 1; g < S.n_regions && !blocked; ++g) {
                float t;
                blocked = analytic_root(S.regions[g], r, t) && t < max_dist;
            }
            if (!blocked) {
                const float4 c = a_c[i];
                const Col cc = col_ld<Col>(c);
                float cpdf = c.w;
                if constexpr (SPECTRAL) cpdf = slot ? pool.sh2_pdf[i] : pool.sh_pdf[i];
                const Col vis(1.0f);
                const Col add = cc * vis * a_lp[i].w / cpdf;
                pool.rad[i] = col_st(col_ld<Col>(pool.rad[i]) + add, 0.0f);
            }
            active = false;
        }
    }
}

template <class Col, bool MEDIA, bool COUNT, bool BATCH, bool ADJ = false>
__global__ void __launch_bounds__(256, PTR_TRACE_MIN_BLOCKS) k_shadow(const __grid_constant__ DevScene S0, PathPool pool, ProgParams P0, BatchTables bt,
                                                                      int slot, AdjParams adj = AdjParams{}) {
    constexpr bool SPECTRAL = sizeof(Col) == sizeof(s4);
    static_assert(!(ADJ && SPECTRAL), "the adjoint replay is RGB only");
    extern __shared__ double s_grad[];
    if constexpr (ADJ) grad_block_init(s_grad, PTR_GRAD_SLOTS * S0.n_materials);
    const unsigned n = pool.cnt[slot ? 4 : 2];
    if (blockIdx.x == 0 && threadIdx.x == 0) pool.stats[1] += n;
    const int* shq = slot ? pool.shq2 : (pool.ray_sort ? sorted_queue(pool.shq_s, pool.shq, n) : pool.shq);
    const Pair<float4> a_o = slot ? pool.sh2_o : pool.sh_o;
    const Pair<float4> a_d = slot ? pool.sh2_d : pool.sh_d;
    const Pair<float4> a_lp = slot ? pool.sh2_lp : pool.sh_lp;
    const Pair<float4> a_c = slot ? pool.sh2_c : pool.sh_c;
    Work wk{0u, 0u, 0u, 0u};
    // the adjoint's walk log: this launch's slot-0 shadow records (two float4 per path after
    // its closest hit: visibility rgb and the media count, then up to two (medium, length)
    // pairs; a count of -1 marks a query the replay walks again)
    float4* slog = nullptr;
    if constexpr (!BATCH && !SPECTRAL)
        if (slot == 0 && hit_log_slice(pool)) slog = hit_log_slice(pool) + 2;
    const bool rec = !ADJ && slog && pool.hit_log_mode == 1;
    const bool rep = ADJ && slog && pool.hit_log_mode == 2;
    if (PTR_REFILL && kHasMesh && !MEDIA && !BATCH && !ADJ && !rec && pool.fetch && S0.flat_region >= 0) {
        const DevBatch& b = S0.batches[S0.regions[S0.flat_region].ref];
        const bool wide = flat_wide_ok(S0, b), binary = flat_binary_ok(S0, b);
        unsigned* ticket = pool.fetch + 1 + slot;
        if (wide) shadow_refill<Col, COUNT, true>(S0, pool, shq, n, slot, a_o, a_d, a_lp, a_c, ticket, &wk);
        else if (binary) shadow_refill<Col, COUNT, false>(S0, pool, shq, n, slot, a_o, a_d, a_lp, a_c, ticket, &wk);
        if (wide || binary) {
            if (COUNT) flush_work(S0, wk);
            return;
        }
    }
    const WaveJobs wj = BATCH ? WaveJobs(pool, bt) : WaveJobs{};
    QueueCursor cur(n, pool.fetch ? pool.fetch + 1 + slot : nullptr);
    unsigned k;
    while (cur.next(k)) {
        if (k >= n) continue;
        int i = shq[k];
        const int job = BATCH ? wj.of(bt, i) : 0;
        const DevScene& S = BATCH ? bt.scenes[job] : S0;
        const ProgParams& P = BATCH ? bt.progs[job] : P0;
        float4 so = a_o[i], sd = a_d[i], lp = a_lp[i], c = a_c[i];
        Col cc = col_ld<Col>(c);
        float cpdf = c.w;
        Wl wl;
        if constexpr (SPECTRAL) {
            cpdf = slot ? pool.sh2_pdf[i] : pool.sh_pdf[i];
            wl.lambda = pool.wl[i];
        }
        Ray sr;
        sr.o = xyz(so);
        sr.d = xyz(sd);
        Col vis;
        ShadowMedia mm;
        bool logged = false;
        if constexpr (ADJ) {
            if (rep) logged = shadow_log_read(slog + 4 * (size_t)i, vis, mm);
        }
        if (!logged)
            vis = shadow_visibility<Col, MEDIA>(S, P, sr, so.w, xyz(lp), __float_as_int(sd.w), wl,
                                                [&] { return shadow_rng(pool.rng[i].x, pool.sh_seed[i]); }, ADJ || rec, ADJ, mm,
                                                COUNT ? &wk : nullptr);
        if constexpr (!ADJ && !SPECTRAL) {
            if (rec) shadow_log_write(slog + 4 * (size_t)i, vis, mm);
        }
        if (!spectrum_is_black(vis)) {
            float w = lp.w;
            Col add = cc * vis * w / cpdf;
            pool.rad[i] = col_st(col_ld<Col>(pool.rad[i]) + add, 0.0f);
            if constexpr (ADJ) {
                GradAcc ga;
                ga.s = s_grad;
                ga.dl = xyz(pool.dl[i]);
                float4 lr = pool.l_rem[i];
                pool.l_rem[i] = make_float4(lr.x - add.x, lr.y - add.y, lr.z - add.z, 0.f);
                const int gm = pool.sh_gm[i];
                const float4 Dg = pool.sh_g[i];
                shadow_grads(S, P, ga, add, gm & 0xFFFF, gm >> 16, xyz(Dg), Dg.w, mm);
            }
        }
    }
    if (COUNT) flush_work(S0, wk);
    if constexpr (ADJ) grad_block_flush(s_grad, PTR_GRAD_SLOTS * S0.n_materials, adj.grads);
}

// ---- the whole walk in one kernel ------------------------------------------------------
// k_walk runs every iteration of a path in one thread, its state in registers: no path
// record, queue or shadow query travels through memory, only 16 bytes of radiance per path
// go to the film pass.  A lane whose path has ended takes the next one at once (warp-aggregated
// tickets), so lanes stay busy whatever the paths' lengths, and a wave is one launch instead
// of three per iteration.  The arithmetic and the order of the random numbers and radiance
// sums are walk_iteration's and shadow_visibility's, so samples are bit-identical to the
// wavefront kernels'.
// What bounds it is instruction issue (70 % of the slots, 17.5 of 32 lanes on the Cornell box)
// and, were its warps to run free, the instruction cache: a walk is 70 to 220 KB of code built for
// a scene, 150 to 710 in the library's form.  A block's warps therefore run each part of an
// iteration together, so that one pass of the part's code through the cache serves them all
// (media and spectral workload, 16.8 M paths: 128 ms with free-running warps, 41 ms in step;
// adjoint 15.4 and 9.3; fog room in tiles 50.0 and 48.4).
// 64 registers (1024 threads per SM) measured faster than 80 or 128, and two blocks of 512
// faster than four of 256 (fewer passes through the cache; the 64-job mix 279 ms at 80
// registers, 276 with four blocks, 267 with two; the adjoint 7.4, 7.1 and 6.5); refilling at
// the first idle lane faster than at the eighth (363 against 372).
struct WalkArgs {
    float4* film;                 // radiance of path base + i at [i]
    float4* aov;                  // first-hit samples, two per path (null: none)
    unsigned* ticket;             // zero at the launch
    unsigned long long* stats;    // [0] closest queries, [1] shadow queries, [2] paths
    long long base;               // the wave's paths: [base, base + n) of the frame or job space
    unsigned n;
    int iters;                    // walk iterations at most
    float4* hit_log;              // PathPool::hit_log of the adjoint (null: none)
    long long hit_log_stride;
    int hit_log_iters;
};

// k_walk's sink: an iteration's queries stay in registers until the walk resolves them.
template <class Col>
struct WalkQuery {
    Ray r;
    float max_dist;
    int crossings;
    f3 light_p;
    float w;
    Col contrib;
    float pdf;
    bool live;
};
template <class Col>
struct WalkSink {
    WalkQuery<Col> seg, vtx;
    unsigned dim;
    float4 prev_n;
    float4* aov_p;
    __device__ __forceinline__ void segment_query(f3 o, f3 d, int crossings, f3 light_p, Col contrib, float pdf) {
        seg = WalkQuery<Col>{Ray{o, d}, 0.0f, crossings, light_p, 1.0f, contrib, pdf, true};
    }
    __device__ __forceinline__ void vertex_query(f3 o, float max_dist, f3 d, int crossings, f3 light_p, float w, Col contrib, float pdf) {
        vtx = WalkQuery<Col>{Ray{o, d}, max_dist, crossings, light_p, w, contrib, pdf, true};
    }
    __device__ __forceinline__ void seed(unsigned d) { dim = d; }
    __device__ __forceinline__ void put_prev_n(float4 n) { prev_n = n; }
    __device__ __forceinline__ float4 get_prev_n() const { return prev_n; }
    __device__ __forceinline__ float4* aov() const { return aov_p; }
};

constexpr int kWalkBlock = 512;   // threads per block at most (2 blocks per SM)
constexpr int kTrackSteps = 32;   // 16, 32 and 128: 50.4, 50.0 and 67.7 ms for the fog room in tiles
template <class Col, int DIRECT, bool MEDIA, bool BATCH, bool ADJ = false>
__global__ void __launch_bounds__(kWalkBlock, 2) k_walk(const __grid_constant__ DevScene S0, ProgParams P0, FrameParams F0, BatchTables bt,
                                                                   WalkArgs wa, AdjParams adj = AdjParams{}) {
    constexpr bool SPECTRAL = sizeof(Col) == sizeof(s4);
    static_assert(!(ADJ && SPECTRAL), "the adjoint replay is RGB only");
    extern __shared__ double s_grad[];
    if constexpr (ADJ) grad_block_init(s_grad, PTR_GRAD_SLOTS * S0.n_materials);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&wa.stats[2], (unsigned long long)wa.n);
    const WaveJobs wj = BATCH ? WaveJobs(wa.base, (long long)wa.n, bt) : WaveJobs{};
    // the region every path starts in (a pinhole's rays share their origin): once per thread
    int cam_med = !BATCH && MEDIA ? scene_region_at(S0, ld3(F0.cam.position)) : -1;
    unsigned n_closest = 0u, n_shadow = 0u;
    WalkState<Col> ws;
    WalkSink<Col> sink;
    GradAcc ga;
    ga.s = s_grad;
    int i = -1, job = 0, it = 0;
    bool active = false, exhausted = false;
    // Delta tracking runs kTrackSteps collisions at a time between the other lanes' iterations:
    // a ray that escapes through an ambient fog takes thousands, one that scatters a few, and
    // a warp that finished each segment in turn would wait for its longest.
    constexpr bool TRACK = MEDIA && !SPECTRAL && !ADJ && PTR_SPEC_HET;
    DeltaTrack track;
    bool tracking = false;
    HitRec hr;
    // the block's warps run each part of an iteration together
    auto phase = [] { __syncthreads(); };
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active);
        if (!exhausted && idle != 0u) {
            unsigned first = 0u;
            if ((threadIdx.x & 31u) == 0u) first = atomicAdd(wa.ticket, (unsigned)__popc(idle));
            first = __shfl_sync(0xffffffffu, first, 0);
            exhausted = first + (unsigned)__popc(idle) >= wa.n;
            const unsigned k = first + __popc(idle & lanemask_lt());
            if (!active && k < wa.n) {
                active = true;
                i = (int)k;
                it = 0;
                if (BATCH) job = wj.of(bt, i);
                const DevScene& S = BATCH ? bt.scenes[job] : S0;
                const FrameParams& F = BATCH ? bt.jobs[job].frame : F0;
                int pix, sample;
                split_path(wa.base + i - (BATCH ? bt.offsets[job] : 0ll), (unsigned)F.width * (unsigned)F.height, pix, sample);
                float4 lambda;
                camera_path<SPECTRAL>(F, pix, sample, ws.rng, ws.r, lambda);
                if constexpr (SPECTRAL) ws.wl.lambda = lambda;
                ws.prev_bsdf_pdf = 0.0f;
                ws.eta_scale = 1.0f;
                ws.thr = Col(1.0f);
                ws.rad = Col(0.0f);
                ws.prev_qp = ws.r.o;
                ws.bounce = 0;
                if (BATCH) cam_med = S.has_media ? scene_region_at(S, ws.r.o) : -1;
                ws.cur_med = cam_med;
                ws.nulls = 0;
                ws.prev_delta = true;
                if constexpr (ADJ) {   // the forward walk left this path's total radiance
                    ws.lrem = xyz(wa.film[i]);
                    const float* g = adj.dl_image + 3 * (size_t)pix;
                    ga.dl = f3(g[0] * adj.inv_spp, g[1] * adj.inv_spp, g[2] * adj.inv_spp);
                }
                sink.aov_p = nullptr;
                if (wa.aov) {
                    sink.aov_p = wa.aov + 2 * (size_t)i;
                    sink.aov_p[0] = make_float4(0.f, 0.f, 0.f, 0.f);
                    sink.aov_p[1] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
        if (!__syncthreads_or(active)) break;
        const DevScene& S = BATCH ? bt.scenes[job] : S0;
        const ProgParams& P = BATCH ? bt.progs[job] : P0;
        // this iteration's record of the adjoint's walk log: the closest hit, then the query
        float4* rec = (!BATCH && !SPECTRAL && active && wa.hit_log && it < wa.hit_log_iters)
                          ? wa.hit_log + 4 * ((size_t)it * (size_t)wa.hit_log_stride + (size_t)i) : nullptr;
        if (active && !tracking) {
            if (ADJ && rec) {
                const float4 hf = rec[0];
                const int4 hi = float4_as_int4(rec[1]);
                hr.t = hf.x; hr.u = hf.y; hr.v = hf.z;
                hr.region = hi.x; hr.element = hi.y; hr.prim = hi.z;
            } else {
                hr = scene_closest(S, ws.r);
                if (!ADJ && rec) {
                    rec[0] = make_float4(hr.t, hr.u, hr.v, 0.f);
                    rec[1] = int4_as_float4(make_int4(hr.region, hr.element, hr.prim, 0));
                }
            }
            n_closest++;
        }
        phase();
        if constexpr (TRACK) {
            if (active && S.has_het) {
                const int med_mat = material_of(S, ws.cur_med);
                if (mat_has_medium(S, med_mat) && mat_is_het(S.materials[med_mat]) && scatter_live(S, P, med_mat)) {
                    const ptr_material& mm = S.materials[med_mat];
                    const float t_max = hr.region >= 0 ? hr.t : kMaxDist;
                    if (!tracking) {
                        const float x0 = ws.rng.next(), x1 = ws.rng.next();
                        track.begin(mm, t_max, x0, x1);
                    }
                    tracking = !track.advance(S, mm, ws.r, t_max, ws.rng, kTrackSteps);
                }
            }
            phase();
        }
        const bool live = active && !tracking;
        bool alive = false;
        int sh_mat = 0;
        NeeGrad sg{kGradKindNone, f3(0.0f), 0.0f};
        sink.seg.live = sink.vtx.live = false;
        alive = walk_iteration<Col, DIRECT, MEDIA, ADJ, TRACK>(S, P, ws, hr, sink, ga, sh_mat, sg, live, phase, &track.ms);
        phase();
        if constexpr (MEDIA && DIRECT == PTR_DIRECT_NEE && !ADJ) {   // the equiangular segment query comes first
            if (sink.seg.live) {
                ShadowMedia none;
                n_shadow++;
                const Col vis = shadow_visibility<Col, MEDIA>(S, P, sink.seg.r, 0.0f, sink.seg.light_p, sink.seg.crossings, ws.wl,
                                                              [&] { return shadow_rng(ws.rng.base, sink.dim); }, false, false, none, nullptr);
                if (!spectrum_is_black(vis)) ws.rad = ws.rad + sink.seg.contrib * vis * sink.seg.w / sink.seg.pdf;
            }
            phase();
        }
        if constexpr (DIRECT != PTR_DIRECT_NONE) {
            if (sink.vtx.live) {
                const WalkQuery<Col>& q = sink.vtx;
                ShadowMedia mm;
                Col vis;
                bool logged = false;
                n_shadow++;
                if constexpr (ADJ) {
                    if (rec) logged = shadow_log_read(rec + 2, vis, mm);
                }
                if (!logged)
                    vis = shadow_visibility<Col, MEDIA>(S, P, q.r, q.max_dist, q.light_p, q.crossings, ws.wl,
                                                        [&] { return shadow_rng(ws.rng.base, sink.dim); }, ADJ || rec, ADJ, mm, nullptr);
                if constexpr (!ADJ && !SPECTRAL) {
                    if (rec) shadow_log_write(rec + 2, vis, mm);
                }
                if (!spectrum_is_black(vis)) {
                    const Col add = q.contrib * vis * q.w / q.pdf;
                    ws.rad = ws.rad + add;
                    if constexpr (ADJ) {
                        ws.lrem = ws.lrem - add;
                        shadow_grads(S, P, ga, add, sh_mat, sg.kind, sg.dnee, sg.dw, mm);
                    }
                }
            }
            phase();
        }
        if (live && (!alive || ++it >= wa.iters)) {
            active = false;
            if constexpr (SPECTRAL) {
                const f3 px = color_to_pixel(S, col_st(ws.rad, 0.0f), ws.wl.lambda, wavelength_pdfs(BATCH ? bt.jobs[job].frame : F0, ws.wl.lambda));
                wa.film[i] = f4(px, 0.0f);
            } else if constexpr (!ADJ) {
                wa.film[i] = f4(ws.rad, 0.0f);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        n_closest += __shfl_xor_sync(0xffffffffu, n_closest, o);
        n_shadow += __shfl_xor_sync(0xffffffffu, n_shadow, o);
    }
    if ((threadIdx.x & 31u) == 0u && n_closest) {
        atomicAdd(&wa.stats[0], (unsigned long long)n_closest);
        atomicAdd(&wa.stats[1], (unsigned long long)n_shadow);
    }
    if constexpr (ADJ) grad_block_flush(s_grad, PTR_GRAD_SLOTS * S0.n_materials, adj.grads);
}

// Adds one pixel's samples of a wave, paths i, i + npix, ... below n, to its film sums in
// sample order; first: the film starts from zero here.  The samples are fetched four ahead of
// the serial FP64 sums, so a pixel keeps several loads in flight.
template <class Get>
__device__ __forceinline__ void film_pixel(double* su, double* sq, bool first, long long i, long long n, long long npix, Get get) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, q0 = 0.0, q1 = 0.0, q2 = 0.0;
    if (!first) { s0 = su[0]; s1 = su[1]; s2 = su[2]; q0 = sq[0]; q1 = sq[1]; q2 = sq[2]; }
    auto add = [&](float4 L) {
        s0 += (double)L.x; s1 += (double)L.y; s2 += (double)L.z;
        q0 += (double)L.x * (double)L.x; q1 += (double)L.y * (double)L.y; q2 += (double)L.z * (double)L.z;
    };
    for (; i + 3 * npix < n; i += 4 * npix) {
        const float4 a = get(i), b = get(i + npix), c = get(i + 2 * npix), d = get(i + 3 * npix);
        add(a); add(b); add(c); add(d);
    }
    for (; i < n; i += npix) add(get(i));
    su[0] = s0; su[1] = s1; su[2] = s2;
    sq[0] = q0; sq[1] = q1; sq[2] = q2;
}
// Fold a wave's radiance (paths [base, base + n) of the frame, path base + i at
// rad[i * stride]) into the film, per pixel in sample order, and its first-hit samples into
// theirs.  color(i, L): the pixel colour of path i's radiance.
template <class Color>
__device__ __forceinline__ void film_wave(const FrameParams& F, const float4* rad, int stride, const float4* aov, double* aov_sum,
                                          long long base, long long n, double* sum, double* sumsq, float* samples_out, Color color) {
    const long long npix = (long long)F.width * F.height;
    const long long nslot = n < npix ? n : npix;
    const unsigned pix0 = (unsigned)(base % npix);
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < nslot; j += (long long)gridDim.x * blockDim.x) {
        const long long p1 = (long long)pix0 + j;
        const size_t pix = (size_t)(p1 < npix ? p1 : p1 - npix);
        const bool first = F.fresh && base + j < npix;
        film_pixel(sum + 3 * pix, sumsq + 3 * pix, first, j, n, npix, [&](long long i) {
            const float4 L = color(i, rad[i * stride]);
            if (samples_out) {
                float* o = samples_out + 3 * (base + i);
                o[0] = L.x; o[1] = L.y; o[2] = L.z;
            }
            return L;
        });
        if (aov_sum) {   // the first-hit pictures, in the same sample order
            double* as = aov_sum + 3 * pix;
            double* ns = aov_sum + 3 * ((size_t)npix + pix);
            double a0 = 0.0, a1 = 0.0, a2 = 0.0, n0 = 0.0, n1 = 0.0, n2 = 0.0;
            if (!first) { a0 = as[0]; a1 = as[1]; a2 = as[2]; n0 = ns[0]; n1 = ns[1]; n2 = ns[2]; }
            for (long long i = j; i < n; i += npix) {
                float4 a = aov[2 * i], b = aov[2 * i + 1];
                a0 += (double)a.x; a1 += (double)a.y; a2 += (double)a.z;
                n0 += (double)b.x; n1 += (double)b.y; n2 += (double)b.z;
            }
            as[0] = a0; as[1] = a1; as[2] = a2;
            ns[0] = n0; ns[1] = n1; ns[2] = n2;
        }
    }
}
// SPECTRAL: each sample's four lanes are projected to linear sRGB first (color_to_pixel).
template <bool SPECTRAL = false>
__global__ void k_film(PathPool pool, const FrameParams* fp, double* sum, double* sumsq, float* samples_out,
                       DevScene S = DevScene{}) {
    const FrameParams F = *fp;
    film_wave(F, pool.rad.p, 2, pool.aov, pool.aov_sum, pool.wave[0], pool.wave[1], sum, sumsq, samples_out, [&](long long i, float4 L) {
        if (!SPECTRAL) return L;
        const f3 px = color_to_pixel(S, L, pool.wl[i], pool.wl_pdf[i]);
        return f4(px, 0.0f);
    });
}

// The film pass after k_walk (its radiance is already the pixel colour), which also clears the
// tickets for the next wave's walk.
__global__ void k_film_walk(FrameParams F, WalkArgs wa, double* aov_sum, double* sum, double* sumsq, float* samples_out) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *wa.ticket = 0u;
    film_wave(F, wa.film, 1, wa.aov, aov_sum, wa.base, wa.n, sum, sumsq, samples_out, [](long long, float4 L) { return L; });
}

// ---- batched renders ------------------------------------------------------------------

// Camera rays for one wave of the concatenated job space.
__global__ void k_generate_batch(PathPool pool, BatchTables bt) {
    long long base = pool.wave[0];
    long long n = bt.total - base;
    if (n > bt.capacity) n = bt.capacity;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        pool.cnt[0] = (unsigned)n;
        pool.wave[1] = n;
        pool.stats[2] += (unsigned long long)n;
        if (pool.fetch) pool.fetch[0] = 0u;
    }
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int j = job_of(bt, base + i);
        const FrameParams& F = bt.jobs[j].frame;
        int pix, sample;
        split_path(base + i - bt.offsets[j], (unsigned)F.width * (unsigned)F.height, pix, sample);
        Rng rng;
        Ray r;
        float4 unused;
        camera_path<false>(F, pix, sample, rng, r, unused);
        const DevScene& S = bt.scenes[j];
        init_slot(pool, i, rng, r, S.has_media ? scene_region_at(S, r.o) : -1);
    }
}

// Fold the wave [base, base + n) of the concatenated job space into each job's film.  The
// wave's paths of job j are one contiguous range of the index space, and one pixel's samples
// lie npix apart in it.  The first npix paths of the range (one per pixel the wave touches)
// each add their pixel's samples to the film in sample order, like k_film: the film is the
// sequential FP64 sum of every pixel's samples in sample order, so a batched film equals the
// job's plain film bit for bit, however the waves split the jobs.  The grid walks the wave's
// jobs one after another, so no path looks its job up.
__device__ __forceinline__ void film_batch(const BatchTables& bt, const float4* rad, int stride, long long base, long long n) {
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nthr = (long long)gridDim.x * blockDim.x;
    for (int j = job_of(bt, base); j < bt.n_jobs && bt.offsets[j] < base + n; ++j) {
        const BatchJob& J = bt.jobs[j];
        const long long npix = (long long)J.frame.width * J.frame.height;
        const long long off = bt.offsets[j], job_end = bt.offsets[j + 1];
        const long long lo = off > base ? off : base, hi = job_end < base + n ? job_end : base + n;
        const long long m = hi - lo < npix ? hi - lo : npix;
        for (long long t = tid; t < m; t += nthr) {
            const long long g = lo + t;
            const bool first = J.frame.fresh && g - off < npix;
            film_pixel(J.sum + 3 * ((g - off) % npix), J.sumsq + 3 * ((g - off) % npix), first, g - base, hi - base, npix,
                       [&](long long k) { return rad[k * stride]; });
        }
    }
}
__global__ void k_film_batch(PathPool pool, BatchTables bt) {
    film_batch(bt, pool.rad.p, 2, pool.wave[0], pool.wave[1]);
}

__global__ void k_film_batch_walk(BatchTables bt, WalkArgs wa) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *wa.ticket = 0u;
    film_batch(bt, wa.film, 1, wa.base, wa.n);
}

// Raw nearest-hit queries (tests and tools): per ray (o.xyz, d.xyz) the region, the
// element (instance), the ORIGINAL triangle index (or -1) and t (kMaxDist on a miss).
__global__ void k_trace_rays(const __grid_constant__ DevScene S, const float* rays, int n, int* region, int* element, int* prim, float* t_out) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        Ray r;
        r.o = f3(rays[6 * k], rays[6 * k + 1], rays[6 * k + 2]);
        r.d = f3(rays[6 * k + 3], rays[6 * k + 4], rays[6 * k + 5]);
        HitRec h = scene_closest(S, r);
        int orig = -1;
        if (h.region >= 0 && h.prim >= 0) {
            const ptr_region& g = S.regions[h.region];
            const DevMesh& m = S.meshes[g.shape == PTR_SHAPE_MESH ? g.ref : S.batches[g.ref].proto_mesh];
            const float4* tri = walks_cwbvh(S, m) ? m.tri_w : m.tri;
            orig = __float_as_int(tri[3 * h.prim].w);
        }
        int el = h.element;
        if (h.region >= 0 && S.regions[h.region].shape == PTR_SHAPE_INSTANCES) {   // the caller's instance index
            const DevBatch& b = S.batches[S.regions[h.region].ref];
            el = ((S.inst_accel == PTR_ACCEL_CWBVH && b.tlas_w) ? b.inst_id_w : b.inst_id)[h.element];
        }
        region[k] = h.region;
        element[k] = el;
        prim[k] = orig;
        t_out[k] = h.t;
    }
}

__global__ void k_set_frame(FrameParams* dst, FrameParams F) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *dst = F;
}

__global__ void k_advance(PathPool pool) {
    if (blockIdx.x == 0 && threadIdx.x == 0) pool.wave[0] += pool.wave[1];
}

// Mean / variance exports from the FP64 film.
__global__ void k_export(const double* sum, const double* sumsq, double nsamples, int npix, int what, float* out) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < npix * 3; j += gridDim.x * blockDim.x) {
        double m = sum[j] / nsamples;
        if (what == 0) out[j] = (float)m;
        else {
            double v = sumsq[j] / nsamples - m * m;
            if (v < 0.0) v = 0.0;
            out[j] = (float)(nsamples > 1.0 ? v * nsamples / (nsamples - 1.0) : 0.0);
        }
    }
}

}  // namespace ptx
