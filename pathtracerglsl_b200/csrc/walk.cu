// walk.cu — the precompiled k_walk of every program form.
//
// Scenes with triangle meshes never take the one-kernel walk, so this unit compiles the
// device headers without the mesh occupants (PTR_SPEC_MESH 0, no mesh lights): the
// two-level mesh walk's stacks and code would otherwise sit in every kernel's frame.  Its own
// namespace keeps these reduced builds of the headers apart from ptx_rt.cu's full ones.
#define ptx ptx_mesh_free
#define PTR_SPEC_MESH 0
#define PTR_SPEC_LIGHTS 0x7u   // quad, sphere, point
#define PTR_SPEC_SHAPES 0x2Fu  // plane, sphere, quad, box, instanced spheres
#include "device/wavefront.cuh"
#include "walk.h"

using namespace ptx;

template <class Col, bool BATCH, bool ADJ>
static const void* pick(int direct, bool media) {
    switch (direct * 2 + (media ? 1 : 0)) {
        case 0: return (const void*)k_walk<Col, PTR_DIRECT_NONE, false, BATCH, ADJ>;
        case 1: return (const void*)k_walk<Col, PTR_DIRECT_NONE, true, BATCH, ADJ>;
        case 2: return (const void*)k_walk<Col, PTR_DIRECT_NEE, false, BATCH, ADJ>;
        case 3: return (const void*)k_walk<Col, PTR_DIRECT_NEE, true, BATCH, ADJ>;
        case 4: return (const void*)k_walk<Col, PTR_DIRECT_MIS, false, BATCH, ADJ>;
        default: return (const void*)k_walk<Col, PTR_DIRECT_MIS, true, BATCH, ADJ>;
    }
}

const void* ptx_host::walk_kernel(int direct, bool media, bool spectral, bool batch, bool adj) {
    if (spectral) return pick<s4, false, false>(direct, media);
    if (batch) return pick<f3, true, false>(direct, media);
    return adj ? pick<f3, false, true>(direct, media) : pick<f3, false, false>(direct, media);
}
