// walk.h — the library's builds of the one-kernel walk (walk.cu).
#pragma once

namespace ptx_host {

// The k_walk of a program form; launch it with k_walk's parameters.  batch: the job tables'
// form (RGB only); adj: the adjoint's replay (RGB only).
const void* walk_kernel(int direct, bool media, bool spectral, bool batch, bool adj);

}  // namespace ptx_host
