// vert_grid.cuh -- host-side entry of the grid-coefficient kernel
// (vert_grid.cu, its own translation unit).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "vert_common.cuh"

namespace gv {

// Rows of one grid column's coefficients: [NGC][G], the boundary meshes, [NGA][G].
__host__ __device__ inline size_t grid_rows(int G) { return size_t(NGC) * G + NBC + size_t(NGA) * G; }

// Whether the kernel may read a grid array where it stands: a double of this
// device's memory or of managed memory.  err, a: what
// cudaPointerGetAttributes(&a, p) gave.  Any other array (host memory, another
// device's, an address that is no multiple of 8, or none) goes through a copy,
// which takes all of these or answers with an error.
inline bool grid_in_place(const void* p, cudaError_t err, const cudaPointerAttributes& a, int device) {
  if (!p || reinterpret_cast<uintptr_t>(p) % sizeof(double) != 0 || err != cudaSuccess) return false;
  return a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == device);
}

// Forms the coefficients of gcols grid columns (device arrays [G][gcols])
// into out [grid_rows(G)][gcols].
cudaError_t grid_launch(int nAlts, int64_t gcols, const double* alt, const double* grav, const double* dalt_c,
                        const double* inv_r, double* out, cudaStream_t stream);

}  // namespace gv
