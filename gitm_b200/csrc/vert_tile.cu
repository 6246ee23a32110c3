// vert_tile.cu -- one tile-kernel instantiation per translation unit, built
// once for every entry of GV_TILE_INSTANCES (vert_instances.h) with
// -DGV_ID=<id> -DGV_SAVE=... -DGV_NA=...; exports the kernel's address and
// the setter of this unit's copy of the constant table.
#include "vert_tile.cuh"
#include "vert_instances.h"

#if !defined(GV_ID) || !defined(GV_SAVE) || !defined(GV_NA)
#error "vert_tile.cu is built once per GV_TILE_INSTANCES entry with its -DGV_* values"
#endif

#define GV_CAT2(a, b) a##b
#define GV_CAT(a, b) GV_CAT2(a, b)

namespace gv {

const void* GV_CAT(step_kernel_, GV_ID)() { return (const void*)vert_tile_kernel<GV_NA, GV_SAVE>; }

cudaError_t GV_CAT(step_consts_, GV_ID)(const Consts& k) { return cudaMemcpyToSymbol(c_k, &k, sizeof k); }

}  // namespace gv
