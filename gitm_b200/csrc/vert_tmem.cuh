// vert_tmem.cuh -- tensor memory as scratch of a thread: doubles kept across
// phases without shared memory or registers (the tile kernel and the adjoint
// kernel).  A warp reaches the 32 lanes of its quarter, a lane per thread; a
// double is two 32-bit columns.
//
// Every call is made by whole warps.  The instructions are .aligned: PTX
// leaves them undefined where lanes of the warp come to them apart, as they
// may after any branch that split them (an argument outside exp_n's range, a
// division's special cases, a cell at a column's end), so each begins by
// bringing the warp together.  That costs little (1 degree globe, 16 steps:
// 38.4 ms without and with; AUSM at 2.5 degrees, 4 steps: 5.96 -> 6.05 ms; a
// rollout of 4 steps at 2.5 degrees: 13.9 -> 14.0 ms), so no access is exempt.
#pragma once

#include <cstdint>

namespace gv {

// Takes `columns` columns for the CTA, the base address to shared memory at
// `where`; gives them back.  By one warp.
template <int columns>
__device__ __forceinline__ void tm_alloc(const void* where) {
  const uint32_t a = uint32_t(__cvta_generic_to_shared(where));
  __syncwarp();
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "n"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int columns>
__device__ __forceinline__ void tm_free(uint32_t base) {
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(columns));
}

__device__ __forceinline__ void tm_put(uint32_t a, double v) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(a), "r"(__double2loint(v)),
               "r"(__double2hiint(v))
               : "memory");
}
__device__ __forceinline__ double tm_get(uint32_t a) {
  __syncwarp();
  uint32_t lo, hi;
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(lo), "=r"(hi)
      : "r"(a)
      : "memory");
  return __hiloint2double(int(hi), int(lo));
}
__device__ __forceinline__ void tm_put_wait() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Groups of N doubles.  get waits in the statement itself, so its outputs are
// ready; three blocks share one wait.
__device__ __forceinline__ void tm_put(uint32_t a, const double (&v)[4]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a),
      "r"(__double2loint(v[0])), "r"(__double2hiint(v[0])), "r"(__double2loint(v[1])), "r"(__double2hiint(v[1])),
      "r"(__double2loint(v[2])), "r"(__double2hiint(v[2])), "r"(__double2loint(v[3])), "r"(__double2hiint(v[3]))
      : "memory");
}
__device__ __forceinline__ void tm_get(uint32_t a, double (&v)[4]) {
  __syncwarp();
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(a)
      : "memory");
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = __hiloint2double(int(r[2 * j + 1]), int(r[2 * j + 0]));
  }
}
__device__ __forceinline__ void tm_get(uint32_t a, uint32_t b, uint32_t c, double (&u)[4], double (&v)[4],
                                       double (&w)[4]) {
  __syncwarp();
  uint32_t r[24];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%25];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%26];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
      : "r"(a), "r"(b), "r"(c)
      : "memory");
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    u[j] = __hiloint2double(int(r[2 * j + 1]), int(r[2 * j + 0]));
    v[j] = __hiloint2double(int(r[2 * j + 9]), int(r[2 * j + 8]));
    w[j] = __hiloint2double(int(r[2 * j + 17]), int(r[2 * j + 16]));
  }
}
__device__ __forceinline__ void tm_put(uint32_t a, const double (&v)[8]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(a),
      "r"(__double2loint(v[0])), "r"(__double2hiint(v[0])), "r"(__double2loint(v[1])), "r"(__double2hiint(v[1])),
      "r"(__double2loint(v[2])), "r"(__double2hiint(v[2])), "r"(__double2loint(v[3])), "r"(__double2hiint(v[3])),
      "r"(__double2loint(v[4])), "r"(__double2hiint(v[4])), "r"(__double2loint(v[5])), "r"(__double2hiint(v[5])),
      "r"(__double2loint(v[6])), "r"(__double2hiint(v[6])), "r"(__double2loint(v[7])), "r"(__double2hiint(v[7]))
      : "memory");
}
__device__ __forceinline__ void tm_get(uint32_t a, double (&v)[8]) {
  __syncwarp();
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(a)
      : "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = __hiloint2double(int(r[2 * j + 1]), int(r[2 * j + 0]));
  }
}
__device__ __forceinline__ void tm_get(uint32_t a, uint32_t b, uint32_t c, double (&u)[8], double (&v)[8],
                                       double (&w)[8]) {
  __syncwarp();
  uint32_t r[48];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%48];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%49];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47}, [%50];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
      : "r"(a), "r"(b), "r"(c)
      : "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    u[j] = __hiloint2double(int(r[2 * j + 1]), int(r[2 * j + 0]));
    v[j] = __hiloint2double(int(r[2 * j + 17]), int(r[2 * j + 16]));
    w[j] = __hiloint2double(int(r[2 * j + 33]), int(r[2 * j + 32]));
  }
}

}  // namespace gv
