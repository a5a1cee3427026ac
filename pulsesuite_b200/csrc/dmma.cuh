// dmma.cuh -- FP64 matrix instructions (mma.sync m8n8k4) for the full-matrix
// kernels, sm_100a.  Per SM they sustain 64 FMAs a clock, as the scalar FMAs
// do at best, from one operand pair per eight FMAs of a lane.
#pragma once

#include <stdint.h>

namespace psb {

// c (8 x 8) += a (8 x 4) b (4 x 8): lane l holds a[l / 4][l % 4], b[l % 4][l / 4]
// and c[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
__device__ __forceinline__ double flip(double x) {
  return __hiloint2double(__double2hiint(x) ^ 0x80000000, __double2loint(x));
}
__device__ __forceinline__ double2 neg(double2 a) { return make_double2(flip(a.x), flip(a.y)); }

// complex accumulator (re, im) of one 8 x 8 tile: += a b, or += conj(a) b
struct CAcc {
  double re[2], im[2];
};
template <bool CONJ>
__device__ __forceinline__ void cmma(CAcc& c, double2 a, double2 b) {
  dmma(c.re, a.x, b.x);
  dmma(c.re, CONJ ? a.y : flip(a.y), b.y);
  dmma(c.im, a.x, b.y);
  dmma(c.im, CONJ ? flip(a.y) : a.y, b.x);
}

// 16 bytes to shared memory, zero when !in (src is then not read)
__device__ __forceinline__ void cp16(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace psb
