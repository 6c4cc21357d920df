// What the element kernels share: the reference's face slots, a face node's
// place in its element, block sizes, and the 8-byte asynchronous copy.
#pragma once

#include <cuda_runtime.h>

namespace nekgpu {
namespace {

// face slot f (reference order) -> reference axis 0=r,1=s,2=t, side, and the
// slot it meets in the neighbour
__host__ __device__ constexpr int slot_axis(int f) { return f == 1 || f == 3 ? 0 : (f < 4 ? 1 : 2); }
__host__ __device__ constexpr int slot_side(int f) { return (f == 0 || f == 3 || f == 4) ? -1 : 1; }
__host__ __device__ constexpr int slot_opp(int f) { return f < 4 ? (f + 2) & 3 : 9 - f; }
constexpr int cmax(int a, int b) { return a > b ? a : b; }
constexpr int round32(int a) { return (a + 31) / 32 * 32; }

template <int NX>
__device__ __forceinline__ int face_vol(int f, int a, int b) {
  const int fixed = slot_side(f) < 0 ? 0 : NX - 1;
  const int ax = slot_axis(f);
  return ax == 0 ? fixed + NX * a + NX * NX * b
                 : (ax == 1 ? a + NX * fixed + NX * NX * b : a + NX * b + NX * NX * fixed);
}

// Field component of the k-th partner value of face f: all six with the face
// terms (EXT 2), else H and E along the two axes tangential to f (k = 0, 1: H;
// k = 2, 3: E; lower axis first).
template <int EXT>
__device__ __forceinline__ int partner_comp(int f, int k) {
  if (EXT == 2) return k;
  const int ax = slot_axis(f);
  const int tang = (k & 1) ? (ax == 2 ? 1 : 2) : (ax == 0 ? 1 : 0);
  return (k < 2 ? 0 : 3) + tang;
}

// 8-byte asynchronous global -> shared copies (element blocks whose size is
// not a multiple of 16 bytes, where a bulk copy cannot start on every element)
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

}  // namespace
}  // namespace nekgpu
