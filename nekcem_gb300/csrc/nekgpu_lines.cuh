// Line tasks of the FP64 kernels on affine elements (forward and reverse
// stage): the element arrays' layout in shared memory, the two contraction
// phases' line types, and one line's outputs in fixed point.
#pragma once

#include <cuda_runtime.h>

#include "nekgpu_elem.cuh"
#include "nekgpu_fixed.cuh"
#include "nekgpu_internal.h"

namespace nekgpu {
namespace {

// x with its sign flipped where neg (no FP64 instruction)
__device__ __forceinline__ double flip(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}

template <int NX>
struct ElemCfg {
  static constexpr int N2 = NX * NX, N3 = N2 * NX, NF = 6 * N2;
  // node (i,j,k) of the element arrays at i + RS*j + SZ*k, an odd row length:
  // lines in every direction are read with at most two threads of a half warp
  // on a bank
  static constexpr int RS = NX | 1, SZ = RS * NX, N3P = NX * SZ;
  // threads per block: half a node each, at NX = 5 a whole one (with 96 threads
  // the 125 nodes and 150 lines took a second, nearly empty turn: 336 elements
  // 11.7 against 10.4 us per stage, 1000 20.7 against 17.9, with incident field
  // and PML 128 elements 37.4 against 27.2)
  static constexpr int NT = NX == 9 ? 384 : (NX == 8 ? 256 : (NX == 5 ? 128 : round32(cmax(3 * N2, (N3 + 1) / 2))));
  static constexpr int FPT = (NF + NT - 1) / NT;
};

template <int NX>
__device__ __forceinline__ int pnode(int v) {  // stored index of node v = i + NX*j + NX^2*k
  return (v % NX) + ElemCfg<NX>::RS * ((v / NX) % NX) + ElemCfg<NX>::SZ * (v / (NX * NX));
}

// The line types of the two contraction phases: the first phase adds (or
// starts) one derivative of each of the six residual components, the second
// the other, so a phase has six component-lines per line and one barrier ends
// it.  Residual index 0..2 = H1..H3 (-curl E), 3..5 = E1..E3 (curl H); field
// 0..2 = H, 3..5 = E:
//   E1 = ds Hz - dt Hy   E2 = dt Hx - dr Hz   E3 = dr Hy - ds Hx
//   H1 = dt Ey - ds Ez   H2 = dr Ez - dt Ex   H3 = ds Ex - dr Ey
// slot: the type's place among the four flux components of a face normal to
// its direction.
struct LineType {
  int dir, comp, res, neg, slot;
};
__constant__ const LineType kLine[2][6] = {
    {{0, 1, 5, 0, 0}, {0, 2, 4, 1, 1}, {0, 4, 2, 1, 2}, {0, 5, 1, 0, 3}, {1, 2, 3, 0, 1}, {1, 5, 0, 1, 3}},
    {{1, 0, 5, 1, 0}, {1, 3, 2, 0, 2}, {2, 0, 4, 0, 0}, {2, 1, 3, 1, 1}, {2, 3, 1, 1, 2}, {2, 4, 0, 0, 3}}};

// One line of component lt.comp along lt.dir through (la, lb): outputs
// [i0, i1) of the fixed-point matrix go to put(i, x).  SPLIT takes the rows of
// the matrix from shared memory (any range of outputs) instead of the
// constant bank (all NX of them).
template <int NX, bool SPLIT, typename Put>
__device__ __forceinline__ void line_outputs(const double* pu, int step, int i0, int i1,
                                             const FixedD& fd, const double* D, const int2* s_D,
                                             Put put) {
  FixedLine<NX> f;
  {
    double u[NX];
#pragma unroll
    for (int l = 0; l < NX; ++l) u[l] = pu[step * l];
    fixed_line<NX>(u, fd.maxexp, f);
  }
  if (fd.ok && !f.special) {
    if (!SPLIT) {
#pragma unroll
      for (int i = 0; i < NX; ++i)
        put(i, fixed_dot<NX>(f, fd.bias, [&](int l, int& hi, int& lo) {
              hi = fd.hi[i + NX * l];
              lo = fd.lo[i + NX * l];
            }));
    } else {
#pragma unroll 1
      for (int i = i0; i < i1; ++i)
        put(i, fixed_dot<NX>(f, fd.bias, [&](int l, int& hi, int& lo) {
              const int2 d = s_D[i + NX * l];
              hi = d.x;
              lo = d.y;
            }));
    }
  } else {  // a line out of the integer form's range: in FP64
#pragma unroll 1
    for (int i = i0; i < i1; ++i) {
      double x = D[i] * pu[0];
#pragma unroll 1
      for (int l = 1; l < NX; ++l) x = fma(D[i + NX * l], pu[step * l], x);
      put(i, x);
    }
  }
}

}  // namespace
}  // namespace nekgpu
