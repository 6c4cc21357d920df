// Fixed-point contractions of one GLL line with the derivative matrix, at
// FP64 accuracy without FP64 instructions.
//
// GB300 issues two FP64 lanes per clock and SM but 32 lanes of 32x32+64-bit
// integer multiply-add (measured: DFMA 2.0, IMAD.WIDE 30, I2F.F64.S64 about
// 16 lanes per clock and SM), so a line of FP64 values is scaled to integers
// by its largest exponent and contracted in integer arithmetic:
//
//   u_l = Q_l 2^(E-1081),  |Q_l| < 2^59, Q_l = h_l 2^31 + l_l (both limbs
//         carry u_l's sign, |h_l| < 2^28, |l_l| < 2^31), E the largest biased
//         exponent of the line: exact for every value down to 2^-6 of the
//         line's largest, truncated below 2^-58 of it otherwise;
//   D(i,l) = P_il 2^-kd, |P_il| < 2^59, the same two limbs: exact down to
//         entries of 2^-6 of the largest;
//   sum_l D(i,l) u_l = [ sum h H 2^62 + sum (h L + l H) 2^31 + (sum l L) ]
//         2^(E-1081-kd): the last sum (below 2^-58 of the largest term) is
//         dropped, the two others are exact 64-bit integer sums (the host
//         checks the row sums of D: fixed_table) and join as
//         sum h (8 H) + ((sum (h L + l H)) >> 28) in units of 2^59, rounded
//         once to FP64.
//
// Every error is below 2^-57 of the line's largest value times the largest
// entry of D, against about 2^-53 for each step of an FP64 sum.  A line that
// holds an infinity, a NaN or a value above 2^1006 (with a D of large entries
// less: FixedD::maxexp, so that no output's exponent leaves FP64's range) or
// lies below 2^-823 as a whole, and a D that does not fit the table
// (FixedD::ok), is contracted in FP64 instead, term by term.
#pragma once

#include <cuda_runtime.h>

#include "nekgpu_internal.h"

namespace nekgpu {
namespace {

// Q of the value u under the line's exponent E (a logical 64-bit shift that
// gives 0 from 64 on)
__device__ __forceinline__ unsigned long long shr64(unsigned long long v, unsigned s) {
  unsigned long long r;
  asm("shr.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}


template <int NX>
struct FixedLine {
  int h[NX], l[NX];
  int E;         // biased exponent the line is scaled by
  bool special;  // contract in FP64
};

// maxexp: FixedD::maxexp
template <int NX>
__device__ __forceinline__ void fixed_line(const double* u, int maxexp, FixedLine<NX>& f) {
  unsigned em = 0;
#pragma unroll
  for (int k = 0; k < NX; ++k) em = max(em, (unsigned)__double2hiint(u[k]) & 0x7FFFFFFFu);
  f.E = max((int)(em >> 20), kFixedMinExp);  // (a line of zeros: any exponent)
  f.special = (em > 0 && em < ((unsigned)kFixedMinExp << 20)) || f.E >= maxexp;
#pragma unroll
  for (int k = 0; k < NX; ++k) {
    const unsigned hi = (unsigned)__double2hiint(u[k]), lo = (unsigned)__double2loint(u[k]);
    // the 53-bit significand at the top of 64 bits, then down to the line's
    // scale (a zero or subnormal value's exponent field is 0: shifted out)
    const unsigned mh = __funnelshift_l(lo, hi, 11) | 0x80000000u;
    const unsigned long long m = ((unsigned long long)mh << 32) | (lo << 11);
    const unsigned long long q = shr64(m, (unsigned)(f.E + 5) - ((hi >> 20) & 0x7FFu));
    const int s = (int)hi >> 31;
    f.h[k] = ((int)(q >> 31) ^ s) - s;
    f.l[k] = ((int)((unsigned)q & 0x7FFFFFFFu) ^ s) - s;
  }
}

// b 2^(E - bias) rounded to FP64, |b| < 2^63, by integer operations: the
// conversion instruction from 64-bit integers takes an FP64-pipe slot per
// output, 12 per node (16^3 box at N=7: 311 us per stage with it, 277 with
// this form).  Ties round away from zero.
__device__ __forceinline__ double fixed_join(long long b, int e) {
  const long long s = b >> 63;
  const unsigned long long mag = (unsigned long long)((b ^ s) - s);
  const int n = __clzll((long long)mag);
  // 53 bits in [2^52, 2^53]: the leading bit adds one to the exponent field
  const unsigned long long m = ((mag << (n - 1)) + 0x200u) >> 10;
  const unsigned hi = (unsigned)(m >> 32) + ((unsigned)(1085 - n + e) << 20);
  return __hiloint2double((int)((mag ? hi : 0u) | ((unsigned)(s >> 32) & 0x80000000u)), (int)(unsigned)m);
}

// sum_l P_l u_l with P_l = hi 2^31 + lo, hi8 = 8 hi given by get(l, hi, lo, hi8)
template <int NX, typename Get>
__device__ __forceinline__ double fixed_dot(const FixedLine<NX>& f, int bias, Get get) {
  int hi[NX], lo[NX], hi8[NX];
#pragma unroll
  for (int l = 0; l < NX; ++l) get(l, hi[l], lo[l], hi8[l]);
  long long b = 0;
#pragma unroll
  for (int l = 0; l < NX; ++l) {
    b += (long long)f.h[l] * lo[l];
    b += (long long)f.l[l] * hi[l];
  }
  b >>= 28;
#pragma unroll
  for (int l = 0; l < NX; ++l) b += (long long)f.h[l] * hi8[l];
  return fixed_join(b, f.E - bias);
}

}  // namespace
}  // namespace nekgpu
