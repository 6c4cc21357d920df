// Fixed-point contractions of one GLL line with the derivative matrix, at
// FP64 accuracy without FP64 instructions.
//
// GB300 issues two FP64 lanes per clock and SM but 32 lanes of 32x32+64-bit
// integer multiply-add (measured: DFMA 2.0, IMAD.WIDE 30, I2F.F64.S64 about
// 16 lanes per clock and SM), so a line of FP64 values is scaled to integers
// by its largest exponent and contracted in integer arithmetic:
//
//   u_l = Q_l 2^(E-1083),  |Q_l| < 2^61, Q_l = h_l 2^31 + l_l with h_l rounded to
//         nearest (|h_l|, |l_l| <= 2^30), E the largest biased exponent of the
//         line: exact for every value down to 2^-8 of the line's largest,
//         truncated below 2^-61 of it otherwise;
//   D(i,l) = P_il 2^-kd, |P_il| <= 2^61, in the same two limbs H, L: exact down
//         to entries of 2^-8 of the largest, rounded otherwise;
//   sum_l D(i,l) u_l = [ sum h H + sum (h L + l H) 2^-31 ] 2^62 2^(E-1083-kd)
//         + sum l L 2^(E-1083-kd): the last sum is dropped, the two others are
//         exact 64-bit integer sums (the host checks the row sums of D:
//         fixed_table); the second joins the first rounded, and the total is
//         rounded once to FP64.
//
// Before that last rounding an output differs from the exact sum by less than
//   (NX + 1)/2 + sum_l |P_il| 2^-62   units of 2^62 2^(E-1083-kd)
// (the dropped sum and P's rounding NX/4 each, the join 1/2, u's truncation
// the rest), a unit being at most 2^-58 of the line's largest value times the
// largest entry of D where kd is the first one tried.  Root mean squares over
// outputs, last rounding included, in units of 2^-57 max|u| max|D|, against
// exact sums (in parentheses the FP64 multiply-add chain), N=7: random lines,
// ends 5.1 (10.9), interior 1.0 (2.0); smooth 0.5 (4.3), 0.5 (1.2); nearly
// constant 0.1 (5.5), 0.1 (1.0).  The same order of the two at N=3 to 8; at N=2,
// and on lines with one value far above the others, the interior's are equal
// within a few per cent.  With limbs truncated and 59 bits a factor the
// interior's were 4.1, 3.1 and 2.8, above the chain's.  The error is relative to
// the line's largest value: where D's entry of that value is zero (the
// diagonal, inside) a chain of much smaller values would keep their own
// relative accuracy.
//
// A line that holds an infinity, a NaN or a value above 2^1006 (with a D of
// large entries less: FixedD::maxexp, so that no output's exponent leaves
// FP64's range) or lies below 2^-823 as a whole, and a D that does not fit the
// table (FixedD::ok), is contracted in FP64 instead, term by term.
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
    const unsigned long long q = shr64(m, (unsigned)(f.E + 3) - ((hi >> 20) & 0x7FFu));
    const int ql = (int)((unsigned)q << 1) >> 1;  // the low 31 bits as a signed number
    const int s = ((int)hi >> 31) | 1;
    f.h[k] = ((int)(q >> 31) - (ql >> 31)) * s;
    f.l[k] = ql * s;
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

// sum_l P_l u_l with P_l = hi 2^31 + lo given by get(l, hi, lo)
template <int NX, typename Get>
__device__ __forceinline__ double fixed_dot(const FixedLine<NX>& f, int bias, Get get) {
  int hi[NX], lo[NX];
#pragma unroll
  for (int l = 0; l < NX; ++l) get(l, hi[l], lo[l]);
  long long b = 1 << 30;  // rounds the shift
#pragma unroll
  for (int l = 0; l < NX; ++l) {
    b += (long long)f.h[l] * lo[l];
    b += (long long)f.l[l] * hi[l];
  }
  b >>= 31;
#pragma unroll
  for (int l = 0; l < NX; ++l) b += (long long)f.h[l] * hi[l];
  return fixed_join(b, f.E - bias);
}

}  // namespace
}  // namespace nekgpu
