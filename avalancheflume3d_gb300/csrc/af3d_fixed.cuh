// af3d_fixed.cuh -- the fast mode's rotation update and sphere centres in 64-bit fixed point.
//
// The FP64 unit retires one warp instruction in 64 to 76 cycles (af3d_intfp64.cuh), and the
// rotation of a clump by its step's angle, the renormalisation of the rotation's columns and
// the four sphere centres took 96 of the fast predictor's 123 FP64 instructions.  A step turns a
// clump by ~10^-4 rad, so R' = R + (dR - 1) R is R plus a small term: in integers of 2^-62 the
// term's error is below 2^-60 and the one rounding that counts is the last one, to double.  The
// results are at least as close to the exact ones as the FP64 formulas' (tests/test_fixed.py).
#pragma once

#include "af3d_intfp64.cuh"

namespace af3d {

#ifdef __CUDACC__
#define AF3D_HD __device__ __forceinline__
AF3D_HD long long mulhi_ll(long long a, long long b) { return __mul64hi(a, b); }
AF3D_HD int leading_zeros(unsigned long long x) { return __clzll((long long)x); }
#else
#define AF3D_HD inline
inline long long mulhi_ll(long long a, long long b) { return (long long)((__int128)a * b >> 64); }
inline int leading_zeros(unsigned long long x) { return x ? __builtin_clzll(x) : 64; }
#endif

// x 2^q to the nearest integer, |x| < 2^(62 - q).
AF3D_HD long long fixed_of(double x, int q) {
  const unsigned long long b = bits_of(x);
  const int e = (int)((b >> 52) & 0x7FFull);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 1ull << 52;
  const int sh = 1075 - q - e;   // the shift to the right
  unsigned long long v;
  if (sh > 0) v = sh > 63 ? 0ull : ((m >> (sh - 1)) + 1ull) >> 1;
  else v = m << -sh;
  return (long long)b < 0 ? -(long long)v : (long long)v;
}

// v 2^-q to the nearest double (normal results).
AF3D_HD double double_of(long long v, int q) {
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int z = leading_zeros(a);
  if (z == 64) return 0.0;
  const unsigned long long n = a << z;
  const unsigned long long m = (n >> 11) + ((n >> 10) & 1ull);   // 53 bits with the leading one, or 2^53
  const unsigned long long r = ((unsigned long long)(unsigned)(1085 - z - q) << 52) + m;   // the one adds to the exponent
  return of_bits(r | ((unsigned long long)v & 0x8000000000000000ull));
}

// dR - 1 of a turn by the angle vector w, |w| < 2^-10, in Q72, each entry as 2^32 hi + lo with both
// halves signed: -(1/2 - t/24) (t 1 - w w^T) + (1 - t/6 + t^2/120) [w]x, t = |w|^2 (Rodrigues'
// matrix by its Maclaurin series; the first omitted terms are below 2^-62).
struct Turn {
  int hi[9], lo[9];
};

// False for a larger angle, which the FP64 formulas take.
AF3D_HD bool turn_fixed(const double *w, Turn &turn) {
  bool small = true;
#pragma unroll
  for (int i = 0; i < 3; i++) small = small && ((bits_of(w[i]) >> 52) & 0x7FFull) < 1013ull;   // |w_i| < 2^-10
  if (!small) return false;
  long long x[3];
#pragma unroll
  for (int i = 0; i < 3; i++) x[i] = fixed_of(w[i], 72);
  long long tt = 0;   // t in Q80
#pragma unroll
  for (int i = 0; i < 3; i++) tt += (x[i] >> 32) * (x[i] >> 32);
  if (tt >> 60) return false;
  const unsigned t = (unsigned)(tt >> 28);   // Q52
  const unsigned t6 = mulhi_u(t, 0x2AAAAAABu) - mulhi_u(mulhi_u(t, t) >> 20, 0x02222222u), t12 = mulhi_u(t, 0x15555555u);
  auto half_product = [&](long long a, long long b) {   // (1/2 - t/24) a b in Q72
    const long long p = mulhi_ll(a, b) >> 9;
    return p - ((long long)(int)(p >> 20) * (long long)t12 >> 32);
  };
  const long long xx = half_product(x[0], x[0]), yy = half_product(x[1], x[1]), zz = half_product(x[2], x[2]),
                  xy = half_product(x[0], x[1]), xz = half_product(x[0], x[2]), yz = half_product(x[1], x[2]);
  long long s[3];
#pragma unroll
  for (int i = 0; i < 3; i++) s[i] = x[i] - ((x[i] >> 32) * (long long)t6 >> 20);
  const long long D[9] = {-(yy + zz), xy - s[2], xz + s[1], xy + s[2], -(xx + zz), yz - s[0],
                          xz - s[1], yz + s[0], -(xx + yy)};
#pragma unroll
  for (int i = 0; i < 9; i++) {
    turn.hi[i] = (int)((D[i] + 0x80000000ll) >> 32);
    turn.lo[i] = (int)D[i];
  }
  return true;
}

// Column j of the turned rotation, renormalised, in units of 2^-62, from the column R.  An exact
// rotation keeps its norm, so what is renormalised is the rounding left by the step before: R_i -
// R_i (|R|^2 - 1) / 2.  False when the squared norm is further than 2^-29 from one (a state read
// from text), which the FP64 formulas take.
AF3D_HD bool column_fixed(const Turn &turn, const double *R, long long *out) {
  bool small = true;
#pragma unroll
  for (int i = 0; i < 3; i++) small = small && ((bits_of(R[i]) >> 52) & 0x7FFull) < 1024ull;   // |R_i| < 2
  if (!small) return false;
  long long f[3];
  int rh[3], rl[3];
  long long norm = -(1ll << 60);   // |R|^2 - 1 in Q60
#pragma unroll
  for (int i = 0; i < 3; i++) {
    f[i] = fixed_of(R[i], 62);
    rh[i] = (int)((f[i] + 0x80000000ll) >> 32);
    rl[i] = (int)f[i];
    norm += mulhi_ll(f[i], f[i]);
  }
  if (norm >= 0x7FFFFFFFll || norm <= -0x7FFFFFFFll) return false;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    long long acc = 0;   // sum over k of D_ik R_k in Q70
    int low = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      acc += (long long)turn.hi[3 * i + k] * rh[k];
      low += mulhi_s(turn.hi[3 * i + k], rl[k]) + mulhi_s(turn.lo[3 * i + k], rh[k]);
    }
    out[i] = f[i] + ((acc + low + 128) >> 8) - ((long long)rh[i] * (long long)(int)norm >> 29);
  }
  return true;
}

// The rotation rows R (row-major) turned by w and renormalised, in units of 2^-62.
AF3D_HD bool rotate_fixed(const double *w, const double *R, long long *out) {
  Turn turn;
  if (!turn_fixed(w, turn)) return false;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const double col[3] = {R[j], R[3 + j], R[6 + j]};
    long long c[3];
    if (!column_fixed(turn, col, c)) return false;
#pragma unroll
    for (int i = 0; i < 3; i++) out[3 * i + j] = c[i];
  }
  return true;
}

// Whether spheres_fixed takes a clump: pos < 2^(60 - q), and coordinates whose units fit.
AF3D_HD bool spheres_fit(const double *r, double pos, int q) {
  bool fits = ((bits_of(pos) >> 52) & 0x7FFull) < (unsigned long long)(1023 + 60 - q);
#pragma unroll
  for (int i = 0; i < 3; i++) fits = fits && ((bits_of(r[i]) >> 52) & 0x7FFull) < (unsigned long long)(1082 - q + 60);
  return fits;
}

// One coordinate of the four sphere centres r + pos R (1,1,1), (1,-1,-1), (-1,-1,1), (-1,1,-1)
// (init_Verlet.cu:130-142) from the row R in units of 2^-62, rounded once.  The offsets are formed
// in units of 2^-q and added to r in units 2^-8 of its last place or finer.
AF3D_HD void spheres_row_fixed(const long long *R, double r, double pos, int q, double *s) {
  const long long p = fixed_of(pos, q) << 2;   // mulhi(p, Q62) is in Q(q)
  const int e = (int)((bits_of(r) >> 52) & 0x7FFull);
  const int qi = q < 1082 - e ? q : 1082 - e, sh = q - qi;   // |r| and the sums below 2^62 units
  const long long a = mulhi_ll(p, R[0] + R[1]), b = mulhi_ll(p, R[0] - R[1]), c = mulhi_ll(p, R[2]);
  const long long o = fixed_of(r, qi);
  s[0] = double_of(o + ((c + a) >> sh), qi);
  s[1] = double_of(o + ((b - c) >> sh), qi);
  s[2] = double_of(o + ((c - a) >> sh), qi);
  s[3] = double_of(o - ((b + c) >> sh), qi);
}

// The four sphere centres (s[3 k + i]); false when r or pos does not fit.
AF3D_HD bool spheres_fixed(const long long *R, const double *r, double pos, int q, double *s) {
  if (!spheres_fit(r, pos, q)) return false;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    double c[4];
    spheres_row_fixed(R + 3 * i, r[i], pos, q, c);
#pragma unroll
    for (int k = 0; k < 4; k++) s[3 * k + i] = c[k];
  }
  return true;
}

#undef AF3D_HD
}  // namespace af3d
