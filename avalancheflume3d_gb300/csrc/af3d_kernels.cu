// af3d_kernels.cu -- the step kernels (compiled with -fmad=false: see af3d_physics.cuh).
//
// Kernels, per step of the fused path (af3d_step):
//   k_predict      init_Verlet (+ cell key, bucket count)              one thread per clump
//   (cells)        scan of bucket counts, scatter, deterministic rank  af3d_cells.cu
//   k_permute      move every plane into (cell, id) order, build the packed neighbour records
//   (near lists)   what may touch within the next steps             af3d_near.cu
//   k_lists_forces each block takes its clumps' contact items from their near lists, then runs
//                  boundaries + sphere contacts + bed + get_accel + finish_Verlet for them,
//                  gathering (never scattering) contributions: no atomics on forces; and the next
//                  step's predictor.  The sort, the permutation and the lists run every few
//                  steps only: the other steps are this one kernel
// The per-routine C-ABI entry points use k_boundary / k_part / k_get_accel / k_finish_verlet,
// which apply the same device functions to the F, T planes one routine at a time.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "af3d_cellwalk.cuh"
#include "af3d_fixed.cuh"

namespace af3d {

namespace {

constexpr int kBlock = 128;   // the per-clump kernels other than the fused force kernel

inline unsigned grid_for(long n, int block = kBlock) {
  return (unsigned)((n + block - 1) / block);
}

__device__ __forceinline__ V3 load3(const Planes &P, int x, long s) {
  return mk(P.p[x][s], P.p[x + 1][s], P.p[x + 2][s]);
}
__device__ __forceinline__ void store3(const Planes &P, int x, long s, V3 v) {
  P.p[x][s] = v.x;
  P.p[x + 1][s] = v.y;
  P.p[x + 2][s] = v.z;
}

__device__ __forceinline__ void raise_status(DevScalars *d, int err) {
  atomicOr(&d->status, 1 << err);
}

// ------------------------------------------------------------------ import / export

// keep_order: slot s keeps the clump it holds (id[s]); otherwise slot s receives clump s.
__global__ void k_aos_to_planes(const af3d_particle *__restrict__ aos, const double *__restrict__ acc,
                                const double *__restrict__ anga, const int *__restrict__ flume_of_id,
                                Planes P, long long *id, int *flume, bool keep_order, long s0, long n) {
  long s = s0 + blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const long long i = keep_order ? id[s] : s;
  const af3d_particle q = aos[i];   // every load before the first store, which might alias
  V3 a = acc ? mk(acc[3 * i], acc[3 * i + 1], acc[3 * i + 2]) : mk(0.0, 0.0, 0.0);
  V3 al = anga ? mk(anga[3 * i], anga[3 * i + 1], anga[3 * i + 2]) : mk(0.0, 0.0, 0.0);
  const int f = flume_of_id[i];
  store3(P, RX, s, mk(q.rr.x, q.rr.y, q.rr.z));
  store3(P, VX, s, mk(q.vv.x, q.vv.y, q.vv.z));
  store3(P, WX, s, mk(q.ww.x, q.ww.y, q.ww.z));
  store3(P, R00, s, mk(q.Rmatx.x, q.Rmatx.y, q.Rmatx.z));
  store3(P, R10, s, mk(q.Rmaty.x, q.Rmaty.y, q.Rmaty.z));
  store3(P, R20, s, mk(q.Rmatz.x, q.Rmatz.y, q.Rmatz.z));
  for (int k = 0; k < 4; k++) store3(P, S0X + 3 * k, s, mk(q.rr_s[k].x, q.rr_s[k].y, q.rr_s[k].z));
  store3(P, AIX, s, a);
  store3(P, ALIX, s, al);
  store3(P, AFX, s, mk(0.0, 0.0, 0.0));
  store3(P, ALFX, s, mk(0.0, 0.0, 0.0));
  store3(P, FX, s, mk(0.0, 0.0, 0.0));
  store3(P, TX, s, mk(0.0, 0.0, 0.0));
  const double r = q.radius, rho = q.density;
  P.p[RAD][s] = r;
  P.p[DEN][s] = rho;
  P.p[MASS][s] = q.mass;
  store3(P, IXX, s, mk(q.moment_of_inertia.x, q.moment_of_inertia.y, q.moment_of_inertia.z));
  P.p[MSPH][s] = kSPH_FACT * rho * r * r * r;   // force_part.cu:58
  P.p[MWALL][s] = kSPH_FACT * r * r * r * rho;  // force_walls.cu:47
  P.p[ADRAG][s] = drag_factor(r, q.mass);       // get_accel.cu:47
  P.p[IMASS][s] = 1.0 / q.mass;
  P.p[IINER][s] = 1.0 / q.moment_of_inertia.x;
  id[s] = i;
  flume[s] = f;
}

// Bound by latency at the counts of one part of a host step: with the planes loaded between the
// stores, which might alias them, the loads came one group after another (25,000 clumps: 18 us, now
// 15).
__global__ void k_planes_to_aos(Planes P, const long long *__restrict__ id, const int *__restrict__ flume,
                                af3d_particle *aos, double *acc, double *anga, const DevScalars *d,
                                long s0, long n) {
  long s = s0 + blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const af3d_system_par &sy = d->flumes[flume[s]].sys;
  const double cost = sy.cost, sint = sy.sint;
  const long long i = id[s];
  af3d_particle q;
  V3 ai, al;
  if (acc) ai = load3(P, AIX, s);
  if (anga) al = load3(P, ALIX, s);
  q.radius = P.p[RAD][s];
  q.mass = P.p[MASS][s];
  q.density = P.p[DEN][s];
  V3 I = load3(P, IXX, s);
  q.moment_of_inertia = {I.x, I.y, I.z};
  V3 r = load3(P, RX, s);
  q.rr = {r.x, r.y, r.z};
  V3 rr = to_slope(r, cost, sint);
  q.rrot = {rr.x, rr.y, rr.z};
  for (int k = 0; k < 4; k++) {
    V3 sk = load3(P, S0X + 3 * k, s);
    q.rr_s[k] = {sk.x, sk.y, sk.z};
    V3 qk = to_slope(sk, cost, sint);
    q.rrot_s[k] = {qk.x, qk.y, qk.z};
  }
  V3 v = load3(P, VX, s), w = load3(P, WX, s);
  q.vv = {v.x, v.y, v.z};
  q.ww = {w.x, w.y, w.z};
  V3 a = load3(P, R00, s), b = load3(P, R10, s), c = load3(P, R20, s);
  q.Rmatx = {a.x, a.y, a.z};
  q.Rmaty = {b.x, b.y, b.z};
  q.Rmatz = {c.x, c.y, c.z};
  aos[i] = q;
  if (acc) {
    acc[3 * i] = ai.x; acc[3 * i + 1] = ai.y; acc[3 * i + 2] = ai.z;
  }
  if (anga) {
    anga[3 * i] = al.x; anga[3 * i + 1] = al.y; anga[3 * i + 2] = al.z;
  }
}

// ------------------------------------------------------------------ neighbour records

__device__ __forceinline__ float f_up(double x) { return to_float_ru(x); }

// x in units of 2^-qs, truncated, modulo 2^32 (|x| below 2^50 units: make_records), from the bits
// of the double: the 53-bit mantissa shifted into place.
__device__ __forceinline__ int to_units(double x, int qs) {
  const unsigned long long b = bits_of(x);
  const int e = (int)((b >> 52) & 0x7FFull);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 1ull << 52;   // (a subnormal shifts out anyway)
  const int sh = 1075 - qs - e;
  const unsigned v = sh > 63 ? 0u : (unsigned)(m >> max(sh, 0));
  return (long long)b < 0 ? (int)(0u - v) : (int)v;
}

// Packed FP64 neighbour record and conservative culling record of one clump.
// The centre test's bound covers the FP32 rounding of the centres.  M32 = max |coordinate| in FP32
// is within 2^-24 of the FP64 maximum M, so mu = 2^-22 * M32 * (1 + 2^-20) is at least 4 x 2^-24
// M: the FP32 difference of a coordinate of this clump and one of a partner is within 2^-24 (M +
// M') (the two roundings) + 2^-24 |difference| of the exact one, so a distance formed from FP32
// coordinates errs by at most sqrt(3) 2^-24 (M + M') + 2^-24 d < mu + mu' + 2^-24 d, and the last
// term is covered by the tests' relative slack (1 + 2^-18) on squared bounds.  The sphere extent
// max_k |s_k - r| is formed in units: each difference of truncated coordinates is within 2 units
// of the exact one, so the extent within 2 sqrt(3) and its FP32 rounding, which the 4 units and
// the factor (1 + 2^-20) cover.
__device__ __forceinline__ void make_records(V3 r, V3 v, V3 w, const V3 *sp, double rad, double msph,
                                             double mwall, Margins m, int key, NbrRec &q, CullRec &c) {
  q.rx = r.x; q.ry = r.y; q.rz = r.z;
  q.vx = v.x; q.vy = v.y; q.vz = v.z;
  q.wx = w.x; q.wy = w.y; q.wz = w.z;
  for (int k = 0; k < 4; k++) {
    q.s[3 * k] = sp[k].x; q.s[3 * k + 1] = sp[k].y; q.s[3 * k + 2] = sp[k].z;
  }
  q.rad = rad; q.msph = msph; q.mwall = mwall;
  const float cx = to_float_rn(r.x), cy = to_float_rn(r.y), cz = to_float_rn(r.z);
  const float radf = f_up(rad);
  const int qi = m.qs;
  const int ux = to_units(r.x, qi), uy = to_units(r.y, qi), uz = to_units(r.z, qi);
  float ext2 = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int x = to_units(sp[k].x, qi), y = to_units(sp[k].y, qi), z = to_units(sp[k].z, qi);
    const float dx = (float)(x - ux), dy = (float)(y - uy), dz = (float)(z - uz);
    ext2 = fmaxf(ext2, __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)));
    c.s[k].x = x; c.s[k].y = y; c.s[k].z = z;
  }
  const float unit = unit_power(-qi), units = unit_power(qi);
  const float extu = sqrtf(ext2) * (1.0f + 9.5367431640625e-07f) + 4.0f;
  float radu = radf * units * (1.0f + 9.5367431640625e-07f) + 2.0f;
  float ext = extu * unit;
  const float M = fmaxf(fmaxf(fabsf(cx), fabsf(cy)), fabsf(cz));
  // A clump too large for the unit, or so far out that its coordinates do not fit the shifts: its
  // extent from the FP32 coordinates, and an infinite radius in the sphere tests.
  if (!(extu + radu <= kCullMaxUnits && (M + 4.0f * kCullMaxUnits * unit) * units <= 1.125899906842624e+15f)) {
    float far2 = 0.0f, most = M;
    for (int k = 0; k < 4; k++) {
      const float x = to_float_rn(sp[k].x), y = to_float_rn(sp[k].y), z = to_float_rn(sp[k].z);
      most = fmaxf(most, fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)));
      const float dx = x - cx, dy = y - cy, dz = z - cz;
      far2 = fmaxf(far2, __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)));
    }
    ext = sqrtf(far2) * (1.0f + 9.5367431640625e-07f) + most * 4.76837158203125e-07f;
    radu = __int_as_float(0x7F800000);
  }
  // 2^-22 * max|coordinate|: see above.
  const float mu = fmaxf(M, radf) * 2.384185791015625e-07f * (1.0f + 9.5367431640625e-07f) + 1e-30f;
  const float bound = (ext * (1.0f + 9.5367431640625e-07f) + 2.0f * mu) + (radf * (1.0f + 9.5367431640625e-07f) + mu);
  c.c = make_float4(cx, cy, cz, bound);
  for (int k = 0; k < 4; k++) c.s[k].w = __float_as_int(radu);
  c.key = key;
  // no sphere moves faster than |v| + |w| bound
  const float vx = magnitude_f(v.x), vy = magnitude_f(v.y), vz = magnitude_f(v.z);
  const float wx = magnitude_f(w.x), wy = magnitude_f(w.y), wz = magnitude_f(w.z);
  const float speed = sqrtf(vx * vx + vy * vy + vz * vz) + sqrtf(wx * wx + wy * wy + wz * wz) * bound;
  c.pace = m.per_speed * speed;
  c.allow = fminf(c.pace + m.floor, m.cap);   // cap for NaN
  c.away = 0;
}

// How far the spheres of a clump moved between two of its records, at most, in cm.  Differences
// of truncated coordinates: within 2 units each, covered by the 4 units; a step longer than 2^31
// units leaves the grid.
__device__ __forceinline__ float sphere_motion(const int4 *from, const CullRec &to, int qs) {
  float d2 = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float dx = (float)(to.s[k].x - from[k].x), dy = (float)(to.s[k].y - from[k].y),
                dz = (float)(to.s[k].z - from[k].z);
    d2 = fmaxf(d2, __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)));
  }
  return (sqrtf(d2) * (1.0f + 9.5367431640625e-07f) + 4.0f) * unit_power(-qs);
}

constexpr int kPermBlock = 128;
// Records are staged in shared memory with an odd stride (25 doubles) so that the per-thread
// writes of a 24-double record hit distinct banks.
constexpr int kRecWords = (int)(sizeof(NbrRec) / 8);   // 24
constexpr int kRecStride = kRecWords + 1;

// One thread's neighbour record into the block's shared-memory staging.
__device__ __forceinline__ void stage_nbr_record(const NbrRec &q, double *s_nbr) {
  const double *qw = reinterpret_cast<const double *>(&q);
#pragma unroll
  for (int k = 0; k < kRecWords; k++) s_nbr[threadIdx.x * kRecStride + k] = qw[k];
}

// One thread's records into the block's shared-memory staging.
__device__ __forceinline__ void stage_record(const NbrRec &q, const CullRec &cr, double *s_nbr, CullRec *s_cull) {
  stage_nbr_record(q, s_nbr);
  s_cull[threadIdx.x] = cr;
}

// The block's staged neighbour records written out as contiguous 16-byte stores (after a
// barrier that follows the staging).
template <int NB>
__device__ __forceinline__ void copy_nbr_records(long base, long n, NbrRec *nbr, const double *s_nbr) {
  const long cnt = n - base < NB ? n - base : NB;
  const int nw = (int)(cnt * kRecWords) / 2;   // double2 words of the block's records
  double2 *b = reinterpret_cast<double2 *>(nbr + base);
  for (int i = threadIdx.x; i < nw; i += NB) {
    const int w0 = 2 * i, r0 = w0 / kRecWords, k0 = w0 - r0 * kRecWords;   // k0 even, k0 + 1 < 24
    b[i] = make_double2(s_nbr[r0 * kRecStride + k0], s_nbr[r0 * kRecStride + k0 + 1]);
  }
}

// ... and the culling records with them.
template <int NB>
__device__ __forceinline__ void copy_records(long base, long n, NbrRec *nbr, CullRec *cull, const double *s_nbr,
                                             const CullRec *s_cull) {
  copy_nbr_records<NB>(base, n, nbr, s_nbr);
  const long cnt = n - base < NB ? n - base : NB;
  const int m16 = (int)(cnt * (long)(sizeof(CullRec) / 16));
  const float4 *c = reinterpret_cast<const float4 *>(s_cull);
  float4 *e = reinterpret_cast<float4 *>(cull + base);
  for (int i = threadIdx.x; i < m16; i += NB) e[i] = c[i];
}

// The block's records, staged in shared memory and written out as contiguous 16-byte stores.
// Every thread of an NB-thread block calls this (slots past n contribute nothing).
template <int NB>
__device__ __forceinline__ void store_records(bool valid, long base, long n, const NbrRec &q, const CullRec &cr,
                                              NbrRec *nbr, CullRec *cull, double *s_nbr, CullRec *s_cull) {
  if (valid) stage_record(q, cr, s_nbr, s_cull);
  __syncthreads();
  copy_records<NB>(base, n, nbr, cull, s_nbr, s_cull);
}

// ------------------------------------------------------------------ init_Verlet (+ cell keys)

// Cell coordinate of cells.cu:69-77 (multiplication by cs_inv, then `== ncell -> ncell-1`).
__device__ __forceinline__ long bin_axis(double x, double xmin, double inv, long n) {
  long i = (long)trunc_to_ll(inv * (x - xmin));
  if (i == n) i--;
  return i;
}

// The same from the FP32 rounding of x and the FP32 grid copies where that is certain (the
// estimate of search_axis_f, which lies on the same side of every integer as the FP64 product).
__device__ __forceinline__ long bin_axis_f(double x, float xminf, float invf, double xmin, double inv, long n) {
  const float xf = to_float_rn(x);
  const float q = (xf - xminf) * invf;
  const float E = 4.76837158203125e-07f * ((fabsf(xf) + fabsf(xminf)) * invf + 3.0f * q);   // 2^-21 (...)
  if (q > E && q < 4.0e6f) {
    const float tq = truncf(q), fr = q - tq;
    if (fr > E && fr < 1.0f - E) {
      const long i = (long)(int)tq;
      return i == n ? i - 1 : i;
    }
  }
  return bin_axis(x, xmin, inv, n);
}

constexpr bool kCall = !kFast;   // k_lists_forces calls its quotients (af3d_physics.cuh)

constexpr double kSmallAngle2 = 9.765625e-04;   // (2^-5)^2

// sin t and cos t of a rotation angle t >= 0 with t2 = t^2 (rounded).  Below 2^-5 rad (a step of
// 2e-6 s turns a clump by ~1e-4) the Maclaurin series, the first omitted terms below 2^-54 of the
// sums, with one final rounding each: 6 or 10 FP64 instructions where CUDA's sincos takes ~26
// (1680 cycles of the FP64 unit, measured).
__device__ __forceinline__ void sincos_step(double t, double t2, double &sn, double &c) {
  if (!in_open_range_bits(t2, 0.0, kSmallAngle2)) {
    sincos(t, &sn, &c);
    return;
  }
  double p = 1.0 / 120.0, q = 1.0 / 24.0;
  if (!in_open_range_bits(t2, 0.0, 9.5367431640625e-07)) {   // 2^-20
    p = __fma_rn(t2, __fma_rn(t2, 1.0 / 362880.0, -1.0 / 5040.0), p);
    q = __fma_rn(t2, __fma_rn(t2, 1.0 / 40320.0, -1.0 / 720.0), q);
  }
  sn = __fma_rn(t * t2, __fma_rn(t2, p, -1.0 / 6.0), t);
  c = __fma_rn(-t2, __fma_rn(-t2, q, 0.5), 1.0);
}

struct Rows {
  V3 x, y, z;
};

// init_Verlet.cu:63-114: the rotation rows turned by the angle vector dO, columns renormalised.
// In the fast mode the path of the device friction law, of turns of 2^-10 rad and more and of
// unnormalised input (the others run in fixed point, predict_state), not inlined there.
template <bool CALL = false>
#ifdef AF3D_FAST
__device__ __noinline__
#else
__device__ __forceinline__
#endif
Rows turn_rows(V3 dO, V3 Rx, V3 Ry, V3 Rz) {
  const double mag2 = dO.x * dO.x + dO.y * dO.y + dO.z * dO.z;
  double mag, imag = 0.0;
  V3 dRx, dRy, dRz;
  if (kFast && in_open_range_bits(mag2, 0.0, kSmallAngle2)) {
    // Fast mode, |dO| < 2^-5: the Rodrigues matrix c I + (sin/|dO|) [dO]x + ((1-c)/|dO|^2) dO dO^T
    // from the Maclaurin series of sin(t)/t and (1 - cos t)/t^2 in t^2 = |dO|^2 (truncated
    // after t^8 and t^10: the first omitted terms are below 2^-53 of the sums), no square
    // root, sine or cosine.
    // Horner form in t2 with the series' coefficients (1/6, 1/120, 1/5040, 1/362880 and
    // 1/2, 1/24, 1/720, 1/40320, 1/3628800): four multiply-adds each.
    // Below |dO| = 2^-10 (t2 < 2^-20, the usual case) the series end after t^4: the first
    // omitted terms, t^6 / 5040 and t^6 / 40320, are below 2^-72.
    const double t2 = mag2;
    double A, Bq;
    if (in_open_range_bits(t2, 0.0, 9.5367431640625e-07)) {
      A = 1.0 + t2 * (-1.0 / 6.0 + t2 * (1.0 / 120.0));
      Bq = 0.5 + t2 * (-1.0 / 24.0 + t2 * (1.0 / 720.0));
    } else {
      A = 1.0 + t2 * (-1.0 / 6.0 + t2 * (1.0 / 120.0 + t2 * (-1.0 / 5040.0 + t2 * (1.0 / 362880.0))));
      Bq = 0.5 + t2 * (-1.0 / 24.0 + t2 * (1.0 / 720.0 + t2 * (-1.0 / 40320.0 + t2 * (1.0 / 3628800.0))));
    }
    const double cc = 1.0 - t2 * Bq;
    const V3 sv = mk(A * dO.x, A * dO.y, A * dO.z);
    const V3 bv = mk(Bq * dO.x, Bq * dO.y, Bq * dO.z);
    dRx = mk(bv.x * dO.x + cc, bv.x * dO.y - sv.z, bv.x * dO.z + sv.y);
    dRy = mk(bv.y * dO.x + sv.z, bv.y * dO.y + cc, bv.y * dO.z - sv.x);
    dRz = mk(bv.z * dO.x - sv.y, bv.z * dO.y + sv.x, bv.z * dO.z + cc);
  } else {
    if (kFast) {
      imag = rsqrt(mag2);
      mag = mag2 * imag;
    } else {
      mag = root<CALL>(mag2);
    }
    if (positive_bits(mag)) {
      // Rodrigues rotation about dO/|dO| by |dO| (init_Verlet.cu:63-83)
      V3 u;
      double c, sn;
      if (kFast) {
        u = mk(dO.x * imag, dO.y * imag, dO.z * imag);
        sincos(mag, &sn, &c);
      } else {
        u = div3<CALL>(dO, mag);
        sincos_step(mag, mag2, sn, c);   // init_Verlet.cu's cos and sin
      }
      const double omc = 1.0 - c;
      dRx = mk(omc * u.x * u.x + c, omc * u.x * u.y - sn * u.z, omc * u.x * u.z + sn * u.y);
      dRy = mk(omc * u.y * u.x + sn * u.z, omc * u.y * u.y + c, omc * u.y * u.z - sn * u.x);
      dRz = mk(omc * u.z * u.x - sn * u.y, omc * u.z * u.y + sn * u.x, omc * u.z * u.z + c);
    } else {
      dRx = mk(1.0, 0.0, 0.0);
      dRy = mk(0.0, 1.0, 0.0);
      dRz = mk(0.0, 0.0, 1.0);
    }
  }
  // R <- dR R (rows), then each column renormalised (init_Verlet.cu:92-114)
  V3 Tx = mk(dRx.x * Rx.x + dRx.y * Ry.x + dRx.z * Rz.x, dRx.x * Rx.y + dRx.y * Ry.y + dRx.z * Rz.y,
             dRx.x * Rx.z + dRx.y * Ry.z + dRx.z * Rz.z);
  V3 Ty = mk(dRy.x * Rx.x + dRy.y * Ry.x + dRy.z * Rz.x, dRy.x * Rx.y + dRy.y * Ry.y + dRy.z * Rz.y,
             dRy.x * Rx.z + dRy.y * Ry.z + dRy.z * Rz.z);
  V3 Tz = mk(dRz.x * Rx.x + dRz.y * Ry.x + dRz.z * Rz.x, dRz.x * Rx.y + dRz.y * Ry.y + dRz.z * Rz.y,
             dRz.x * Rx.z + dRz.y * Ry.z + dRz.z * Rz.z);
  if (kFast) {
    // 1/sqrt(n2) for a column norm n2 within 2^-26 of 1 (a rotation times a rotation):
    // one Newton step from 1, 1.5 - n2/2, whose error 3/8 (n2 - 1)^2 is below 2^-54.
    auto inv_norm = [](double n2) {   // |n2 - 1| < 2^-26, tested on the bits
      return in_open_range_bits(n2, 1.0 - 1.4901161193847656e-08, 1.0 + 1.4901161193847656e-08) ? 1.5 - 0.5 * n2
                                                                                                 : rsqrt(n2);
    };
    double in = inv_norm(Tx.x * Tx.x + Ty.x * Ty.x + Tz.x * Tz.x);
    Rx.x = Tx.x * in; Ry.x = Ty.x * in; Rz.x = Tz.x * in;
    in = inv_norm(Tx.y * Tx.y + Ty.y * Ty.y + Tz.y * Tz.y);
    Rx.y = Tx.y * in; Ry.y = Ty.y * in; Rz.y = Tz.y * in;
    in = inv_norm(Tx.z * Tx.z + Ty.z * Ty.z + Tz.z * Tz.z);
    Rx.z = Tx.z * in; Ry.z = Ty.z * in; Rz.z = Tz.z * in;
  } else {
    V3 q = div3<CALL>(mk(Tx.x, Ty.x, Tz.x), root<CALL>(Tx.x * Tx.x + Ty.x * Ty.x + Tz.x * Tz.x));
    Rx.x = q.x; Ry.x = q.y; Rz.x = q.z;
    q = div3<CALL>(mk(Tx.y, Ty.y, Tz.y), root<CALL>(Tx.y * Tx.y + Ty.y * Ty.y + Tz.y * Tz.y));
    Rx.y = q.x; Ry.y = q.y; Rz.y = q.z;
    q = div3<CALL>(mk(Tx.z, Ty.z, Tz.z), root<CALL>(Tx.z * Tx.z + Ty.z * Ty.z + Tz.z * Tz.z));
    Rx.z = q.x; Ry.z = q.y; Rz.z = q.z;
  }
  return Rows{Rx, Ry, Rz};
}

// init_Verlet.cu:130-142: one coordinate of the sphere centres r + (radius/sqrt2) R (+-1,+-1,+-1)
// from the rotation row R.
__device__ __forceinline__ void place_row(double r0, V3 R, double pos, double *s) {
  if (kFast) {
    // the four patterns (a + c, b - c, c - a, -(b + c)) with a = x + y, b = x - y, from the
    // two partial sums r0 + pos c and r0 - pos c: eight operations per row
    const double a = R.x + R.y, b = R.x - R.y;
    const double up = r0 + pos * R.z, dn = r0 - pos * R.z;
    s[0] = up + pos * a;
    s[2] = up - pos * a;
    s[1] = dn + pos * b;
    s[3] = dn - pos * b;
    return;
  }
  s[0] = r0 + pos * (R.x + R.y + R.z);
  s[1] = r0 + pos * (R.x - R.y - R.z);
  s[2] = r0 + pos * (-R.x - R.y + R.z);
  s[3] = r0 + pos * (-R.x + R.y - R.z);
}

__device__ __forceinline__ void place_spheres(V3 r, V3 Rx, V3 Ry, V3 Rz, double pos, V3 *sp) {
  double x[4], y[4], z[4];
  place_row(r.x, Rx, pos, x);
  place_row(r.y, Ry, pos, y);
  place_row(r.z, Rz, pos, z);
#pragma unroll
  for (int k = 0; k < 4; k++) sp[k] = mk(x[k], y[k], z[k]);
}

// init_Verlet.cu:25-148 for one clump that is not removed: r, v, w and the rotation rows move
// one step with a_i, alpha_i; sp receives the new sphere centres.  Fast mode: the rotation and the
// spheres in fixed point (af3d_fixed.cuh), 18 FP64 instructions instead of 123: a step of
// 262,144 clumps 198 -> 190 us, of 582,320 in 64 flumes 414 -> 398 us (2,048 clumps, where one warp
// has an SM's sub-partition to itself and latency counts: 35.4 -> 37.3 us).  dev: the device friction
// law, whose runs show every last bit (af3d_physics.cuh): in FP64.
template <bool CALL = false>
__device__ __forceinline__ void predict_state(V3 &r, V3 &v, V3 &w, V3 a, V3 al, V3 &Rx, V3 &Ry, V3 &Rz, V3 *sp,
                                              double rad, double dt, double hdt, int qs, bool dev) {
  r.x += dt * (v.x + hdt * a.x);
  r.y += dt * (v.y + hdt * a.y);
  r.z += dt * (v.z + hdt * a.z);
  v.x += dt * a.x;
  v.y += dt * a.y;
  v.z += dt * a.z;
  const V3 dO = mk(dt * (w.x + hdt * al.x), dt * (w.y + hdt * al.y), dt * (w.z + hdt * al.z));
  w.x += dt * al.x;
  w.y += dt * al.y;
  w.z += dt * al.z;
  constexpr Divisor root2 = constant_divisor(kROOT2, 0x3FF6A09E667F3BCCull);
  const double pos = kFast ? rad * (1.0 / kROOT2) : div_by(rad, root2);
  if (kFast && !dev) {
    const double angle[3] = {dO.x, dO.y, dO.z};
    const double R[9] = {Rx.x, Rx.y, Rx.z, Ry.x, Ry.y, Ry.z, Rz.x, Rz.y, Rz.z};
    long long turned[9];
    if (rotate_fixed(angle, R, turned)) {
      Rx = mk(double_of(turned[0], 62), double_of(turned[1], 62), double_of(turned[2], 62));
      Ry = mk(double_of(turned[3], 62), double_of(turned[4], 62), double_of(turned[5], 62));
      Rz = mk(double_of(turned[6], 62), double_of(turned[7], 62), double_of(turned[8], 62));
      const double at[3] = {r.x, r.y, r.z};
      double c[12];
      if (spheres_fixed(turned, at, pos, qs + 38, c)) {
        for (int k = 0; k < 4; k++) sp[k] = mk(c[3 * k], c[3 * k + 1], c[3 * k + 2]);
        return;
      }
    } else {
      const Rows t = turn_rows<CALL>(dO, Rx, Ry, Rz);
      Rx = t.x; Ry = t.y; Rz = t.z;
    }
  } else {
    const Rows t = turn_rows<CALL>(dO, Rx, Ry, Rz);
    Rx = t.x; Ry = t.y; Rz = t.z;
  }
  place_spheres(r, Rx, Ry, Rz, pos, sp);
}

// cell_locate's bucket of a clump at r (cells.cu:60-92) at time t: the flume's cell offset + cell
// index, or ncell_total + id for a clump that is not binned (removed, or non-finite).
__device__ __forceinline__ long bucket_key(V3 r, const DevFlume &fl, DevScalars *d, long long id, double t) {
  const af3d_cell_par &g = fl.grid;
  if (is_removed(t, r.x, fl.sys.side.x)) return d->ncell_total + id;
  if (!(finite_bits(r.x) && finite_bits(r.y) && finite_bits(r.z))) {
    raise_status(d, AF3D_ERR_NAN);
    return d->ncell_total + id;
  }
  const GridF &gf = fl.gridf;
  long i = bin_axis_f(r.x, gf.xmin, gf.ix, g.rr_min.x, g.cs_inv.x, g.ncell.x);
  long j = bin_axis_f(r.y, gf.ymin, gf.iy, g.rr_min.y, g.cs_inv.y, g.ncell.y);
  long k = bin_axis_f(r.z, gf.zmin, gf.iz, g.rr_min.z, g.cs_inv.z, g.ncell.z);
  if (i < 0 || j < 0 || k < 0) {
    raise_status(d, AF3D_ERR_NEGATIVE_CELL);
    i = i < 0 ? 0 : i; j = j < 0 ? 0 : j; k = k < 0 ? 0 : k;
  }
  if (i >= g.ncell.x || j >= g.ncell.y || k >= g.ncell.z) {
    raise_status(d, AF3D_ERR_GRID_ESCAPE);
    i = i < g.ncell.x ? i : g.ncell.x - 1;
    j = j < g.ncell.y ? j : g.ncell.y - 1;
    k = k < g.ncell.z ? k : g.ncell.z - 1;
  }
  return fl.cell_off + i + g.ncell.x * (j + k * g.ncell.y);
}

// A clump's place in a step that keeps its near lists: counted in its cell for the capacity check
// of cells.cu:96-102 (at most ntags - 1 clumps), and its motion since the previous step's record
// (old) against its allowance: with none left it is away at tick `tick` (true, for its record).
__device__ __forceinline__ bool keep_place(long s, const int4 *old, const CullRec &cr, const DevFlume &fl,
                                           DevScalars *d, int *occ, long ntags, const NearLists &near,
                                           const int *__restrict__ start, const int *__restrict__ order,
                                           const Margins &m, int tick, long n) {
  if (ntags > 0 && cr.key < d->ncell_total && atomicAdd(&occ[cr.key], 1) + 1 >= ntags)
    raise_status(d, AF3D_ERR_CELL_CAPACITY);
  const float rem = near.rem[s] - sphere_motion(old, cr, m.qs);
  near.rem[s] = rem;
  CellAt at;
  if (rem >= 0.0f || !cell_at(cr.key, fl.cell_off, fl.gridf, at)) return false;
  go_away(s, cr.c, cr.key, at, m, fl, d, start, order, near, tick, n);
  return true;
}

// init_Verlet.cu:25-148 for one clump (PREDICT), and/or cell_locate's binning (cells.cu:60-92)
// with the current time (KEYS): the bucket key, the bucket count and the clump's arrival rank.
// Clumps that are not binned (removed, or non-finite) get the unique bucket ncell_total + id, so every
// bucket holds its clumps in id order after the rank pass.  `t_prev`: init_Verlet's removal test
// uses the time before the advance (the fused step advances time first).  RECORDS: also write
// the clump's neighbour records at its own slot (steps that keep the slot order).  count_only: the
// step does not sort but keeps its near lists (keep_place; with RECORDS).
template <bool PREDICT, bool KEYS, bool RECORDS>
__global__ void __launch_bounds__(kBlock) k_predict(const __grid_constant__ Planes P, DevScalars *d, bool t_prev,
                                                    Cells cells,
                                                    const long long *__restrict__ id,
                                                    const int *__restrict__ flume, long ntags,
                                                    const __grid_constant__ NearLists near,
                                                    const int *__restrict__ order, bool count_only, NbrRec *nbr,
                                                    CullRec *cull, long s0, long n) {
  __shared__ double s_nbr[RECORDS ? kPermBlock * kRecStride : 1];
  __shared__ CullRec s_cull[RECORDS ? kPermBlock : 1];
  const long base = s0 + blockIdx.x * (long)blockDim.x;
  const long s = base + threadIdx.x;
  const bool valid = s < n;
  if (!RECORDS && !valid) return;
  NbrRec q;
  CullRec cr;
  if (valid) {
    const DevFlume &fl = d->flumes[flume[s]];
    V3 r = load3(P, RX, s);
    V3 v, w, sp[4];
    bool have = false;   // v, w, sp hold the clump's current values
    if (PREDICT) {
      const double t_init = t_prev ? d->time_prev : d->time;
      if (is_removed(t_init, r.x, fl.sys.side.x)) {
        P.p[RAD][s] = 0.0;
      } else {
        v = load3(P, VX, s);
        w = load3(P, WX, s);
        V3 Rx = load3(P, R00, s), Ry = load3(P, R10, s), Rz = load3(P, R20, s);
        predict_state(r, v, w, load3(P, AIX, s), load3(P, ALIX, s), Rx, Ry, Rz, sp, P.p[RAD][s], fl.sys.dt,
                      fl.sys.hdt, P.m.qs, d->variant == AF3D_FRICTION_DEV);
        store3(P, RX, s, r);
        store3(P, VX, s, v);
        store3(P, WX, s, w);
        store3(P, R00, s, Rx);
        store3(P, R10, s, Ry);
        store3(P, R20, s, Rz);
        for (int k = 0; k < 4; k++) store3(P, S0X + 3 * k, s, sp[k]);
        have = true;
      }
    }
    long key = 0;
    if (KEYS) {
      key = bucket_key(r, fl, d, id[s], d->time);
      cells.key[s] = (int)key;
      if (!(RECORDS && count_only)) cells.rank_tmp[s] = arrive_in_bucket(cells, key);
    }
    if (RECORDS) {
      if (!have) {
        v = load3(P, VX, s);
        w = load3(P, WX, s);
        for (int k = 0; k < 4; k++) sp[k] = load3(P, S0X + 3 * k, s);
      }
      make_records(r, v, w, sp, P.p[RAD][s], P.p[MSPH][s], P.p[MWALL][s], P.m, (int)key, q, cr);
      if (count_only) {
        int4 old[4];
        for (int k = 0; k < 4; k++) old[k] = cull[s].s[k];
        cr.away = keep_place(s, old, cr, fl, d, cells.occ, ntags, near, cells.start, order, P.m, d->tick, n);
      }
    }
  }
  if (RECORDS) store_records<kPermBlock>(valid, base, n, q, cr, nbr, cull, s_nbr, s_cull);
}

// ------------------------------------------------------------------ permutation + records

// dst[p][s] = src[p][perm[s]] for every plane (the force/torque accumulators and a_f only with
// `ft`: the fused step rewrites them before reading), plus the packed records of the new slot,
// assembled in shared memory and written out as contiguous 16-byte stores.  Latency-bound at
// small counts: the planes are loaded a group at a time before the group is stored (a store might
// alias the next load, which then waits for it): 8,192 clumps took 36.7 us, now 10.2.
constexpr int kPermGroup = 16;
__global__ void __launch_bounds__(kPermBlock) k_permute(Planes src, Planes dst, const int *__restrict__ perm,
                                                        const int *__restrict__ key,
                                                        const long long *__restrict__ id_src,
                                                        long long *id_dst, const int *__restrict__ fl_src,
                                                        int *fl_dst, NbrRec *nbr, CullRec *cull,
                                                        bool ft, long n) {
  __shared__ double s_nbr[kPermBlock * kRecStride];
  __shared__ CullRec s_cull[kPermBlock];
  const long base = blockIdx.x * (long)kPermBlock;
  const long s = base + threadIdx.x;
  const long o = s < n && perm ? perm[s] : s;
  if (s < n && perm) {
    const long long i = id_src[o];
    const int f = fl_src[o];
#pragma unroll
    for (int p0 = 0; p0 < NPLANES; p0 += kPermGroup) {
      double v[kPermGroup];
#pragma unroll
      for (int k = 0; k < kPermGroup; k++) {
        const int p = p0 + k;
        if (p < NPLANES && (ft || ((p < FX || p > TZ) && (p < AFX || p > ALFZ)))) v[k] = src.p[p][o];
      }
#pragma unroll
      for (int k = 0; k < kPermGroup; k++) {
        const int p = p0 + k;
        if (p < NPLANES && (ft || ((p < FX || p > TZ) && (p < AFX || p > ALFZ)))) dst.p[p][s] = v[k];
      }
    }
    id_dst[s] = i;
    fl_dst[s] = f;
  }
  if (!nbr) return;
  NbrRec q;
  CullRec cr;
  if (s < n) {
    V3 sp[4];
    for (int k = 0; k < 4; k++) sp[k] = load3(src, S0X + 3 * k, o);
    make_records(load3(src, RX, o), load3(src, VX, o), load3(src, WX, o), sp, src.p[RAD][o], src.p[MSPH][o],
                 src.p[MWALL][o], dst.m, perm ? key[o] : 0, q, cr);
  }
  store_records<kPermBlock>(s < n, base, n, q, cr, nbr, cull, s_nbr, s_cull);
}

// ------------------------------------------------------------------ particle contacts

constexpr int kCandCap = 48;
// The sixteen sph_id passes of force_part for one clump are summed in the reference order:
// sph_id outer, then cells, then slots.  Phase 1 walks the 27 neighbour cells once and keeps the
// FP32-surviving partners with their 16-bit pair masks; phase 2 flattens them into one item list
// per clump in that order (sph_id-major); the items are then run through the exact FP64 test and
// contact law one by one and added in list order.  Returns false when a list would overflow.
constexpr int kItemCap = 96;

__device__ __forceinline__ bool gather_items(long s, const Own &o, const af3d_cell_par &g,
                                             long long off, const CullRec *__restrict__ cull,
                                             const int *__restrict__ start, const int *__restrict__ order,
                                             unsigned want, unsigned *items, int cap, int &nitems) {
  const CullRec me = cull[s];
  const Search q = search_centre(o.r, g, off);
  int cand_t[kCandCap];
  unsigned short cand_m[kCandCap];
  int ncand = 0;
  bool overflow = false;
  for_neighbour_slots_pre(q, g, start, order, [&](int t) {
    if (t == s) return;
    const unsigned m = pair_mask(me, cull[t]) & want;
    if (!m) return;
    if (ncand < kCandCap) {
      cand_t[ncand] = t;
      cand_m[ncand] = (unsigned short)m;
      ncand++;
    } else {
      overflow = true;
    }
  });
  nitems = 0;
  if (overflow) return false;
#pragma unroll 1
  for (int p = 0; p < 16; p++) {
    if (!((want >> p) & 1u)) continue;
#pragma unroll 1
    for (int k = 0; k < ncand; k++) {
      if (!((cand_m[k] >> p) & 1u)) continue;
      if (nitems == cap) return false;
      items[nitems++] = ((unsigned)cand_t[k] << 4) | (unsigned)p;   // (partner slot, sph_id - 1)
    }
  }
  return true;
}

// Every pair of clump s walked cell by cell once per sph_id (the order of sixteen force_part
// launches); used when a clump has more partners than the item lists hold.
__device__ __forceinline__ int contacts_by_pass(long s, const Own &o, const Consts &c,
                                                const af3d_cell_par &g, long long off,
                                                const NbrRec *__restrict__ nbr,
                                                const CullRec *__restrict__ cull,
                                                const int *__restrict__ start,
                                                const int *__restrict__ order, unsigned want, V3 &F,
                                                V3 &T) {
  const bool xi0 = c.variant == AF3D_FRICTION_DEV;
  const CullRec me = cull[s];
  const Search q = search_centre(o.r, g, off);
  int active = 0;
#pragma unroll 1
  for (int p = 0; p < 16; p++) {
    if (!((want >> p) & 1u)) continue;
    const int sl = p & 3, sm = p >> 2;
    for_neighbour_slots(q, g, start, order, [&](int t) {
      if (t == s) return;
      if (!((pair_mask(me, cull[t]) >> p) & 1u)) return;
      active += part_pair(o.r, o.v, o.w, o.s[sl], o.rad, o.msph, nbr[t], sm, c, xi0, F, T) == 2;
    });
  }
  return active;
}

// Per-clump contact pass (one thread, its own item list): the per-routine force_part entry.
__device__ __forceinline__ int particle_contacts(long s, const Own &o, const Consts &c,
                                                 const af3d_cell_par &g, long long off,
                                                 const NbrRec *__restrict__ nbr,
                                                 const CullRec *__restrict__ cull,
                                                 const int *__restrict__ start,
                                                 const int *__restrict__ order, int only_p, V3 &F,
                                                 V3 &T) {
  const bool xi0 = c.variant == AF3D_FRICTION_DEV;
  const unsigned want = only_p < 0 ? 0xffffu : (1u << only_p);
  unsigned items[kItemCap];
  int nitems = 0;
  if (!gather_items(s, o, g, off, cull, start, order, want, items, kItemCap, nitems))
    return contacts_by_pass(s, o, c, g, off, nbr, cull, start, order, want, F, T);
  int active = 0;
#pragma unroll 1
  for (int i = 0; i < nitems; i++) {
    const int t = (int)(items[i] >> 4), p = (int)(items[i] & 15u);
    active += part_pair(o.r, o.v, o.w, o.s[p & 3], o.rad, o.msph, nbr[t], p >> 2, c, xi0, F, T) == 2;
  }
  return active;
}

// Block-cooperative pass of the fused kernel over every contact of a clump: the boundary routines
// that run before the particle contacts, the sixteen sph_id passes, and the routines that run
// after them (avalanche: hop x3, funnel, fcorners, walls | part x16 | flume; fill: part x16 |
// hop x3).  The list phase (lists_body) has published every clump's item list in that
// order: boundary items (routine, sphere) for the spheres the routine's 1-Lipschitz gate cannot
// rule out, and particle items (partner slot, sph_id) of overlapping sphere pairs in sph_id-major
// order.  The block concatenates the lists of its clumps and works through them in batches of
// kBatch items, 32 items a round per warp, one item per lane, reading the owner clump from its
// record; after each batch every owner adds its items' force and torque terms to its own sums in
// list order.  The FP64 contact laws thus run with nearly all lanes busy whatever the spread of
// contacts and walls over the clumps, and each clump's summation order stays the reference's.
// Every thread of the block must call this; `act` is false for threads without a clump to
// process (and for removed clumps).  A clump whose lists overflowed runs alone afterwards, in
// the same order.
constexpr int kBatch = 256;
template <int NB>
struct BlockQueue {
  int base[NB + 1];   // exclusive prefix of the clumps' item counts
  int pbase[NB + 1];  // ... of their particle item counts (kind-sorted pass)
  int qbase[NB + 1];  // ... of their boundary item counts (kind-sorted pass)
  int wsum[3][NB / 32];
  double res[6][kBatch];  // [component][item in the batch]
  unsigned item[kBatch];        // the batch's items in the order they are processed
  unsigned char owner[kBatch];  // ... their owners' threads
  unsigned char place[kBatch];  // ... and places in the owners' lists
  unsigned char flag[kBatch];
};
static_assert(kBatch <= 256, "owners and places are bytes");

// Block-wide exclusive prefixes of three per-thread counts (all threads call this).
template <int NB>
__device__ __forceinline__ void block_prefix3(BlockQueue<NB> &bq, int a, int b, int c) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int v[3] = {a, b, c};
#pragma unroll
  for (int q = 0; q < 3; q++) {
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v[q], k);
      if (lane >= k) v[q] += u;
    }
    if (lane == 31) bq.wsum[q][warp] = v[q];
  }
  __syncthreads();
  int *dst[3] = {bq.base, bq.pbase, bq.qbase};
  const int own[3] = {a, b, c};
#pragma unroll
  for (int q = 0; q < 3; q++) {
    int wofs = 0, total = 0;
#pragma unroll
    for (int w = 0; w < NB / 32; w++) {
      const int t = bq.wsum[q][w];
      wofs += w < warp ? t : 0;
      total += t;
    }
    dst[q][tid] = wofs + v[q] - own[q];
    if (tid == NB - 1) dst[q][NB] = total;
  }
  __syncthreads();
}

__device__ __forceinline__ Own own_from_record(const NbrRec &q) {
  Own o;
  o.r = mk(q.rx, q.ry, q.rz);
  o.v = mk(q.vx, q.vy, q.vz);
  o.w = mk(q.wx, q.wy, q.wz);
  for (int k = 0; k < 4; k++) o.s[k] = mk(q.s[3 * k], q.s[3 * k + 1], q.s[3 * k + 2]);
  o.rad = q.rad;
  o.msph = q.msph;
  o.mwall = q.mwall;
  return o;
}

__device__ __forceinline__ Own own_from_planes(const Planes &P, long s) {
  Own o;
  o.r = load3(P, RX, s);
  o.v = load3(P, VX, s);
  o.w = load3(P, WX, s);
  for (int k = 0; k < 4; k++) o.s[k] = load3(P, S0X + 3 * k, s);
  o.rad = P.p[RAD][s];
  o.msph = P.p[MSPH][s];
  o.mwall = P.p[MWALL][s];
  return o;
}

// Visits the sphere pairs of clump s that the tests in units cannot rule out: the clumps around it in
// the built order and those away in the 27 cells around it (an oversize clump may be both).
// f(key, item): the pair's place in the reference's order -- by sph_id, then the partner's cell in the
// 27-cell visiting order, then its id (force_part.cu:88-106) -- and partner slot << 4 | sph_id - 1.
template <typename F>
__device__ __forceinline__ void for_pairs(long s, const DevScalars *d, const int *__restrict__ flume,
                                          const NbrRec *__restrict__ nbr, const CullRec *__restrict__ cull,
                                          const int *__restrict__ start, const int *__restrict__ order,
                                          const long long *__restrict__ id, const NearLists &near, const Margins &m,
                                          long n, F &&f) {
  const DevFlume &fl = d->flumes[flume[s]];
  const GridF &g = fl.gridf;
  const CullRec me = cull[s];
  CellAt at;
  if (!cell_at(me.key, fl.cell_off, g, at)) return;
  const Search q = search_centre_f(me.c, mk(nbr[s].rx, nbr[s].ry, nbr[s].rz), fl.grid, g, 0);
  auto look = [&](int t) {
    unsigned mask = pair_mask(me, cull[t]);
    CellAt a;
    if (!mask || !cell_at(cull[t].key, fl.cell_off, g, a)) return;
    const long dx = a.x - q.ci + 1, dy = a.y - q.cj + 1, dz = a.z - q.ck + 1;
    if (dx < 0 || dx > 2 || dy < 0 || dy > 2 || dz < 0 || dz > 2) return;
    const unsigned long long place = (unsigned long long)(9 * dx + 3 * dy + dz) << 32 | (unsigned long long)id[t];
    while (mask) {
      const int p = __ffs(mask) - 1;
      mask &= mask - 1u;
      f(((unsigned long long)(p * 27) << 32) + place + 1ull, (unsigned)t << 4 | (unsigned)p);
    }
  };
  for_slots_around(me.c, at, m, g, fl.cell_off, start, order, [&](int t) {
    if (t != s && !cull[t].away) look(t);
  });
  const int tick = d->tick;
  if (d->away > tick) return;
#pragma unroll 1
  for (int k = 0; k < 27; k++) {
    const long x = q.ci + k / 9 - 1, y = q.cj + k / 3 % 3 - 1, z = q.ck + k % 3 - 1;
    if (x < 0 || y < 0 || z < 0 || x >= g.nx || y >= g.ny || z >= g.nz) continue;
    for_chain(near, cull, (int)(fl.cell_off + x + (long)g.nx * (y + (long)g.ny * z)), tick, n, [&](int t) {
      if (t != s) look(t);
    });
  }
}

// The particle items of a clump whose near list does not hold (too many entries, or a clump around it is
// away): the items the list would have given, put in order as they are found.  To the column `col` from
// entry `nitems` on; returns the entries then, -1 if they would overflow it.  Not inlined: rare.
__device__ __noinline__ int search_items(long s, const DevScalars *d, const int *__restrict__ flume,
                                          const NbrRec *__restrict__ nbr, const CullRec *__restrict__ cull,
                                          const int *__restrict__ start, const int *__restrict__ order,
                                          const long long *__restrict__ id, const NearLists &near, const Margins &m,
                                          long n, unsigned *col, int nitems) {
  unsigned long long keys[kListCap] = {};
  unsigned items[kListCap];
  const int room = kListCap - nitems;
  int found = 0;
  bool over = false;
  for_pairs(s, d, flume, nbr, cull, start, order, id, near, m, n, [&](unsigned long long key, unsigned item) {
    int i = found;
    while (i > 0 && keys[i - 1] > key) i--;
    if (i > 0 && keys[i - 1] == key) return;
    if (found == room) {
      over = true;
      return;
    }
    for (int j = found++; j > i; j--) {
      keys[j] = keys[j - 1];
      items[j] = items[j - 1];
    }
    keys[i] = key;
    items[i] = item;
  });
  if (over) return -1;
  for (int i = 0; i < found; i++) col[n * nitems++] = items[i];
  return nitems;
}

// The next overlapping sphere pair of clump s after the one of key `done` (for_pairs): its key, ~0 after
// the last one.
__device__ __forceinline__ unsigned long long next_contact(long s, const DevScalars *d, const int *__restrict__ flume,
                                                           const NbrRec *__restrict__ nbr,
                                                           const CullRec *__restrict__ cull,
                                                           const int *__restrict__ start,
                                                           const int *__restrict__ order,
                                                           const long long *__restrict__ id,
                                                           const NearLists &near, const Margins &m, long n,
                                                           unsigned long long done, unsigned &item) {
  const NbrRec &mine = nbr[s];
  unsigned long long best = ~0ull;
  for_pairs(s, d, flume, nbr, cull, start, order, id, near, m, n, [&](unsigned long long key, unsigned it) {
    if (key <= done || key >= best) return;
    V3 dd;
    double dist2, sep;
    const int k = it & 3;
    if (!spheres_overlap(mk(mine.s[3 * k], mine.s[3 * k + 1], mine.s[3 * k + 2]), mine.rad, nbr[it >> 4],
                         (it >> 2) & 3, dd, dist2, sep))
      return;
    best = key;
    item = it;
  });
  return best;
}

// The contacts of a clump with more items than its list holds, added to (F, T) in the reference's
// order: the boundary routines before the particles, the overlapping sphere pairs, the routines
// after.  Not inlined: it runs rarely, and inlined its registers and spills would weigh on the
// pooled path of every clump.  The clump's state, bound and grid are read here again.
struct SlowSums {
  V3 F, T;
  int active;
};
__device__ __noinline__ SlowSums slow_contacts(long s, int pre0, int pre1, int post0, int post1, const Consts &c,
                                               const DevScalars *d, const int *__restrict__ flume,
                                               const NbrRec *__restrict__ nbr, const CullRec *__restrict__ cull,
                                               const int *__restrict__ start, const int *__restrict__ order,
                                               const long long *__restrict__ id, const NearLists &near,
                                               const Margins &m, long n, V3 F, V3 T) {
  const Own o = own_from_record(nbr[s]);
  const double B = (double)cull[s].c.w;
  for (int rt = pre0; rt <= pre1; rt++)
    if (bnd_may_touch(rt, o.r, B, c)) bnd_routine(rt, o, false, c, F, T);
  const bool xi0 = c.variant == AF3D_FRICTION_DEV;
  int active = 0;
  unsigned item = 0u;
  for (unsigned long long done = 0ull;;) {
    done = next_contact(s, d, flume, nbr, cull, start, order, id, near, m, n, done, item);
    if (done == ~0ull) break;
    const int p = (int)(item & 15u);
    active += part_pair(o.r, o.v, o.w, o.s[p & 3], o.rad, o.msph, nbr[item >> 4], p >> 2, c, xi0, F, T) == 2;
  }
  for (int rt = post0; rt <= post1; rt++)
    if (bnd_may_touch(rt, o.r, B, c)) bnd_routine(rt, o, false, c, F, T);
  return SlowSums{F, T, active};
}

// A removed clump's contacts: hop, funnel and fcorners only (walls, part and flume skip it).  B: its
// sphere offsets + radius, rounded up.  Not inlined: rare.
__device__ __noinline__ SlowSums removed_contacts(const NbrRec *me, double B, const Consts &c) {
  const Own o = own_from_record(*me);
  SlowSums r = {mk(0.0, 0.0, 0.0), mk(0.0, 0.0, 0.0), 0};
  for (int rt = R_HOP0; rt <= R_FCORNERS; rt++)
    if (bnd_may_touch(rt, o.r, B, c)) bnd_routine(rt, o, true, c, r.F, r.T);
  return r;
}

// A boundary item of owner record `me`: its force and torque terms into res (components `stride`
// apart); 3 with a force, else 0.  Not inlined: the seven routines' inputs raise the register
// pressure of whatever they are inlined into, and a round of items is of one kind.
template <bool CALL = false>
__device__ __noinline__ int bnd_contact(unsigned it, const NbrRec *me, const Consts &co, double *res, int stride) {
  const int rt = (int)((it >> 2) & 7u), ns = (int)(it & 3u);
  Sph q;
  q.r = mk(me->rx, me->ry, me->rz);
  q.v = mk(me->vx, me->vy, me->vz);
  q.w = mk(me->wx, me->wy, me->wz);
  q.s = mk(me->s[3 * ns], me->s[3 * ns + 1], me->s[3 * ns + 2]);
  q.rad = me->rad;
  q.mwall = me->mwall;
  V3 fs, tq;
  if (!bnd_sphere<CALL>(rt, q, co, fs, tq)) return 0;
  res[0] = fs.x; res[stride] = fs.y; res[2 * stride] = fs.z;
  res[3 * stride] = tq.x; res[4 * stride] = tq.y; res[5 * stride] = tq.z;
  return 3;
}

// UNIFORM: every clump of the launch belongs to one flume, whose constants `c` are (a
// reference to) a kernel parameter.  lc: the clump's list layout (pre boundary items, particle
// items, the rest boundary items).  RECORD: a pass that keeps its lists (`record`) leaves only the items
// with a force in them, and `listed` and lc say so: the adjoint has nothing to reverse at the others.
template <int NB, bool UNIFORM, bool RECORD>
__device__ __forceinline__ int block_contacts(BlockQueue<NB> &bq, long bbase, long s, bool act, bool aval,
                                              const Consts &c, const DevScalars *d, const int *__restrict__ flume,
                                              const NbrRec *__restrict__ nbr,
                                              const CullRec *__restrict__ cull,
                                              const int *__restrict__ start,
                                              const int *__restrict__ order, const long long *__restrict__ id,
                                              const NearLists &near, const Margins &m, unsigned *items, bool record,
                                              int &listed, ListCounts &lc, long n, V3 &F, V3 &T) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pre0 = aval ? R_HOP0 : 1, pre1 = aval ? R_WALLS : 0;         // fill: none before
  const int post0 = aval ? R_FLUME : R_HOP0, post1 = aval ? R_FLUME : R_HOP2;
  const bool slow = act && listed < 0;
  const int nitems = act && listed > 0 ? listed : 0;
  const int npair = nitems > 0 ? lc.pair : 0;
  block_prefix3<NB>(bq, nitems, npair, nitems - npair);
  const int base = bq.base[tid], total = bq.base[NB];
  const int ptotal = bq.pbase[NB];
  // One item: its contact into its owner's place of the batch.
  auto constants_of = [&](long os) -> const Consts & {
    if constexpr (UNIFORM) {
      return c;
    } else {   // the owner's flume may differ from this thread's at a flume boundary of an ensemble
      const int of = flume[os];
      return of == flume[s] ? c : d->flumes[of].c;
    }
  };
  auto pair = [&](unsigned it, long os, int jb) {
    const NbrRec &me = nbr[os];
    const Consts &co = constants_of(os);
    const int t = (int)(it >> 4), p = (int)(it & 15u), k = p & 3;
    const V3 rl = mk(me.rx, me.ry, me.rz);
    ContactIn ci;
    V3 fs, tq;
    int r = 0;
    if (pair_input<kCall>(rl, mk(me.vx, me.vy, me.vz), mk(me.wx, me.wy, me.wz),
                   mk(me.s[3 * k], me.s[3 * k + 1], me.s[3 * k + 2]), me.rad, me.msph, nbr[t], p >> 2, co,
                   co.variant == AF3D_FRICTION_DEV, ci) &&
        apply_law<kCall>(ci, rl, co, fs, tq)) {
      r = 2;
      bq.res[0][jb] = fs.x; bq.res[1][jb] = fs.y; bq.res[2][jb] = fs.z;
      bq.res[3][jb] = tq.x; bq.res[4][jb] = tq.y; bq.res[5][jb] = tq.z;
    }
    bq.flag[jb] = (unsigned char)r;
  };
  int active = 0;
  int kept = 0;
  ListCounts kc = {0, 0};
  // Owners add their items' terms in list order.
  auto gather = [&](int b0, int bn) {
    if (nitems <= 0) return;
    const int a = base > b0 ? base : b0;
    const int b = base + nitems < b0 + bn ? base + nitems : b0 + bn;
    for (int e = a - b0; e < b - b0; e++) {
      const int fl = bq.flag[e];
      if (fl < 2) continue;
      T.x += bq.res[3][e]; T.y += bq.res[4][e]; T.z += bq.res[5][e];
      F.x += bq.res[0][e]; F.y += bq.res[1][e]; F.z += bq.res[2][e];
      active += fl == 2;   // sphere-sphere contacts only
      if (RECORD && record) {   // (never past the entries that are still to be laid out)
        const int at = e + b0 - base;
        items[n * kept++ + s] = items[(long)at * n + s];
        kc.pre += at < lc.pre;
        kc.pair += fl == 2;
      }
    }
  };
  // A block whose items fit one batch takes them in kind order: every particle item of the
  // block, then every boundary item, 32 a round, so that a round is of one kind and no lane is
  // idle but in each kind's last round; results go to the items' places in the owners' lists.
  // Otherwise batches of kBatch items in the owners' order, particle items then boundary items of
  // each.  The owners first lay their items out in shared memory in that order.
  constexpr int kWarps = NB / 32;
  const bool kind_order = total <= kBatch;
  const int pb = bq.pbase[tid], qb = ptotal + bq.qbase[tid];
  for (int b0 = 0; b0 < total; b0 += kBatch) {
    const int bn = total - b0 < kBatch ? total - b0 : kBatch;
    const int e0 = base > b0 ? 0 : b0 - base, e1 = nitems < b0 + bn - base ? nitems : b0 + bn - base;
    for (int e = e0; e < e1; e++) {
      const unsigned it = items[(long)e * n + s];
      const int at = base + e - b0;
      const int j = !kind_order ? at : it < kBndItem ? pb + (e - lc.pre) : qb + (e < lc.pre ? e : e - npair);
      bq.item[j] = it;
      bq.owner[j] = (unsigned char)tid;
      bq.place[j] = (unsigned char)at;
    }
    __syncthreads();
    const int np = kind_order ? ptotal : bn, q0 = kind_order ? ptotal : 0;
    for (int i = tid; i < np; i += NB) {
      const unsigned it = bq.item[i];
      if (it < kBndItem) pair(it, bbase + bq.owner[i], bq.place[i]);
    }
    // the boundary rounds go to the warps after those that took the last particle rounds
    const int w0 = (warp + kWarps - (np + 31) / 32 % kWarps) % kWarps;
    for (int i = q0 + 32 * w0 + lane; i < bn; i += NB) {
      const unsigned it = bq.item[i];
      const int at = bq.place[i];
      if (it >= kBndItem) {
        const long os = bbase + bq.owner[i];
        bq.flag[at] = (unsigned char)bnd_contact<kCall>(it, nbr + os, constants_of(os), &bq.res[0][at], kBatch);
      }
    }
    __syncthreads();
    gather(b0, bn);
    __syncthreads();
  }
  if (RECORD && record && nitems > 0) {
    listed = kept;
    lc = kc;
  }
  if (slow) {
    const SlowSums r = slow_contacts(s, pre0, pre1, post0, post1, c, d, flume, nbr, cull, start, order, id, near, m, n,
                                     F, T);
    F = r.F;
    T = r.T;
    active += r.active;
  }
  return active;
}

__device__ __forceinline__ void warp_count(DevScalars *d, int active) {
  unsigned v = (unsigned)active;
  for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(&d->contacts, (unsigned long long)v);
}

// Candidate pairs of one warp's clumps in shared memory, one column per lane: (sph_id - 1) * 32 +
// cell place << 6 | entry of the near list.
struct PassLists {
  unsigned short cand[kListCap][32];
};
static_assert(kNearCap <= 64, "candidates hold 6 bits of entry");

// Of the routine and sphere bits `bits` of one clump, those whose FP32 gates admit the sphere:
// every sphere the routine can touch (and a few more, which its exact test rejects).
__device__ __forceinline__ unsigned touching(unsigned bits, const NbrRec &me, float rad, const Consts &c) {
  const bool door_closed = *c.tp < 0.0;
  unsigned out = 0u;
#pragma unroll 1
  while (bits) {
    const unsigned b = (unsigned)__ffs(bits) - 1u;
    bits &= bits - 1u;
    const int ns = (int)(b & 3u);
    const float4 p = make_float4(to_float_rn(me.s[3 * ns]), to_float_rn(me.s[3 * ns + 1]),
                                 to_float_rn(me.s[3 * ns + 2]), 0.0f);
    if (!(rad < kCullMaxUnits) || bnd_may_touch_f((int)(b >> 2), p, rad, c, door_closed)) out |= 1u << b;
  }
  return out;
}

// The near-list pairs of clump s within a few units of overlap into its column of pl, in the
// reference's order; returns their count, -1 for more than an item list holds.  Four entries a turn
// are loaded and tested together; the few hits are put in order by the current cells (the
// entries are in id order, so equal places stay so).  The exact test is the force pass's.
__device__ __forceinline__ int near_pairs(long s, int entries, const DevFlume &fl, const NbrRec &me,
                                          const CullRec *__restrict__ cull, const unsigned *list, long n,
                                          PassLists &pl) {
  const int lane = threadIdx.x & 31;
  const CullRec &rec = cull[s];
  const float radu = __int_as_float(rec.s[0].w);
  int ncand = 0;
  bool have_cell = false;
  int ci = 0, cj = 0, ck = 0;
#pragma unroll 1
  for (int e0 = 0; e0 < entries; e0 += 4) {
    unsigned it[4];
    int4 a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) it[k] = e0 + k < entries ? list[(long)(e0 + k) * n] : 0xFFFFFFFFu;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (it[k] != 0xFFFFFFFFu) {
        a[k] = rec.s[it[k] & 3u];
        b[k] = cull[it[k] >> 4].s[(it[k] >> 2) & 3u];
      }
    unsigned hit = 0u;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float r = radu + __int_as_float(b[k].w);
      const float dx = unit_difference(b[k].x, a[k].x), dy = unit_difference(b[k].y, a[k].y),
                  dz = unit_difference(b[k].z, a[k].z);
      if (it[k] != 0xFFFFFFFFu &&
          !(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > r * r * (1.0f + 9.5367431640625e-07f)))
        hit |= 1u << k;
    }
#pragma unroll 1
    while (hit) {
      const int k = __ffs(hit) - 1;
      hit &= hit - 1u;
      const unsigned item = k == 0 ? it[0] : k == 1 ? it[1] : k == 2 ? it[2] : it[3];
      if (!have_cell) {
        const Search q = search_centre_f(rec.c, mk(me.rx, me.ry, me.rz), fl.grid, fl.gridf, 0);
        ci = (int)max(-3L, min(q.ci, (long)fl.gridf.nx + 2));
        cj = (int)max(-3L, min(q.cj, (long)fl.gridf.ny + 2));
        ck = (int)max(-3L, min(q.ck, (long)fl.gridf.nz + 2));
        have_cell = true;
      }
      CellAt at;
      if (!cell_at(cull[item >> 4].key, fl.cell_off, fl.gridf, at)) continue;   // not binned any more
      const int dx = at.x - ci + 1, dy = at.y - cj + 1, dz = at.z - ck + 1;
      if ((unsigned)dx > 2u || (unsigned)dy > 2u || (unsigned)dz > 2u) continue;   // not a neighbour cell
      if (ncand == kListCap) return -1;
      const unsigned code = (item & 15u) << 5 | (unsigned)(9 * dx + 3 * dy + dz);
      int i = ncand++;
      for (; i > 0 && (unsigned)(pl.cand[i - 1][lane] >> 6) > code; i--) pl.cand[i][lane] = pl.cand[i - 1][lane];
      pl.cand[i][lane] = (unsigned short)(code << 6 | (unsigned)(e0 + k));
    }
  }
  return ncand;
}

// Boundary routines before and after the particles, as bits of NearLists::bnd.
__device__ __forceinline__ unsigned bits_before(bool aval) { return aval ? 0x00FFFFFFu : 0u; }
__device__ __forceinline__ unsigned bits_after(bool aval) { return aval ? 0x0F000000u : 0x00000FFFu; }

// Whether clump s must search for its pairs because its near list does not hold.
__device__ __forceinline__ bool must_search(long s, const DevScalars *d, const NearLists &near, int info) {
  return info < 0 || near.loose[s] <= d->tick;
}

// The list phase of k_lists_forces for one clump: its item list (see block_contacts) from its near
// list, in the reference's order, into `lists`; returns the item count (-1: more than the list
// holds, see slow_contacts) and their layout in lc.  A list that does not hold is replaced by a
// search that gives the same items.  overflow: the clump's list or items were too many.
__device__ __forceinline__ int lists_body(const Consts &c, const DevScalars *d, const int *__restrict__ flume,
                                          const NbrRec *__restrict__ nbr, const CullRec *__restrict__ cull,
                                          const int *__restrict__ start, const int *__restrict__ order,
                                          const long long *__restrict__ id, const NearLists &near,
                                          ContactLists lists, long s0, long n, Margins m, PassLists &pl,
                                          ListCounts &lc, bool &overflow) {
  const int lane = threadIdx.x & 31;
  const long s = s0 + blockIdx.x * (long)blockDim.x + threadIdx.x;
  lc.pre = lc.pair = 0;
  overflow = false;
  if (s >= n) return 0;
  const NbrRec &me = nbr[s];
  if (is_removed(*c.tp, me.rx, c.side_x)) return 0;
  const int info = near.info[s];
  const bool search = must_search(s, d, near, info);
  overflow = info < 0;
  const bool aval = c.phase == AF3D_PHASE_AVALANCHE;
  const float rad = __int_as_float(cull[s].s[0].w) * unit_power(-m.qs);
  unsigned *col = lists.items + s;
  const unsigned bnd = touching(search ? 0x0FFFFFFFu : near.bnd[s], me, rad, c);
  unsigned before = bnd & bits_before(aval), after = bnd & bits_after(aval);
  const int npre = __popc(before);
  int nitems = 0;
  for (; before; before &= before - 1u) col[n * nitems++] = kBndItem | ((unsigned)__ffs(before) - 1u);
  if (search) {
    nitems = search_items(s, d, flume, nbr, cull, start, order, id, near, m, n, col, nitems);
    if (nitems < 0) return -1;
  } else {
    const unsigned *list = near.items + s;
    const int np = near_pairs(s, info, d->flumes[flume[s]], me, cull, list, n, pl);
    if (np < 0 || nitems + np > kListCap) return -1;
#pragma unroll 1
    for (int i = 0; i < np; i++) col[n * nitems++] = list[(long)(pl.cand[i][lane] & 63u) * n];
  }
  lc.pair = nitems - npre;
  if (nitems + __popc(after) > kListCap) return -1;
  for (; after; after &= after - 1u) col[n * nitems++] = kBndItem | ((unsigned)__ffs(after) - 1u);
  lc.pre = npre;
  return nitems;
}

// Shared memory of the force kernel: the list phase, the force phase and the look-ahead's record
// staging run one after another.  Kept small because the SM's L1 cache gets what the resident
// blocks' shared memory leaves of 256 KB.
template <int NB>
union ForceShared {
  PassLists pl[NB / 32];
  BlockQueue<NB> bq;
  struct {
    double nbr[NB * kRecStride];
  } rec;
};

// sys_par.time += dt (avalanche_hst.cu:672), keeping the previous value for init_Verlet.  The
// flumes of an ensemble share dt and the clock.
__device__ __forceinline__ void advance_clock(DevScalars *d) {
  d->time_prev = d->time;
  d->time = d->time + d->flumes[0].sys.dt;
  d->tick++;
}

template <int NB, bool WRITE_FT, bool UNIFORM>
__device__ __forceinline__ void fused_body(const Consts &c, Planes P, Planes out, DevScalars *d,
                                           const int *__restrict__ flume, const NbrRec *__restrict__ nbr,
                                           const CullRec *__restrict__ cull, const Cells &cells,
                                           const int *__restrict__ order, const long long *__restrict__ id,
                                           const NearLists &near, ContactLists lists, int listed, ListCounts lc,
                                           bool overflow, long ntags, bool counted, long s0, long n,
                                           bool warm,
                                           const LookAhead &la, ForceShared<NB> &sh) {
  const long s = s0 + blockIdx.x * (long)blockDim.x + threadIdx.x;
  const bool valid = s < n;
  const long sv = valid ? s : n - 1;   // in-range slot for lanes past n (nothing is written for them)
  const int f = flume[sv];
  const bool removed = is_removed(*c.tp, nbr[sv].rx, c.side_x);
  V3 F = mk(0.0, 0.0, 0.0), T = mk(0.0, 0.0, 0.0);
  const bool aval = c.phase == AF3D_PHASE_AVALANCHE;
  if (valid && removed && aval) {
    const SlowSums r = removed_contacts(nbr + sv, (double)cull[sv].c.w, c);
    F = r.F;
    T = r.T;
  }
  const long bbase = s0 + blockIdx.x * (long)blockDim.x;
  if (!valid) listed = 0;
  const int active =
      block_contacts<NB, UNIFORM, WRITE_FT>(sh.bq, bbase, sv, valid && !removed, aval, c, d, flume, nbr, cull,
                                            cells.start, order, id, near, P.m, lists.items, lists.cnt != nullptr,
                                            listed, lc, n, F, T);
  if (la.nbr) __syncthreads();   // the force phase's shared memory is free for the record staging
  if (valid) {
    if (lists.cnt) lists.cnt[s] = pack_list_counts(listed, lc.pre, lc.pair);
    if (lists.ovf && listed < 0) *lists.ovf = 1;
    if (overflow) atomicAdd(&d->overflows, 1ull);   // rare: counted for the diagnostics
    if (counted) cells.occ[cull[s].key] = 0;
    if (WRITE_FT) {
      store3(P, FX, s, F);
      store3(P, TX, s, T);
    }
    // this step's predicted state, read again from the record (not held across the contacts);
    // its rotation rows from the RN planes when the previous pass predicted it
    const NbrRec &me = nbr[s];
    const V3 r = mk(me.rx, me.ry, me.rz);
    const V3 v = mk(me.vx, me.vy, me.vz), w = mk(me.wx, me.wy, me.wz);
    const int R0 = warm ? RN00 : R00;
    V3 Rx = load3(P, R0, s), Ry = load3(P, R0 + 3, s), Rz = load3(P, R0 + 6, s);
    if (warm && !la.keep) {   // commit the predicted state to the planes
      store3(P, RX, s, r);
      for (int k = 0; k < 4; k++) store3(P, S0X + 3 * k, s, mk(me.s[3 * k], me.s[3 * k + 1], me.s[3 * k + 2]));
      store3(P, R00, s, Rx);
      store3(P, R10, s, Ry);
      store3(P, R20, s, Rz);
    }
    V3 v2, w2, a, al;
    if (!removed) {
      get_accel_one<kCall>(F, T, v, w, Rx, Ry, Rz, P.p[MASS][s], P.p[ADRAG][s], load3(P, IXX, s), a, al, P.p[IMASS][s],
                    P.p[IINER][s], c.variant == AF3D_FRICTION_DEV);
      store3(P, AFX, s, a);
      store3(P, ALFX, s, al);
      const V3 ai = load3(P, AIX, s), ali = load3(P, ALIX, s);
      // finish_Verlet.cu:43-48
      v2 = mk(v.x + c.hdt * (a.x - ai.x), v.y + c.hdt * (a.y - ai.y), v.z + c.hdt * (a.z - ai.z));
      w2 = mk(w.x + c.hdt * (al.x - ali.x), w.y + c.hdt * (al.y - ali.y), w.z + c.hdt * (al.z - ali.z));
      if (!(finite_bits(a.x) && finite_bits(a.y) && finite_bits(a.z) && finite_bits(al.x) && finite_bits(al.y) &&
            finite_bits(al.z)))
        raise_status(d, AF3D_ERR_NAN);
    } else {
      v2 = mk(0.0, 0.0, 0.0);                 // finish_Verlet.cu:28-32
      w2 = w;
      a = al = mk(0.0, 0.0, 0.0);             // the reference leaves stale values here
      store3(P, AFX, s, a);
      store3(P, ALFX, s, al);
    }
    if (!la.keep) {
      store3(out, VX, s, v2);
      store3(out, WX, s, w2);
    }
    if (la.nbr) {
      // The next step's init_Verlet (removal test at this step's time, a_i = this a_f), cell key
      // (at the next step's time) and records, exactly as k_predict<1,1,1> would make them
      // after this step.
      const DevFlume &fl = d->flumes[f];
      const double t_next = *c.tp + d->flumes[0].sys.dt;   // k_advance_time's expression
      V3 rn = r, vn = v2, wn = w2, sp[4];
      if (is_removed(*c.tp, r.x, fl.sys.side.x)) {
        P.p[RAD][s] = 0.0;
        for (int k = 0; k < 4; k++) sp[k] = mk(me.s[3 * k], me.s[3 * k + 1], me.s[3 * k + 2]);
        store3(P, RN00, s, Rx);
        store3(P, RN10, s, Ry);
        store3(P, RN20, s, Rz);
      } else {
        predict_state<kCall>(rn, vn, wn, a, al, Rx, Ry, Rz, sp, P.p[RAD][s], fl.sys.dt, fl.sys.hdt, P.m.qs,
                      c.variant == AF3D_FRICTION_DEV);
        store3(P, RN00, s, Rx);
        store3(P, RN10, s, Ry);
        store3(P, RN20, s, Rz);
      }
      const long key = bucket_key(rn, fl, d, id[s], t_next);
      if (la.build) cells.key[s] = (int)key;
      {
        NbrRec q;
        CullRec cr;
        make_records(rn, vn, wn, sp, P.p[RAD][s], P.p[MSPH][s], P.p[MWALL][s], P.m, (int)key, q, cr);
        stage_nbr_record(q, sh.rec.nbr);
        la.cull[s] = cr;   // stored directly: staged too, it would set the block's shared memory size
        if (la.build) {
          cells.rank_tmp[s] = arrive_in_bucket(cells, key);
        } else {
          int4 old[4];
          for (int k = 0; k < 4; k++) old[k] = cull[s].s[k];
          if (keep_place(s, old, cr, fl, d, cells.occ_next, ntags, near, cells.start, order, P.m, d->tick + 1, n))
            la.cull[s].away = 1;
        }
      }
    }
  }
  warp_count(d, active);
  if (la.nbr) {
    __syncthreads();   // every neighbour record of the block is staged
    copy_nbr_records<NB>(bbase, n, la.nbr, sh.rec.nbr);
    // The pass's last block advances the clock for the step it has looked ahead to: every block
    // reads the time before its barrier above.
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicInc(&d->ticket, gridDim.x - 1) == gridDim.x - 1) advance_clock(d);
    }
  }
}

// One boundary routine added to the F, T planes (per-routine entry points).
__global__ void k_boundary(Planes P, DevScalars *d, const int *__restrict__ flume, int routine, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const Own o = own_from_planes(P, s);
  V3 F = load3(P, FX, s), T = load3(P, TX, s);
  const Consts c = load_consts(d, flume[s]);
  const bool removed = is_removed(*c.tp, o.r.x, c.side_x);
  bnd_routine(routine, o, removed, c, F, T);
  store3(P, FX, s, F);
  store3(P, TX, s, T);
}

// force_part for one sph_id (1..16) or all sixteen (0), added to the F, T planes.
__global__ void __launch_bounds__(kBlock) k_part(Planes P, DevScalars *d, const int *__restrict__ flume,
                                                 const NbrRec *__restrict__ nbr,
                                                 const CullRec *__restrict__ cull,
                                                 const int *__restrict__ start, int sph_id, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int f = flume[s];
  const Consts c = load_consts(d, f);
  const af3d_cell_par g = d->flumes[f].grid;
  const Own o = own_from_planes(P, s);
  if (is_removed(*c.tp, o.r.x, c.side_x)) return;
  V3 F = load3(P, FX, s), T = load3(P, TX, s);
  particle_contacts(s, o, c, g, d->flumes[f].cell_off, nbr, cull, start, nullptr, sph_id - 1, F, T);
  store3(P, FX, s, F);
  store3(P, TX, s, T);
}

__global__ void k_get_accel(Planes P, DevScalars *d, const int *__restrict__ flume, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  if (is_removed(d->time, P.p[RX][s], d->flumes[flume[s]].sys.side.x)) return;
  V3 a, al;
  get_accel_one(load3(P, FX, s), load3(P, TX, s), load3(P, VX, s), load3(P, WX, s), load3(P, R00, s),
                load3(P, R10, s), load3(P, R20, s), P.p[MASS][s], P.p[ADRAG][s], load3(P, IXX, s), a, al,
                P.p[IMASS][s], P.p[IINER][s], d->variant == AF3D_FRICTION_DEV);
  store3(P, AFX, s, a);
  store3(P, ALFX, s, al);
}

__global__ void k_finish_verlet(Planes P, DevScalars *d, const int *__restrict__ flume, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const af3d_system_par &sy = d->flumes[flume[s]].sys;
  const double hdt = sy.hdt;
  if (is_removed(d->time, P.p[RX][s], sy.side.x)) {
    store3(P, VX, s, mk(0.0, 0.0, 0.0));
    return;
  }
  V3 v = load3(P, VX, s), w = load3(P, WX, s);
  V3 af = load3(P, AFX, s), ai = load3(P, AIX, s), alf = load3(P, ALFX, s), ali = load3(P, ALIX, s);
  v.x += hdt * (af.x - ai.x);
  v.y += hdt * (af.y - ai.y);
  v.z += hdt * (af.z - ai.z);
  w.x += hdt * (alf.x - ali.x);
  w.y += hdt * (alf.y - ali.y);
  w.z += hdt * (alf.z - ali.z);
  store3(P, VX, s, v);
  store3(P, WX, s, w);
}

__global__ void k_clear_forces(Planes P, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  store3(P, FX, s, mk(0.0, 0.0, 0.0));
  store3(P, TX, s, mk(0.0, 0.0, 0.0));
}

__global__ void k_advance_time(DevScalars *d) { advance_clock(d); }

// ------------------------------------------------------------------ re-grid (cell_dim)

__device__ __forceinline__ unsigned long long ord(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double unord(unsigned long long k) {
  unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)u);
}

__global__ void k_bbox_init(DevScalars *d, int nflumes) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nflumes) return;
  unsigned long long *b = d->flumes[f].bbox;
  for (int i = 0; i < 3; i++) {
    b[i] = ~0ull;    // min x, y, z
    b[3 + i] = 0ull; // max x, y, z
  }
  b[6] = 0ull;       // max vx
  b[7] = ~0ull;      // min vz
}

// Min/max of clump centres, max vx and min vz over every clump of each flume (cell_dim.cu:21-54),
// warp-reduced when a warp's clumps belong to one flume.
__global__ void k_bbox_reduce(Planes P, DevScalars *d, const int *__restrict__ flume, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const long sv = s < n ? s : n - 1;
  const int f = flume[sv];
  unsigned long long mn[3], mx[3], vx, vz;
  for (int i = 0; i < 3; i++) mn[i] = mx[i] = ord(P.p[RX + i][sv]);
  vx = ord(P.p[VX][sv]);
  vz = ord(P.p[VZ][sv]);
  const int f0 = __shfl_sync(0xffffffffu, f, 0);
  const bool uniform = __all_sync(0xffffffffu, f == f0);
  if (uniform) {
    for (int off = 16; off; off >>= 1) {
      for (int i = 0; i < 3; i++) {
        mn[i] = min(mn[i], __shfl_xor_sync(0xffffffffu, mn[i], off));
        mx[i] = max(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], off));
      }
      vx = max(vx, __shfl_xor_sync(0xffffffffu, vx, off));
      vz = min(vz, __shfl_xor_sync(0xffffffffu, vz, off));
    }
  }
  if (!uniform || (threadIdx.x & 31) == 0) {
    unsigned long long *b = d->flumes[f].bbox;
    for (int i = 0; i < 3; i++) {
      atomicMin(&b[i], mn[i]);
      atomicMax(&b[3 + i], mx[i]);
    }
    atomicMax(&b[6], vx);
    atomicMin(&b[7], vz);
  }
}

// cell_dim.cu:56-66 padding and the grid derivation of avalanche_hst.cu:314-333, per flume, into
// the flume's pending grid.
__global__ void k_grid_derive(DevScalars *d, int nflumes) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nflumes) return;
  DevFlume &fl = d->flumes[f];
  if (fl.bbox[0] == ~0ull) {
    // A flume without clumps keeps its grid (a one-cell grid if it never had one): nothing is
    // binned there, and cell_dim would read a clump that does not exist.
    af3d_cell_par g = fl.grid;
    if (g.ncell3 <= 0) {
      g.rr_min = {0.0, 0.0, 0.0};
      g.rr_max = g.length = g.cell_side = g.cs_inv = {1.0, 1.0, 1.0};
      g.ncell = {1, 1, 1};
      g.ncell3 = 1;
      g.ntot = g.ntags;
    }
    fl.pending = g;
    return;
  }
  const af3d_system_par &sy = fl.sys;
  const double rgyr = 0.5 * sy.gyr_max, ddt = 2000.0 * sy.dt;
  const double vxmax = unord(fl.bbox[6]), vzmin = unord(fl.bbox[7]);
  V3 hi = mk(unord(fl.bbox[3]), unord(fl.bbox[4]), unord(fl.bbox[5]));
  V3 lo = mk(unord(fl.bbox[0]), unord(fl.bbox[1]), unord(fl.bbox[2]));
  hi.x += 1.05 * rgyr + vxmax * ddt;
  lo.x -= 1.05 * rgyr;
  hi.y += 1.05 * rgyr;
  lo.y -= 1.05 * rgyr;
  hi.z += 1.05 * rgyr;
  lo.z -= 1.05 * rgyr - vzmin * ddt;
  af3d_cell_par g = fl.grid;
  const double dist = kGYR + (double)0.05f;   // avalanche_hst.cu:115 adds a float literal
  g.rr_max = {hi.x, hi.y, hi.z};
  g.rr_min = {lo.x, lo.y, lo.z};
  g.length = {hi.x - lo.x, hi.y - lo.y, hi.z - lo.z};
  g.ncell.x = (long)(g.length.x / (dist * sy.rmax));
  g.ncell.y = (long)(g.length.y / (dist * sy.rmax));
  g.ncell.z = (long)(g.length.z / (dist * sy.rmax));
  g.cell_side.x = g.length.x / ((double)g.ncell.x);
  g.cell_side.y = g.length.y / ((double)g.ncell.y);
  g.cell_side.z = g.length.z / ((double)g.ncell.z);
  g.cs_inv.x = 1.0 / g.cell_side.x;
  g.cs_inv.y = 1.0 / g.cell_side.y;
  g.cs_inv.z = 1.0 / g.cell_side.z;
  g.ncell3 = g.ncell.x * g.ncell.y * g.ncell.z;
  g.ntot = g.ncell3 * g.ntags;
  fl.pending = g;
}

// Commit the pending grids with their bucket offsets when every grid is non-empty and the
// buckets fit; otherwise record the buckets needed (-1: an empty grid) and keep the old grids.
__global__ void k_grid_commit(DevScalars *d, int nflumes, long n, long bucket_cap) {
  long long total = 0;
  bool ok = true;
  for (int f = 0; f < nflumes; f++) {
    const long long c = d->flumes[f].pending.ncell3;
    ok = ok && c > 0;
    total += c > 0 ? c : 0;
  }
  if (!ok) {
    d->pending = -1;
    return;
  }
  if (total + n + 1 > bucket_cap) {
    d->pending = total;
    return;
  }
  long long off = 0;
  for (int f = 0; f < nflumes; f++) {
    d->flumes[f].grid = d->flumes[f].pending;
    d->flumes[f].gridf = grid_floats(d->flumes[f].grid);
    d->flumes[f].cell_off = off;
    off += d->flumes[f].grid.ncell3;
  }
  d->ncell_total = total;
  d->pending = 0;
}

// ------------------------------------------------------------------ diagnostics

__global__ void k_contact_pairs(Planes P, DevScalars *d, const int *__restrict__ flume,
                                const NbrRec *__restrict__ nbr, const CullRec *__restrict__ cull,
                                const int *__restrict__ start, const long long *__restrict__ id,
                                long long *out, unsigned long long *count, long cap, int active_only,
                                long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int f = flume[s];
  const Consts c = load_consts(d, f);
  const af3d_cell_par g = d->flumes[f].grid;
  const Own o = own_from_planes(P, s);
  if (is_removed(*c.tp, o.r.x, c.side_x)) return;
  const CullRec me = cull[s];
  const Search q = search_centre(o.r, g, d->flumes[f].cell_off);
  for_neighbour_slots(q, g, start, nullptr, [&](int t) {
    if (t == s) return;
    unsigned m = pair_mask(me, cull[t]);
    while (m) {
      const int p = __ffs(m) - 1;
      m &= m - 1;
      V3 F = mk(0.0, 0.0, 0.0), T = mk(0.0, 0.0, 0.0);
      const int r = part_pair(o.r, o.v, o.w, o.s[p & 3], o.rad, o.msph, nbr[t], p >> 2, c, false, F, T);
      if (r == 2 || (r == 1 && !active_only)) {
        unsigned long long k = atomicAdd(count, 1ull);
        if ((long)k < cap) {
          out[3 * k] = id[s];
          out[3 * k + 1] = id[t];
          out[3 * k + 2] = p + 1;
        }
      }
    }
  });
}

// Bucket of every clump by id (-1 when not binned): the flume's cell offset plus the cell index.
__global__ void k_cells_by_id(const int *__restrict__ key, const long long *__restrict__ id,
                              const DevScalars *d, long long *cell_of_id, long n) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int k = key[s];
  cell_of_id[id[s]] = k < d->ncell_total ? k : -1;
}

}  // namespace

// ------------------------------------------------------------------ launchers

// Built twice: the exact launchers in namespace af3d, and (with -DAF3D_FAST) the fast-mode
// build of the same kernels, whose predictor and force launchers the context uses in fast mode.
#ifdef AF3D_FAST
namespace fast {
#endif

void launch_predict(const Launch &L, Planes cur, DevScalars *d, bool predict, bool keys, bool t_prev,
                    Cells cells, const long long *id, const int *flume, long ntags, NearLists near, const int *order,
                    bool count_only, NbrRec *nbr, CullRec *cull, long s0, long count) {
  // slots [s0, s0 + count) of L.n (count < 0: to the end); s0 a multiple of kBlock
  const long m = count < 0 ? L.n - s0 : std::min(count, L.n - s0);
  if (L.n <= 0 || m <= 0 || s0 % kBlock != 0) return;
  const unsigned g = grid_for(m);
  auto run = [&](auto kernel) {
    kernel<<<g, kBlock, 0, L.st>>>(cur, d, t_prev, cells, id, flume, ntags, near, order, count_only, nbr, cull, s0,
                                   L.n);
  };
  if (predict && keys && nbr) run(k_predict<true, true, true>);
  else if (predict && keys) run(k_predict<true, true, false>);
  else if (predict) run(k_predict<true, false, false>);
  else if (keys && nbr) run(k_predict<false, true, true>);
  else if (keys) run(k_predict<false, true, false>);
}

void launch_permute_records(const Launch &L, Planes src, Planes dst, const int *perm, const int *key,
                            const long long *id_src, long long *id_dst, const int *fl_src, int *fl_dst,
                            NbrRec *nbr, CullRec *cull, bool ft) {
  if (L.n <= 0) return;
  k_permute<<<grid_for(L.n, kPermBlock), kPermBlock, 0, L.st>>>(src, dst, perm, key, id_src, id_dst, fl_src, fl_dst,
                                                                nbr, cull, ft, L.n);
}

void launch_build_records(const Launch &L, Planes cur, NbrRec *nbr, CullRec *cull) {
  if (L.n <= 0) return;
  k_permute<<<grid_for(L.n, kPermBlock), kPermBlock, 0, L.st>>>(cur, cur, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                                nullptr, nbr, cull, true, L.n);
}

// The contact items and the force pass of one block's clumps in one launch: the block takes its
// clumps' item lists from their near lists, then processes them.  The lists pass through global
// memory (the block's own entries, visible to its threads after the barrier).
template <int NB, int MINB, bool WRITE_FT, bool UNIFORM>
__global__ void __launch_bounds__(NB, MINB)
    k_lists_forces(const __grid_constant__ Planes P, const __grid_constant__ Planes out, DevScalars *d,
                   const int *__restrict__ flume, const NbrRec *__restrict__ nbr,
                   const CullRec *__restrict__ cull, const __grid_constant__ Cells cells,
                   const int *__restrict__ order, const long long *__restrict__ id,
                   const __grid_constant__ NearLists near, ContactLists lists, long ntags, bool counted,
                   const __grid_constant__ Consts kc, bool warm, const __grid_constant__ LookAhead la, long s0,
                   long n) {
  __shared__ ForceShared<NB> sh;
  ListCounts lc;
  bool overflow;
  auto body = [&](const Consts &c) {
    const int listed = lists_body(c, d, flume, nbr, cull, cells.start, order, id, near, lists, s0, n, P.m,
                                  sh.pl[threadIdx.x >> 5], lc, overflow);
    overflow = overflow || listed < 0;
    __syncthreads();
    fused_body<NB, WRITE_FT, UNIFORM>(c, P, out, d, flume, nbr, cull, cells, order, id, near, lists, listed, lc,
                                      overflow, ntags, counted, s0, n, warm, la, sh);
  };
  if constexpr (UNIFORM) {
    body(kc);
  } else {
    // the flume's constants read where they lie (a reference, not a register copy)
    const long s = s0 + blockIdx.x * (long)blockDim.x + threadIdx.x;
    body(d->flumes[flume[s < n ? s : n - 1]].c);
  }
}

#include "af3d_wide.cuh"

void launch_lists_forces(const Launch &L, Planes cur, Planes out, DevScalars *d, const int *flume,
                         const NbrRec *nbr, const CullRec *cull, Cells cells, const int *order, const long long *id,
                         NearLists near, ContactLists lists, long ntags, bool write_ft, bool counted, bool wide,
                         const Consts *uniform, bool warm, LookAhead look, long s0, long count, int shape) {
  // slots [s0, s0 + count) of L.n (count < 0: to the end); s0 a multiple of the shape's block,
  // so the launch's blocks are those of the whole pass
  const long m = count < 0 ? L.n - s0 : std::min(count, L.n - s0);
  if (L.n <= 0 || m <= 0 || shape < 0 || shape >= kForceShapes || s0 % kForceShapeBlock[shape] != 0) return;
  static_assert(kForceShapes == 4 && kForceShapeBlock[0] == 128 && kForceShapeBlock[1] == 96 &&
                    kForceShapeBlock[2] == 64 && kForceShapeBlock[3] == 192, "the instantiated shapes");
  const Consts kc = uniform ? *uniform : Consts{};
  if (wide) {
    auto run = [&](auto kernel) {
      kernel<<<grid_for(m, kWide), kWideThreads, 0, L.st>>>(cur, out, d, flume, nbr, cull, cells, order, id, near,
                                                           lists, ntags, write_ft, counted, kc, warm, look, s0, L.n);
    };
    if (uniform) run(k_forces_wide<true>);
    else run(k_forces_wide<false>);
    return;
  }
  auto run = [&](auto kernel, int nb) {
    kernel<<<grid_for(m, nb), nb, 0, L.st>>>(cur, out, d, flume, nbr, cull, cells, order, id, near, lists, ntags,
                                             counted, kc, warm, look, s0, L.n);
  };
  auto shaped = [&](auto ft, auto uni) {
    constexpr bool FT = decltype(ft)::value, UNI = decltype(uni)::value;
    if (shape == 0) run(k_lists_forces<128, kForceShapeMinb[0], FT, UNI>, 128);
    else if (shape == 1) run(k_lists_forces<96, kForceShapeMinb[1], FT, UNI>, 96);
    else if (shape == 2) run(k_lists_forces<64, kForceShapeMinb[2], FT, UNI>, 64);
    else run(k_lists_forces<192, kForceShapeMinb[3], FT, UNI>, 192);
  };
  if (uniform) {
    if (write_ft) shaped(std::true_type{}, std::true_type{});
    else shaped(std::false_type{}, std::true_type{});
  } else {
    if (write_ft) shaped(std::true_type{}, std::false_type{});
    else shaped(std::false_type{}, std::false_type{});
  }
}

void launch_boundary(const Launch &L, Planes cur, DevScalars *d, const int *flume, int routine) {
  if (L.n <= 0) return;
  k_boundary<<<grid_for(L.n), kBlock, 0, L.st>>>(cur, d, flume, routine, L.n);
}

void launch_part(const Launch &L, Planes cur, DevScalars *d, const int *flume, const NbrRec *nbr,
                 const CullRec *cull, const int *start, int sph_id) {
  if (L.n <= 0) return;
  k_part<<<grid_for(L.n), kBlock, 0, L.st>>>(cur, d, flume, nbr, cull, start, sph_id, L.n);
}

void launch_get_accel(const Launch &L, Planes cur, DevScalars *d, const int *flume) {
  if (L.n <= 0) return;
  k_get_accel<<<grid_for(L.n), kBlock, 0, L.st>>>(cur, d, flume, L.n);
}

void launch_finish_verlet(const Launch &L, Planes cur, DevScalars *d, const int *flume) {
  if (L.n <= 0) return;
  k_finish_verlet<<<grid_for(L.n), kBlock, 0, L.st>>>(cur, d, flume, L.n);
}

void launch_clear_forces(const Launch &L, Planes cur) {
  if (L.n <= 0) return;
  k_clear_forces<<<grid_for(L.n), kBlock, 0, L.st>>>(cur, L.n);
}

void launch_advance_time(cudaStream_t st, DevScalars *d) { k_advance_time<<<1, 1, 0, st>>>(d); }

void launch_regrid(const Launch &L, Planes cur, DevScalars *d, const int *flume, int nflumes,
                   long bucket_cap) {
  const unsigned gf = (unsigned)((nflumes + 127) / 128);
  k_bbox_init<<<gf, 128, 0, L.st>>>(d, nflumes);
  if (L.n > 0) k_bbox_reduce<<<grid_for(L.n, 256), 256, 0, L.st>>>(cur, d, flume, L.n);
  k_grid_derive<<<gf, 128, 0, L.st>>>(d, nflumes);
  k_grid_commit<<<1, 1, 0, L.st>>>(d, nflumes, L.n, bucket_cap);
}

void launch_commit_grids(cudaStream_t st, DevScalars *d, int nflumes, long n, long bucket_cap) {
  k_grid_commit<<<1, 1, 0, st>>>(d, nflumes, n, bucket_cap);
}

void launch_aos_to_planes(const Launch &L, const af3d_particle *aos, const double *acc,
                          const double *anga, const int *flume_of_id, Planes cur, long long *id,
                          int *flume, bool keep_order, long s0, long count) {
  const long m = count < 0 ? L.n - s0 : std::min(count, L.n - s0);
  if (L.n <= 0 || m <= 0) return;
  k_aos_to_planes<<<grid_for(m), kBlock, 0, L.st>>>(aos, acc, anga, flume_of_id, cur, id, flume, keep_order, s0,
                                                    L.n);
}

void launch_planes_to_aos(const Launch &L, Planes cur, const long long *id, const int *flume,
                          af3d_particle *aos, double *acc, double *anga, DevScalars *d, long s0, long count) {
  const long m = count < 0 ? L.n - s0 : std::min(count, L.n - s0);
  if (L.n <= 0 || m <= 0) return;
  k_planes_to_aos<<<grid_for(m), kBlock, 0, L.st>>>(cur, id, flume, aos, acc, anga, d, s0, L.n);
}

void launch_contact_pairs(const Launch &L, Planes cur, DevScalars *d, const int *flume,
                          const NbrRec *nbr, const CullRec *cull, const int *start,
                          const long long *id, long long *out, unsigned long long *count, long cap,
                          int active) {
  if (L.n <= 0) return;
  k_contact_pairs<<<grid_for(L.n), kBlock, 0, L.st>>>(cur, d, flume, nbr, cull, start, id, out, count, cap,
                                                      active, L.n);
}

void launch_cells_by_id(const Launch &L, const int *key, const long long *id, DevScalars *d,
                        long long *cell_of_id) {
  if (L.n <= 0) return;
  k_cells_by_id<<<grid_for(L.n), kBlock, 0, L.st>>>(key, id, d, cell_of_id, L.n);
}

#ifdef AF3D_FAST
}  // namespace fast
#endif

}  // namespace af3d
