// af3d_cellwalk.cuh -- the FP32 culling tests and the neighbour-cell walk of the sorted cell
// list, shared by the step kernels and the adjoint kernels.
#pragma once

#include "af3d_physics.cuh"

namespace af3d {
namespace {

constexpr float kCullSlack = 1.0f + 3.814697265625e-06f;  // 1 + 2^-18

// Squared distance for the conservative FP32 culling tests (fused multiply-adds: their rounding
// error is below the unfused one, and the tests' 2^-18 slack covers either).
__device__ __forceinline__ float d2f(float4 a, float4 b) {
  const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
  return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// A clump's own side of the sphere tests: its spheres relative to its first one in units (exact in
// FP32: below 2^22 units), that sphere's centre and the sphere radius in units.
struct OwnSpheres {
  float x[4], y[4], z[4], rad;
  int cx, cy, cz;
};

// 2^e, |e| <= 126.
__device__ __forceinline__ float unit_power(int e) { return __int_as_float((127 + e) << 23); }

// a - b of two coordinates in units, |a - b| < 2^22, as a float (exact): the integer difference
// placed in the mantissa of 1.5 x 2^23.
__device__ __forceinline__ float unit_difference(int a, int b) {
  return __int_as_float(0x4B400000 + (a - b)) - 12582912.0f;
}

__device__ __forceinline__ OwnSpheres own_spheres(const CullRec &m) {
  OwnSpheres o;
  o.rad = __int_as_float(m.s[0].w);
  o.cx = m.s[0].x; o.cy = m.s[0].y; o.cz = m.s[0].z;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    o.x[k] = unit_difference(m.s[k].x, o.cx);
    o.y[k] = unit_difference(m.s[k].y, o.cy);
    o.z[k] = unit_difference(m.s[k].z, o.cz);
  }
  return o;
}

// 16-bit mask of the sphere pairs closer than `margin` units: bit p = sph_id - 1 = 4 * (partner
// sphere) + (own sphere).  The truncated coordinates leave each difference within 2 units of the
// exact one (so a distance within 2 sqrt(3)), which the records' radii, inflated by 2 units each,
// cover; the FP32 squares round by less than the 2^-20 slack.  An infinite radius (kCullMaxUnits)
// lets every pair pass whatever the differences are.
__device__ __forceinline__ unsigned sphere_mask(const OwnSpheres &o, const int4 *ms, float margin) {
  const float r = o.rad + __int_as_float(ms[0].w) + margin;
  const float r2 = r * r * (1.0f + 9.5367431640625e-07f);
  unsigned mask = 0u;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float px = unit_difference(ms[j].x, o.cx), py = unit_difference(ms[j].y, o.cy),
                pz = unit_difference(ms[j].z, o.cz);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float dx = px - o.x[k], dy = py - o.y[k], dz = pz - o.z[k];
      if (!(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > r2)) mask |= 1u << (4 * j + k);
    }
  }
  return mask;
}

// The mask of the pairs that may overlap, after the FP32 centre test of the bounding spheres.
__device__ __forceinline__ unsigned pair_mask(const CullRec &me, const CullRec &m) {
  const float lim = me.c.w + m.c.w;
  if (d2f(me.c, m.c) > lim * lim * kCullSlack) return 0u;
  return sphere_mask(own_spheres(me), m.s, 0.0f);
}

struct Search {
  long ci, cj, ck;
  long long off;   // the flume's first cell bucket
};

// Search-centre cell of force_part.cu:77-85: (long)((x - xmin)/side).  The quotient is first
// estimated with the reciprocal cs_inv = 1/side.  For |q| < 1e6 the estimate is within
// 4.4e-16 |Q| < 1e-9 of the true quotient Q, so when it is more than 1e-9 away from an integer,
// Q and its correctly rounded value lie in the same open unit interval and truncate to the same
// index; the division is only carried out near a cell boundary.  Same index as the reference.
__device__ __forceinline__ long search_axis(double x, double xmin, double side, double inv, long n) {
  const double dx = x - xmin;
  const double q = dx * inv;
  const double fl = floor(q);
  long i;
  if (q - fl > 1e-9 && q - fl < 1.0 - 1e-9 && fabs(q) < 1.0e6)   // |q - Q| <= 4.4e-16 |Q| < 1e-9
    i = (long)q;
  else
    i = (long)(dx / side);
  if (i == n) i--;
  return i;
}

// The same index from the FP32 culling coordinate xf and the FP32 grid copies: the estimate
// q = (xf - xmin) * inv is within 2^-24 ((|x| + |xmin|) inv + 3 q) (1 + 2^-20) of the exact
// quotient (four roundings), so when it is farther than eight times that bound from every
// integer it truncates to the reference's index; otherwise (and for q near 0 or below) the FP64
// path decides.
__device__ __forceinline__ long search_axis_f(float xf, float xminf, float invf, double x, double xmin, double side,
                                              double inv, long n) {
  const float q = (xf - xminf) * invf;
  const float E = 4.76837158203125e-07f * ((fabsf(xf) + fabsf(xminf)) * invf + 3.0f * q);   // 2^-21 (...)
  if (q > E && q < 4.0e6f) {
    const float tq = truncf(q);
    const float fr = q - tq;   // exact: q and tq lie within a factor two of each other
    if (fr > E && fr < 1.0f - E) {
      long i = (long)tq;
      if (i == n) i--;
      return i;
    }
  }
  return search_axis(x, xmin, side, inv, n);
}

__device__ __forceinline__ Search search_centre_f(float4 cf, V3 r, const af3d_cell_par &g, const GridF &gf,
                                                  long long off) {
  Search q;
  q.off = off;
  q.ci = search_axis_f(cf.x, gf.xmin, gf.ix, r.x, g.rr_min.x, g.cell_side.x, g.cs_inv.x, g.ncell.x);
  q.cj = search_axis_f(cf.y, gf.ymin, gf.iy, r.y, g.rr_min.y, g.cell_side.y, g.cs_inv.y, g.ncell.y);
  q.ck = search_axis_f(cf.z, gf.zmin, gf.iz, r.z, g.rr_min.z, g.cell_side.z, g.cs_inv.z, g.ncell.z);
  return q;
}

__device__ __forceinline__ Search search_centre(V3 r, const af3d_cell_par &g, long long off) {
  Search q;
  q.off = off;
  q.ci = search_axis(r.x, g.rr_min.x, g.cell_side.x, g.cs_inv.x, g.ncell.x);
  q.cj = search_axis(r.y, g.rr_min.y, g.cell_side.y, g.cs_inv.y, g.ncell.y);
  q.ck = search_axis(r.z, g.rr_min.z, g.cell_side.z, g.cs_inv.z, g.ncell.z);
  return q;
}

// Visit the occupied slots of the 27 neighbour cells in the reference's order
// (idel, jdel, kdel from -1 to 1; force_part.cu:88-106); slots inside a cell are in id order.
// `order` (may be null): the slot of the clump at each position of the (cell, id) order, for
// steps that do not move the clumps into that order.
template <typename F>
__device__ __forceinline__ void for_neighbour_slots(const Search &q, const af3d_cell_par &g,
                                                    const int *__restrict__ start,
                                                    const int *__restrict__ order, F &&f) {
#pragma unroll 1
  for (int di = -1; di <= 1; di++)
#pragma unroll 1
    for (int dj = -1; dj <= 1; dj++)
#pragma unroll 1
      for (int dk = -1; dk <= 1; dk++) {
        const long in = q.ci + di, jn = q.cj + dj, kn = q.ck + dk;
        if (in < 0 || jn < 0 || kn < 0 || in >= g.ncell.x || jn >= g.ncell.y || kn >= g.ncell.z)
          continue;
        const long c = q.off + in + g.ncell.x * (jn + g.ncell.y * kn);
        const int t0 = __ldg(&start[c]), t1 = __ldg(&start[c + 1]);
#pragma unroll 1
        for (int t = t0; t < t1; t++) f(order ? __ldg(&order[t]) : t);
      }
}

// The same visit with every cell boundary loaded up front.  The three cells of one (jdel, kdel)
// row are consecutive in the linear cell index, so their members form one slot range split by
// four start[] values; the 9 rows x 4 boundaries are issued as independent loads before the walk
// (instead of 27 dependent round trips), then the cells are walked in the reference's order.
template <typename F>
__device__ __forceinline__ void for_neighbour_slots_pre(const Search &q, const af3d_cell_par &g,
                                                        const int *__restrict__ start,
                                                        const int *__restrict__ order, F &&f) {
  int bnd[9][4];
  const long x0 = q.ci - 1;
#pragma unroll
  for (int r = 0; r < 9; r++) {
    const long jn = q.cj + (r / 3 - 1), kn = q.ck + (r % 3 - 1);
    const bool row_ok = jn >= 0 && kn >= 0 && jn < g.ncell.y && kn < g.ncell.z;
    const long rb = q.off + g.ncell.x * (jn + g.ncell.y * kn);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      // boundary e of the row: start of cell x0 + e, clamped into the row (empty cells outside)
      long x = x0 + e;
      x = x < 0 ? 0 : (x > g.ncell.x ? g.ncell.x : x);
      bnd[r][e] = row_ok ? __ldg(&start[rb + x]) : 0;
    }
  }
#pragma unroll 1
  for (int di = 0; di < 3; di++)
#pragma unroll 1
    for (int r = 0; r < 9; r++) {
      const int t0 = bnd[r][di], t1 = bnd[r][di + 1];
#pragma unroll 1
      for (int t = t0; t < t1; t++) f(order ? __ldg(&order[t]) : t);
    }
}

constexpr unsigned kBndItem = 0xFFFFFF00u;   // boundary item: kBndItem | routine << 2 | sphere

// Cell (x, y, z) of bucket `key` of a flume with cell offset `off`; false for a bucket of another
// flume or of a clump that is not binned.
struct CellAt {
  int x, y, z;
};
__device__ __forceinline__ bool cell_at(int key, long long off, const GridF &g, CellAt &c) {
  const int nxy = g.nx * g.ny;
  const long long lin = (long long)key - off;
  if (lin < 0 || lin >= (long long)nxy * g.nz) return false;
  const unsigned l = (unsigned)lin;
  c.z = (int)(l / (unsigned)nxy);
  const unsigned r = l - (unsigned)(c.z * nxy);
  c.y = (int)(r / (unsigned)g.nx);
  c.x = (int)(r - (unsigned)(c.y * g.nx));
  return true;
}

// Visits the slots that the last built cell order holds in the 5 x 5 x 5 cells around `c`.
template <typename F>
__device__ __forceinline__ void for_slots_around(const CellAt &c, const GridF &g, long long off,
                                                 const int *__restrict__ start, const int *__restrict__ order, F &&f) {
  const int x0 = max(c.x - 2, 0), x1 = min(c.x + 2, g.nx - 1);
#pragma unroll 1
  for (int z = max(c.z - 2, 0); z <= min(c.z + 2, g.nz - 1); z++)
#pragma unroll 1
    for (int y = max(c.y - 2, 0); y <= min(c.y + 2, g.ny - 1); y++) {
      const int *row = start + off + (long long)g.nx * (y + (long long)g.ny * z);
      const int t1 = __ldg(row + x1 + 1);
#pragma unroll 1
      for (int t = __ldg(row + x0); t < t1; t++) f(order ? __ldg(&order[t]) : t);
    }
}

// Clump s, in cell `c` of key `key`, may meet clumps that their near lists do not hold: those around it as
// built search for themselves from tick `from` on (a plain look first: most were marked before).
__device__ __forceinline__ void mark_around(const CellAt &c, const GridF &g, long long off,
                                            const int *__restrict__ start, const int *__restrict__ order, int *loose,
                                            int from) {
  for_slots_around(c, g, off, start, order, [&](int t) {
    if (loose[t] > from) atomicMin(&loose[t], from);
  });
}

// Clump s joins the chain of its cell's key for tick `from`; once for a clump and tick.
__device__ __forceinline__ void join_chain(const NearLists &near, long s, int key, int from, long n) {
  const long half = (from & 1) * n;
  const unsigned long long old =
      atomicExch(&near.chain[half + key % n], (unsigned long long)(unsigned)from << 32 | (unsigned)s);
  near.chain_next[half + s] = (unsigned)(old >> 32) == (unsigned)from ? (int)(unsigned)old : -1;
}

// Visits the runaways in cell `key` at tick `tick`.
template <typename F>
__device__ __forceinline__ void for_chain(const NearLists &near, const CullRec *__restrict__ cull, int key, int tick,
                                          long n, F &&f) {
  const long half = (tick & 1) * n;
  const unsigned long long head = near.chain[half + key % n];
  int t = (unsigned)(head >> 32) == (unsigned)tick ? (int)(unsigned)head : -1;
#pragma unroll 1
  for (; t >= 0; t = near.chain_next[half + t])
    if (cull[t].key == key) f(t);
}

// A clump's list layout: `pre` boundary items, then `pair` particle items, then the rest.
struct ListCounts {
  int pre, pair;
};

}  // namespace
}  // namespace af3d
