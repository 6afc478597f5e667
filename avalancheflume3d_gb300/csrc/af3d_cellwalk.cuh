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

// The cells that a bounding sphere of `reach` around `c` meets, in FP32 with slack.
struct CellRange {
  int x0, x1, y0, y1, z0, z1;
};
__device__ __forceinline__ CellRange cells_within(float4 c, float reach, const GridF &g) {
  auto range = [&](float x, float xmin, float inv, int cells, int &lo, int &hi) {
    const float q = (x - xmin) * inv, r = reach * inv;
    const float e = 2e-6f * ((fabsf(x) + fabsf(xmin)) * inv + fabsf(q) + r + 1.0f);
    lo = (int)fminf(fmaxf(floorf(q - r - e), 0.0f), (float)(cells - 1));
    hi = (int)fminf(fmaxf(floorf(q + r + e), 0.0f), (float)(cells - 1));
  };
  CellRange b;
  range(c.x, g.xmin, g.ix, g.nx, b.x0, b.x1);
  range(c.y, g.ymin, g.iy, g.ny, b.y0, b.y1);
  range(c.z, g.zmin, g.iz, g.nz, b.z0, b.z1);
  return b;
}

// The largest bounding radius and allowance of a clump of the near lists, about the centre c.
__device__ __forceinline__ float partner_reach(float4 c, const Margins &m) {
  return m.most + 1e-6f * (fabsf(c.x) + fabsf(c.y) + fabsf(c.z) + 20.0f) + m.cap;
}

// Visits the slots of the clumps that may touch a clump with the bounding sphere c (radius c.w) in cell
// `at` and are not away: in the last built cell order, where none of them is further than its allowance
// from its place.  Whatever c.w is, that is the cells next to `at` (contacts are between neighbour
// cells) and as many more as an allowance spans.
template <typename F>
__device__ __forceinline__ void for_slots_around(float4 c, const CellAt &at, const Margins &m, const GridF &g,
                                                 long long off, const int *__restrict__ start,
                                                 const int *__restrict__ order, F &&f) {
  CellRange b = cells_within(c, (c.w + partner_reach(c, m)) * (1.0f + 1e-5f), g);
  auto clip = [&](int &lo, int &hi, int k, float inv) {
    const int more = 2 + (int)fminf(m.cap * inv, 1e6f);
    lo = max(lo, k - more);
    hi = min(hi, k + more);
  };
  clip(b.x0, b.x1, at.x, g.ix);
  clip(b.y0, b.y1, at.y, g.iy);
  clip(b.z0, b.z1, at.z, g.iz);
  if (b.x0 > b.x1 || b.y0 > b.y1 || b.z0 > b.z1) return;
  const int ny = b.y1 - b.y0 + 1, rows = ny * (b.z1 - b.z0 + 1);
#pragma unroll 1
  for (int r0 = 0; r0 < rows; r0 += 4) {   // four rows' ends side by side
    int k[4], end[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      k[q] = end[q] = 0;
      if (r0 + q < rows) {
        const int z = (r0 + q) / ny, y = r0 + q - z * ny;
        const int *row = start + off + (long long)g.nx * (b.y0 + y + (long long)g.ny * (b.z0 + z));
        k[q] = __ldg(row + b.x0);
        end[q] = __ldg(row + b.x1 + 1);
      }
    }
#pragma unroll 1
    for (int q = 0; q < 4; q++)   // (one copy of f's code)
#pragma unroll 1
      for (; k[q] < end[q]; k[q]++) f(order ? __ldg(&order[k[q]]) : k[q]);
  }
}

// Clump s with the bounding sphere c, in cell `at` of bucket `key`, is away at tick `tick`: it joins the
// chain of its cell, and the clumps around it, whose near lists may not hold it, are loose (a plain
// look first: most were marked before).  Once for a clump and tick.  Not inlined: rare.
static __device__ __noinline__ void go_away(long s, float4 c, int key, CellAt at, const Margins &m, const DevFlume &fl,
                                            DevScalars *d, const int *__restrict__ start,
                                            const int *__restrict__ order, const NearLists &near, int tick, long n) {
  const long half = (tick & 1) * n;
  const unsigned long long old =
      atomicExch(&near.chain[half + key % n], (unsigned long long)(unsigned)tick << 32 | (unsigned)s);
  near.chain_next[half + s] = (unsigned)(old >> 32) == (unsigned)tick ? (int)(unsigned)old : -1;
  if (d->away > tick) atomicMin(&d->away, tick);
  auto mark = [&](int t) {
    if (near.loose[t] > tick) atomicMin(&near.loose[t], tick);
  };
  for_slots_around(c, at, m, fl.gridf, fl.cell_off, start, order, mark);
  mark((int)s);
}

// Visits the clumps away in cell `key` at tick `tick`.
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
