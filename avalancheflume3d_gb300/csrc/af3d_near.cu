// af3d_near.cu -- the near lists: per clump, the sphere pairs and boundary spheres that may touch
// while no clump moves farther than its allowance (NearLists in af3d_internal.h).
//
// Integer and FP32 work on the culling records; built from the sorted cell list once every
// 2 to 16 steps (list_interval).
#include "af3d_cellwalk.cuh"

namespace af3d {

namespace {

constexpr int kNearClumps = 32;   // clumps a block
constexpr int kNearBlock = 128;
constexpr int kPartners = 32;     // partners whose bounding spheres may meet; with more, the per-clump search
constexpr int kSide = 2;          // partners a thread tests side by side
constexpr int kWarpPartners = 24;  // ... that one warp of the block finds

struct NearShared {
  unsigned pos[4][kWarpPartners][kNearClumps];   // [warp][entry][clump] position in the sorted order, then slot
  int count[4][kNearClumps];
  unsigned id[kPartners][kNearClumps];           // the clump's partners, all warps': id (~0: the clump itself)
  unsigned char pairs[kPartners][kNearClumps];   // ... and how many sphere pairs are near
};

// A block's four warps share 32 clumps (lane = clump).  Each warp walks every fourth row of the
// cells a clump's bounding sphere may reach within the allowances, four rows side by side, and
// keeps the partners whose bounding spheres may meet; then it tests the sixteen sphere pairs of
// the partners it found and writes the near ones at their place in partner id order (equal
// contacts of one cell are summed in id order, force_part.cu:88-106), which it gets by counting
// the partners with smaller ids.  Bound by the latency of its chain of loads and tests, so it is
// split over four warps: a whole clump per thread took 47 us at 8,192 clumps, 49 at 32,768 and
// about 200 for 100,003 in four parts; so it is 31, 38 and 75 (in one launch).
__global__ void __launch_bounds__(kNearBlock) k_build_lists(const __grid_constant__ Margins m, DevScalars *d,
                                                            const int *__restrict__ flume,
                                                            const CullRec *__restrict__ cull,
                                                            const int *__restrict__ start,
                                                            const int *__restrict__ order,
                                                            const float4 *__restrict__ csort,
                                                            const long long *__restrict__ id,
                                                            const __grid_constant__ NearLists near, long s0, long s1,
                                                            long n) {
  __shared__ NearShared sh;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long s = s0 + blockIdx.x * (long)kNearClumps + lane;
  const bool valid = s < s1;
  const long sv = valid ? s : s1 - 1;
  const DevFlume &fl = d->flumes[flume[sv]];
  const GridF &g = fl.gridf;
  const CullRec &rec = cull[sv];
  const float4 mc = rec.c;
  const float allow = rec.allow, grown = allow * (1.0f + 1e-5f);
  const bool coarse = beyond_reach(rec, m);
  if (w == 0 && valid) {
    near.rem[s] = coarse ? -1.0f : allow * (1.0f - 1e-5f);
    // boundaries: the routines' gates are 1-Lipschitz in the sphere centre, so the allowance adds
    // to the bound; a door that is closed now may open, one that is open stays open
    const Consts &c = fl.c;
    unsigned bnd = 0u;
    const bool door_closed = *c.tp < 0.0;
    const int last = c.phase == AF3D_PHASE_AVALANCHE ? R_FLUME : R_HOP2;
    for (int rt = R_HOP0; rt <= last; rt++)
      if (bnd_may_touch_f(rt, mc, mc.w + grown, c, door_closed)) bnd |= 15u << (4 * rt);
    near.bnd[s] = bnd;
    CellAt at;   // (with `order` the sort has marked them)
    if (coarse && !order && cell_at(rec.key, fl.cell_off, g, at))
      go_away(s, mc, rec.key, at, m, fl, d, start, order, near, d->tick, n);
  }
  // the clumps that lists kept for each interval would not serve: their speed (the allowance is for half as
  // much again) takes them past the largest allowance, with 5 % to spare
  if (w == 0 && m.cap > 0.0f) {
    const float pace = valid && (unsigned)rec.key < (unsigned)d->ncell_total ? 0.7f * rec.pace / m.steps : 0.0f;
    for (int b = 0; b < kIntervals - 1; b++) {
      const unsigned past = __ballot_sync(0xffffffffu, pace * (float)(kBuildEvery >> b) > m.cap);
      if (!past) break;
      if (lane == 0) atomicAdd(&d->outrun[b], __popc(past));
    }
  }
  // the cells within reach of any partner's bound and allowance, FP32 with slack
  const CellRange b = cells_within(mc, (mc.w + grown + partner_reach(mc, m)) * (1.0f + 1e-5f), g);
  const int ny = b.y1 - b.y0 + 1, rows = valid && !coarse ? ny * (b.z1 - b.z0 + 1) : 0;
  const float mine = mc.w + grown;
  auto centre = [&](int k) {
    if (order) return __ldg(&csort[k]);
    float4 p = cull[k].c;
    p.w += cull[k].allow * (1.0f + 1e-5f);
    return p;
  };
  int found = 0;
#pragma unroll 1
  for (int r0 = w; r0 < rows; r0 += 16) {
    int k[4], end[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = r0 + 4 * q;
      k[q] = end[q] = 0;
      if (r < rows) {
        const int z = r / ny, y = r - z * ny;
        const int *row = start + fl.cell_off + (long long)g.nx * (b.y0 + y + (long long)g.ny * (b.z0 + z));
        k[q] = __ldg(row + b.x0);
        end[q] = __ldg(row + b.x1 + 1);
      }
    }
#pragma unroll 1
    while (k[0] < end[0] || k[1] < end[1] || k[2] < end[2] || k[3] < end[3]) {
      float4 p[4];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (k[q] < end[q]) p[q] = centre(k[q]);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (k[q] >= end[q]) continue;
        const float lim = mine + p[q].w;
        if (!(d2f(mc, p[q]) > lim * lim * kCullSlack)) {
          if (found < kWarpPartners) sh.pos[w][found][lane] = (unsigned)k[q];
          found++;
        }
        k[q]++;
      }
    }
  }
  sh.count[w][lane] = found;
  __syncthreads();
  const int c0 = sh.count[0][lane], c1 = sh.count[1][lane], c2 = sh.count[2][lane], c3 = sh.count[3][lane];
  const int total = c0 + c1 + c2 + c3, first = (w > 0 ? c0 : 0) + (w > 1 ? c1 : 0) + (w > 2 ? c2 : 0);
  const bool fits = total <= kPartners && max(max(c0, c1), max(c2, c3)) <= kWarpPartners;
  const OwnSpheres o = own_spheres(rec);
  const float units = unit_power(m.qs);
  unsigned masks[kWarpPartners / 2];   // the found partners' sixteen pairs, two to a word
#pragma unroll
  for (int i = 0; i < kWarpPartners / 2; i++) masks[i] = 0u;
  if (fits) {
    // kSide partners side by side: their slots, then their records, then the tests
#pragma unroll
    for (int i0 = 0; i0 < kWarpPartners; i0 += kSide) {
      if (i0 >= found) break;
      int t[kSide];
      long long tid[kSide];
      int4 ms[kSide][4];
      float ta[kSide];
#pragma unroll
      for (int k = 0; k < kSide; k++) {
        const int pos = (int)sh.pos[w][min(i0 + k, found - 1)][lane];
        t[k] = order ? __ldg(&order[pos]) : pos;
      }
#pragma unroll
      for (int k = 0; k < kSide; k++) {
        tid[k] = id[t[k]];
        ta[k] = cull[t[k]].allow;
#pragma unroll
        for (int q = 0; q < 4; q++) ms[k][q] = cull[t[k]].s[q];
      }
#pragma unroll
      for (int k = 0; k < kSide; k++) {
        const int i = i0 + k;
        if (i >= found) break;
        const bool self = t[k] == s;
        const unsigned mask = self ? 0u : sphere_mask(o, ms[k], (grown + ta[k] * (1.0f + 1e-5f)) * units + 4.0f);
        masks[i >> 1] |= mask << (16 * (i & 1));
        sh.id[first + i][lane] = self ? 0xFFFFFFFFu : (unsigned)tid[k];
        sh.pairs[first + i][lane] = (unsigned char)__popc(mask);
      }
#pragma unroll
      for (int k = 0; k < kSide; k++)   // after the group's reads, of which the last may be repeats
        if (i0 + k < found) sh.pos[w][i0 + k][lane] = (unsigned)t[k];
    }
  }
  __syncthreads();
  if (!valid) return;
  int entries = 0;
  if (fits) {
#pragma unroll
    for (int i = 0; i < kWarpPartners; i++) {
      if (i >= found) break;
      unsigned mask = (masks[i >> 1] >> (16 * (i & 1))) & 0xFFFFu;
      if (!mask) continue;
      const unsigned mid = sh.id[first + i][lane], t = sh.pos[w][i][lane];
      int at = 0;
      for (int j = 0; j < total; j++) at += sh.id[j][lane] < mid ? sh.pairs[j][lane] : 0;
      for (; mask; mask &= mask - 1u, at++)
        if (at < kNearCap) near.items[(long)at * n + s] = t << 4 | ((unsigned)__ffs(mask) - 1u);
    }
    if (w == 3)
      for (int j = 0; j < total; j++) entries += sh.pairs[j][lane];
  }
  if (w == 3) near.info[s] = coarse || !fits || entries > kNearCap ? -1 : entries;
}

}  // namespace

void launch_build_lists(const Launch &L, Margins m, DevScalars *d, const int *flume, const CullRec *cull, Cells cells,
                        const int *order, const long long *id, NearLists near, long s0, long count) {
  if (count < 0) count = L.n - s0;
  if (count <= 0) return;
  k_build_lists<<<(unsigned)((count + kNearClumps - 1) / kNearClumps), kNearBlock, 0, L.st>>>(
      m, d, flume, cull, cells.start, order, cells.csort, id, near, s0, s0 + count, L.n);
}

}  // namespace af3d
