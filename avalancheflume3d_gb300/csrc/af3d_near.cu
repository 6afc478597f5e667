// af3d_near.cu -- the near lists: per clump, the sphere pairs and boundary spheres that may touch
// while no clump moves farther than its allowance (NearLists in af3d_internal.h).
//
// Integer and FP32 work on the culling records; built from the sorted cell list once every
// kBuildEvery steps.
#include <climits>

#include "af3d_cellwalk.cuh"

namespace af3d {

namespace {

constexpr int kNearBlock = 128;
constexpr int kPartners = 32;   // partners whose bounding spheres may meet; with more, the per-clump search

// One thread per clump: walk the cells its bounding sphere may reach within the allowances, keep
// the partners whose bounding spheres may meet (positions in the sorted order), order them by
// clump id (equal contacts of one cell are summed in id order, force_part.cu:88-106), and test
// the sixteen sphere pairs of each.  Bound by the latency of the walk's loads and by its
// branches (18,500 + 12,000 cycles of a warp's 80,000 in a step when every step walked); two
// entries a turn are loaded together.  Building every 16 steps instead of every step is what
// takes it out of the step.
__global__ void __launch_bounds__(kNearBlock) k_build_lists(Margins m, DevScalars *d, const int *__restrict__ flume,
                                                            const CullRec *__restrict__ cull,
                                                            const int *__restrict__ start,
                                                            const int *__restrict__ order,
                                                            const float4 *__restrict__ csort,
                                                            const long long *__restrict__ id, NearLists near,
                                                            long s0, long n) {
  __shared__ unsigned s_slot[kPartners][kNearBlock];
  __shared__ unsigned s_id[kPartners][kNearBlock];
  const int tid = threadIdx.x;
  const long s = s0 + blockIdx.x * (long)kNearBlock + tid;
  if (s >= n) return;
  const DevFlume &fl = d->flumes[flume[s]];
  const GridF &g = fl.gridf;
  const Consts &c = fl.c;
  const CullRec &rec = cull[s];
  const float4 mc = rec.c;
  const float allow = rec.allow;
  near.loose[s] = INT_MAX;
  near.rem[s] = allow * (1.0f - 1e-5f);
  // boundaries: the routines' gates are 1-Lipschitz in the sphere centre, so the allowance adds
  // to the bound; a door that is closed now may open, one that is open stays open
  const float unit = unit_power(-m.qs);
  unsigned bnd = 0u;
  const bool door_closed = *c.tp < 0.0;
  const int last = c.phase == AF3D_PHASE_AVALANCHE ? R_FLUME : R_HOP2;
  const float grown = allow * (1.0f + 1e-5f);
  for (int rt = R_HOP0; rt <= last; rt++)
    if (bnd_may_touch_f(rt, mc, mc.w + grown, c, door_closed)) bnd |= 15u << (4 * rt);
  near.bnd[s] = bnd;
  const float rad = __int_as_float(rec.s[0].w);
  if (!(rad < kCullMaxUnits)) {   // too large for the lists: every clump searches for itself
    near.info[s] = -1;
    atomicMin(&d->all_slow, d->tick);
    return;
  }
  // the cells within reach of any partner's bound and allowance, FP32 with slack
  const float most = kCullMaxUnits * unit + 1e-6f * (fabsf(mc.x) + fabsf(mc.y) + fabsf(mc.z) + 10.0f) + m.cap;
  const float reach = (mc.w + grown + most) * (1.0f + 1e-5f);
  auto range = [&](float x, float xmin, float inv, int cells, int &lo, int &hi) {
    const float q = (x - xmin) * inv, w = reach * inv;
    const float e = 2e-6f * ((fabsf(x) + fabsf(xmin)) * inv + fabsf(q) + w + 1.0f);
    lo = (int)fminf(fmaxf(floorf(q - w - e), 0.0f), (float)(cells - 1));
    hi = (int)fminf(fmaxf(floorf(q + w + e), 0.0f), (float)(cells - 1));
  };
  int x0, x1, y0, y1, z0, z1;
  range(mc.x, g.xmin, g.ix, g.nx, x0, x1);
  range(mc.y, g.ymin, g.iy, g.ny, y0, y1);
  range(mc.z, g.zmin, g.iz, g.nz, z0, z1);
  int npass = 0;
  const float mine = mc.w + grown;
  auto keep = [&](int k, float4 pc) {
    const float lim = mine + pc.w;
    if (d2f(mc, pc) > lim * lim * kCullSlack) return;
    if (npass < kPartners) s_slot[npass][tid] = (unsigned)k;
    npass++;
  };
  auto centre = [&](int k) {
    if (order) return __ldg(&csort[k]);
    float4 p = cull[k].c;
    p.w += cull[k].allow;
    return p;
  };
#pragma unroll 1
  for (int z = z0; z <= z1; z++) {
    int next0, next1;
    const int *row = start + fl.cell_off + (long long)g.nx * (y0 + (long long)g.ny * z);
    next0 = __ldg(row + x0);
    next1 = __ldg(row + x1 + 1);
#pragma unroll 1
    for (int y = y0; y <= y1; y++) {
      int k = next0;
      const int end = next1;
      if (y < y1) {   // the next row's range is loaded while this one is walked
        row += g.nx;
        next0 = __ldg(row + x0);
        next1 = __ldg(row + x1 + 1);
      }
#pragma unroll 1
      for (; k + 1 < end; k += 2) {
        const float4 p0 = centre(k), p1 = centre(k + 1);
        keep(k, p0);
        keep(k + 1, p1);
      }
      if (k < end) keep(k, centre(k));
    }
  }
  if (npass > kPartners) {
    near.info[s] = -1;
    return;
  }
  // slots and ids of the partners, in id order
  int np = 0;
#pragma unroll 1
  for (int i = 0; i < npass; i++) {
    const int pos = (int)s_slot[i][tid];
    const int t = order ? __ldg(&order[pos]) : pos;
    if (t == s) continue;
    const unsigned pid = (unsigned)id[t];
    int j = np++;
    for (; j > 0 && s_id[j - 1][tid] > pid; j--) {
      s_id[j][tid] = s_id[j - 1][tid];
      s_slot[j][tid] = s_slot[j - 1][tid];
    }
    s_id[j][tid] = pid;
    s_slot[j][tid] = (unsigned)t;
  }
  const OwnSpheres o = own_spheres(rec);
  const float units = unit_power(m.qs);
  int cnt = 0;
#pragma unroll 1
  for (int i = 0; i < np; i++) {
    const unsigned t = s_slot[i][tid];
    int4 ms[4];
#pragma unroll
    for (int k = 0; k < 4; k++) ms[k] = cull[t].s[k];
    const float margin = (grown + cull[t].allow * (1.0f + 1e-5f)) * units + 4.0f;
    unsigned mask = sphere_mask(o, ms, margin);
    while (mask) {
      const unsigned p = (unsigned)__ffs(mask) - 1u;
      mask &= mask - 1u;
      if (cnt < kNearCap) near.items[(long)cnt * n + s] = t << 4 | p;
      cnt++;
    }
  }
  near.info[s] = cnt > kNearCap ? -1 : cnt;
}

}  // namespace

void launch_build_lists(const Launch &L, Margins m, DevScalars *d, const int *flume, const CullRec *cull, Cells cells,
                        const int *order, const long long *id, NearLists near, long s0, long count) {
  const long c = count < 0 ? L.n - s0 : (count < L.n - s0 ? count : L.n - s0);
  if (L.n <= 0 || c <= 0) return;
  // a part ends inside its own slots: the launch's last block may reach into the next part's,
  // whose lists that part builds again
  k_build_lists<<<(unsigned)((c + kNearBlock - 1) / kNearBlock), kNearBlock, 0, L.st>>>(
      m, d, flume, cull, cells.start, order, cells.csort, id, near, s0, L.n);
}

}  // namespace af3d
