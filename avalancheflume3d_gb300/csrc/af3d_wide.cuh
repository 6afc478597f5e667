// af3d_wide.cuh -- the force pass of small clump counts: 32 clumps on a block of 128 threads.
//
// Up to about 20,000 clumps (wide_clumps) k_lists_forces leaves most of the chip idle (2,048 clumps are 64 warps on
// 608 sub-partitions) and a pass takes as long as one warp's chain of instructions: an FP64
// instruction every 64 cycles, ~400 of them, and as many cycles again in integer work and loads.
// Here a block's four warps share its 32 clumps (lane = clump): warp 0 tests the near pairs while
// warp 1 tests the boundaries; the contact items go round by round to all four; then warps 0..2 take
// one component each of the sums, of get_accel, finish_Verlet and the next step's predictor
// (exchanging vectors in shared memory), and warp 3 the clump's key, its records and its place.
// Each component is formed by k_lists_forces' operations in their order: the same results.
// Included by af3d_kernels.cu, whose helpers it uses.
#pragma once

constexpr int kWide = 32;
constexpr int kWideThreads = 128;

struct WideShared {
  PassLists pl;
  int npair[kWide];
  unsigned bnd[kWide];
  unsigned item[kBatch];
  unsigned char owner[kBatch], place[kBatch], flag[kBatch];
  double res[6][kBatch];
  double vec[12][kWide];        // exchanged vectors: torque, alpha in the body frame, turn, position
  double aux[3][kWide];
  float spin[3][kWide];
  unsigned char ok[3][kWide];
  union {
    long long fixed[9][kWide];
    double row[9][kWide];
  };
  double col[9][kWide];
  double rec[kWide * kRecStride];
};

// Component i of a vector in registers.
__device__ __forceinline__ double comp(V3 v, int i) { return i == 0 ? v.x : i == 1 ? v.y : v.z; }

struct Accel {
  V3 a, al;
};
// get_accel of a whole clump (inertia that is not isotropic, spins whose signs FP32 leaves open).
__device__ __noinline__ Accel get_accel_whole(V3 f, V3 t, V3 v, V3 w, Rows R, double m, double adrag0, V3 I, double im,
                                              double iI, bool dev) {
  Accel r;
  get_accel_one(f, t, v, w, R.x, R.y, R.z, m, adrag0, I, r.a, r.al, im, iI, dev);
  return r;
}

template <bool UNIFORM>
__global__ void __launch_bounds__(kWideThreads, 4)
    k_forces_wide(const __grid_constant__ Planes P, const __grid_constant__ Planes out, DevScalars *d,
                  const int *__restrict__ flume, const NbrRec *__restrict__ nbr,
                  const CullRec *__restrict__ cull, const __grid_constant__ Cells cells,
                  const int *__restrict__ order, const long long *__restrict__ id,
                  const __grid_constant__ NearLists near, ContactLists lists, long ntags, bool write_ft, bool counted,
                  const __grid_constant__ Consts kc, bool warm, const __grid_constant__ LookAhead la, long s0, long n) {
  __shared__ WideShared sh;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const long bbase = s0 + blockIdx.x * (long)kWide, s = bbase + lane;
  const bool valid = s < n;
  const long sv = valid ? s : n - 1;   // in-range slot for lanes past n (nothing is written for them)
  const int f = flume[sv];
  const DevFlume &fl = d->flumes[f];
  auto body = [&](const Consts &c) {
    const NbrRec &me = nbr[sv];
    const bool removed = is_removed(*c.tp, me.rx, c.side_x), act = valid && !removed;
    const bool aval = c.phase == AF3D_PHASE_AVALANCHE, dev = c.variant == AF3D_FRICTION_DEV;
    const int info = near.info[sv];
    const bool search = act && must_search(sv, d, near, info);
    const unsigned *list = near.items + sv;
    unsigned *col = lists.items + sv;
    // the clumps' items: near pairs (warp 0), boundary spheres (warp 1)
    if (w == 0) {
      int np = 0;
      if (search) np = search_items(sv, d, flume, nbr, cull, cells.start, order, id, near, P.m, n, col, 0);
      else if (act) np = near_pairs(sv, info, fl, me, cull, list, n, sh.pl);
      sh.npair[lane] = np;
    } else if (w == 1) {
      unsigned b = 0u;
      if (act)
        b = touching(search ? 0x0FFFFFFFu : near.bnd[sv], me,
                     __int_as_float(cull[sv].s[0].w) * unit_power(-P.m.qs), c);
      sh.bnd[lane] = b;
    }
    __syncthreads();
    int npair = sh.npair[lane];
    const unsigned bnd = sh.bnd[lane];
    const int npre = __popc(bnd & bits_before(aval)), npost = __popc(bnd & bits_after(aval));
    const bool slow = npair < 0 || npre + npair + npost > kListCap;
    if (slow) npair = 0;
    const int nitems = slow ? 0 : npre + npair + npost;
    // exclusive prefixes over the clumps: items, particle items
    int base = nitems, pb = npair;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, base, k), v = __shfl_up_sync(0xffffffffu, pb, k);
      if (lane >= k) {
        base += u;
        pb += v;
      }
    }
    const int total = __shfl_sync(0xffffffffu, base, 31), ptotal = __shfl_sync(0xffffffffu, pb, 31);
    base -= nitems;
    pb -= npair;
    const bool kind_order = total <= kBatch;
    if (w == 2 && valid) {
      if (slow || (act && info < 0)) atomicAdd(&d->overflows, 1ull);
      if (lists.ovf && slow) *lists.ovf = 1;
      if (counted) cells.occ[cull[s].key] = 0;
    }
    double Fi = 0.0, Ti = 0.0;   // warps 0..2: this component of the sums
    int active = 0;              // warp 3: sphere-sphere contacts
    int kept = 0, kept_pre = 0;  // ... and the recorded items, those with a force (block_contacts)
    if (valid && removed && aval && w < 3) {
      const SlowSums r = removed_contacts(&me, (double)cull[sv].c.w, c);
      Fi = comp(r.F, w);
      Ti = comp(r.T, w);
    }
    auto constants_of = [&](long os) -> const Consts & {
      if constexpr (UNIFORM) {
        return c;
      } else {
        return d->flumes[flume[os]].c;
      }
    };
    for (int b0 = 0; b0 < total; b0 += kBatch) {
      const int bn = total - b0 < kBatch ? total - b0 : kBatch;
      auto lay = [&](unsigned it, int e, int j) {   // item e of the clump's list, j-th in kind order
        const int at = base + e - b0;
        if (lists.cnt && b0 == 0) col[(long)e * n] = it;   // recorded for the adjoint
        if (at < 0 || at >= bn) return;
        if (!kind_order) j = at;
        sh.item[j] = it;
        sh.owner[j] = (unsigned char)lane;
        sh.place[j] = (unsigned char)at;
      };
      if (w == 0 && !slow)
        for (int e = npair - 1; e >= 0; e--)   // (a search left its items in the column: the last first)
          lay(search ? col[(long)(e + (lists.cnt && b0 > 0 ? npre : 0)) * n]
                     : list[(long)(sh.pl.cand[e][lane] & 63u) * n],
              npre + e, pb + e);
      __syncthreads();   // (the recorded column's head may hold a search's items until here)
      if (w == 1 && !slow) {
        int e = 0, j = ptotal + (base - pb);
        for (unsigned b = bnd & bits_before(aval); b; b &= b - 1u) lay(kBndItem | ((unsigned)__ffs(b) - 1u), e++, j++);
        e += npair;
        for (unsigned b = bnd & bits_after(aval); b; b &= b - 1u) lay(kBndItem | ((unsigned)__ffs(b) - 1u), e++, j++);
      }
      __syncthreads();
      const int np = kind_order ? ptotal : bn, q0 = kind_order ? ptotal : 0;
      for (int i = tid; i < np; i += kWideThreads) {
        const unsigned it = sh.item[i];
        if (it >= kBndItem) continue;
        const long os = bbase + sh.owner[i];
        const int at = sh.place[i];
        const NbrRec &mo = nbr[os];
        const Consts &co = constants_of(os);
        const int t = (int)(it >> 4), p = (int)(it & 15u), k = p & 3;
        const V3 rl = mk(mo.rx, mo.ry, mo.rz);
        ContactIn ci;
        V3 fs, tq;
        int r = 0;
        if (pair_input(rl, mk(mo.vx, mo.vy, mo.vz), mk(mo.wx, mo.wy, mo.wz),
                       mk(mo.s[3 * k], mo.s[3 * k + 1], mo.s[3 * k + 2]), mo.rad, mo.msph, nbr[t], p >> 2, co,
                       co.variant == AF3D_FRICTION_DEV, ci) &&
            apply_law(ci, rl, co, fs, tq)) {
          r = 2;
          sh.res[0][at] = fs.x; sh.res[1][at] = fs.y; sh.res[2][at] = fs.z;
          sh.res[3][at] = tq.x; sh.res[4][at] = tq.y; sh.res[5][at] = tq.z;
        }
        sh.flag[at] = (unsigned char)r;
      }
      const int w0 = (w + 4 - (np + 31) / 32 % 4) % 4;
      for (int i = q0 + 32 * w0 + lane; i < bn; i += kWideThreads) {
        const unsigned it = sh.item[i];
        if (it < kBndItem) continue;
        const long os = bbase + sh.owner[i];
        const int at = sh.place[i];
        sh.flag[at] = (unsigned char)bnd_contact<>(it, nbr + os, constants_of(os), &sh.res[0][at], kBatch);
      }
      __syncthreads();
      const int e1 = base + nitems < b0 + bn ? base + nitems - b0 : bn;
      for (int e = base > b0 ? base - b0 : 0; e < e1; e++) {
        const int k = sh.flag[e];
        if (k < 2) continue;
        if (w < 3) {
          Ti += sh.res[3 + w][e];
          Fi += sh.res[w][e];
        } else {
          active += k == 2;
          if (lists.cnt) {
            const int at = e + b0 - base;
            col[n * kept++] = col[(long)at * n];
            kept_pre += at < npre;
          }
        }
      }
      __syncthreads();
    }
    if (slow) {
      const int pre0 = aval ? R_HOP0 : 1, pre1 = aval ? R_WALLS : 0;
      const int post0 = aval ? R_FLUME : R_HOP0, post1 = aval ? R_FLUME : R_HOP2;
      const V3 zero = mk(0.0, 0.0, 0.0);
      const SlowSums r = slow_contacts(sv, pre0, pre1, post0, post1, c, d, flume, nbr, cull, cells.start, order, id,
                                       near, P.m, n, zero, zero);
      if (w < 3) {
        Fi = comp(r.F, w);
        Ti = comp(r.T, w);
      } else {
        active = r.active;
      }
    }
    if (w == 3) {
      warp_count(d, active);
      if (lists.cnt && valid) lists.cnt[s] = pack_list_counts(slow ? -1 : kept, kept_pre, slow ? 0 : active);
    }

    // get_accel and finish_Verlet, one component a warp (i = w)
    const int i = w, i1 = w == 2 ? 0 : w + 1, i2 = w == 0 ? 2 : w - 1;
    const int R0 = warm ? RN00 : R00;
    const V3 v = mk(me.vx, me.vy, me.vz), om = mk(me.wx, me.wy, me.wz);
    const double *mr = &me.rx, *mv = &me.vx, *mw = &me.wx;   // (three consecutive doubles each)
    double Rc[3] = {0.0, 0.0, 0.0}, Rr[3] = {0.0, 0.0, 0.0};   // column and row i of the rotation
    if (w < 3) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        Rc[k] = P.p[R0 + 3 * k + i][sv];
        Rr[k] = P.p[R0 + 3 * i + k][sv];
      }
      sh.vec[w][lane] = Ti;
      sh.aux[w][lane] = Fi;
    }
    __syncthreads();
    const V3 T = mk(sh.vec[0][lane], sh.vec[1][lane], sh.vec[2][lane]);
    const V3 I = load3(P, IXX, sv);
    const double mass = P.p[MASS][sv], im = P.p[IMASS][sv], iI = P.p[IINER][sv], adrag0 = P.p[ADRAG][sv];
    const bool isotropic =
        bits_of(I.x) == bits_of(I.y) && bits_of(I.y) == bits_of(I.z) && positive_bits(I.x) && finite_bits(I.x);
    if (w < 3) {
      const double tb = T.x * Rc[0] + T.y * Rc[1] + T.z * Rc[2];
      if (kFast) {
        sh.vec[3 + w][lane] = tb * iI;
        sh.ok[w][lane] = isotropic && finite_bits(om.x) && finite_bits(om.y) && finite_bits(om.z);
      } else {
        sh.vec[3 + w][lane] = div_by(tb, divisor_of(I.x));
        // the sign of the body-frame spin's component, certain or not (as get_accel_one)
        const float wx = truncated_f(om.x), wy = truncated_f(om.y), wz = truncated_f(om.z);
        const float r0 = truncated_f(Rc[0]), r1 = truncated_f(Rc[1]), r2 = truncated_f(Rc[2]);
        const float x = wx * r0, y = wy * r1, z = wz * r2, sum = x + y + z;
        sh.spin[w][lane] = sum;
        sh.ok[w][lane] = isotropic && fabsf(wx) < 1e18f && fabsf(wy) < 1e18f && fabsf(wz) < 1e18f &&
                         fabsf(r0) < 4.0f && fabsf(r1) < 4.0f && fabsf(r2) < 4.0f &&
                         fabsf(sum) > 1e-5f * (fabsf(x) + fabsf(y) + fabsf(z)) + 1e-30f;
      }
    }
    __syncthreads();
    double ai = 0.0, ali = 0.0, v2 = 0.0, w2 = 0.0;   // this component of a_f, alpha_f and the corrected velocities
    if (w < 3 && valid) {
      if (write_ft) {
        P.p[FX + i][s] = Fi;
        P.p[TX + i][s] = Ti;
      }
      if (warm && !la.keep) {   // commit the predicted state to the planes
        P.p[RX + i][s] = mr[i];
#pragma unroll
        for (int k = 0; k < 4; k++) P.p[S0X + 3 * k + i][s] = me.s[3 * k + i];
#pragma unroll
        for (int k = 0; k < 3; k++) P.p[R00 + 3 * i + k][s] = Rr[k];
      }
      if (!removed) {
        if (sh.ok[0][lane] && sh.ok[1][lane] && sh.ok[2][lane]) {
          V3 ab = mk(sh.vec[3][lane], sh.vec[4][lane], sh.vec[5][lane]);
          if (!kFast) {
            const float sb[3] = {sh.spin[0][lane], sh.spin[1][lane], sh.spin[2][lane]};
            ab = mk(plus_signed_zero(ab.x, sb[1], sb[2]), plus_signed_zero(ab.y, sb[2], sb[0]),
                    plus_signed_zero(ab.z, sb[0], sb[1]));
          }
          const double v2s = v.x * v.x + v.y * v.y + v.z * v.z;
          const double adrag = adrag0 * speed_of<false>(v2s, dev);
          const double vi = comp(v, i);
          if (kFast) ai = Fi * im - adrag * vi;
          else ai = div_by(Fi, divisor_of(mass)) - adrag * vi;
          if (i == 2) ai = ai - kGRAV;
          ali = ab.x * Rr[0] + ab.y * Rr[1] + ab.z * Rr[2];
        } else {
          const Rows R = {load3(P, R0, s), load3(P, R0 + 3, s), load3(P, R0 + 6, s)};
          const Accel r = get_accel_whole(mk(sh.aux[0][lane], sh.aux[1][lane], sh.aux[2][lane]), T, v, om, R, mass,
                                          adrag0, I, im, iI, dev);
          ai = comp(r.a, i);
          ali = comp(r.al, i);
        }
        const double a0 = P.p[AIX + i][s], al0 = P.p[ALIX + i][s];
        // finish_Verlet.cu:43-48
        v2 = mv[i] + c.hdt * (ai - a0);
        w2 = mw[i] + c.hdt * (ali - al0);
        if (!(finite_bits(ai) && finite_bits(ali))) raise_status(d, AF3D_ERR_NAN);
      } else {
        w2 = mw[i];   // finish_Verlet.cu:28-32 (the reference leaves stale accelerations here)
      }
      P.p[AFX + i][s] = ai;
      P.p[ALFX + i][s] = ali;
      if (!la.keep) {
        out.p[VX + i][s] = v2;
        out.p[WX + i][s] = w2;
      }
    }
    if (!la.nbr) return;

    // The next step's init_Verlet, as predict_state, one component a warp; removal test at this
    // step's time, a_i = this a_f.
    const double dt = fl.sys.dt, hdt = fl.sys.hdt;
    const double rad = removed ? 0.0 : P.p[RAD][sv];
    double rn = 0.0, vn = v2, wn = w2, c4[4] = {0.0, 0.0, 0.0, 0.0};
    if (w < 3) {
      rn = mr[i];
      if (!removed) {
        rn += dt * (v2 + hdt * ai);
        vn += dt * ai;
        sh.vec[6 + w][lane] = dt * (w2 + hdt * ali);
        wn += dt * ali;
      }
      sh.vec[9 + w][lane] = rn;
      double *o = sh.rec + lane * kRecStride;
      o[i] = rn;
      o[3 + i] = vn;
      o[6 + i] = wn;
#pragma unroll
      for (int k = 0; k < 3; k++) sh.col[3 * k + i][lane] = Rc[k];
    }
    __syncthreads();
    const V3 dO = mk(sh.vec[6][lane], sh.vec[7][lane], sh.vec[8][lane]);
    const V3 r1 = mk(sh.vec[9][lane], sh.vec[10][lane], sh.vec[11][lane]);
    const double t_next = *c.tp + d->flumes[0].sys.dt;   // k_advance_time's expression
    long key = 0;
    if (w == 3 && valid) {
      key = bucket_key(r1, fl, d, id[s], t_next);
      if (la.build) cells.key[s] = (int)key;
      if (removed) P.p[RAD][s] = 0.0;
    }
    constexpr Divisor root2 = constant_divisor(kROOT2, 0x3FF6A09E667F3BCCull);
    const double pos = kFast ? rad * (1.0 / kROOT2) : div_by(rad, root2);
    const bool turns = valid && !removed;
    if constexpr (kFast) {
      bool ok = false;
      if (turns && w < 3 && !dev) {
        const double angle[3] = {dO.x, dO.y, dO.z};
        Turn turn;
        long long t[3];
        ok = turn_fixed(angle, turn) && column_fixed(turn, Rc, t);
        if (ok)
#pragma unroll
          for (int k = 0; k < 3; k++) sh.fixed[3 * k + i][lane] = t[k];
      }
      if (w < 3) sh.ok[w][lane] = ok;
      __syncthreads();
      if (turns && w < 3) {
        if (sh.ok[0][lane] && sh.ok[1][lane] && sh.ok[2][lane]) {
          long long row[3];
#pragma unroll
          for (int k = 0; k < 3; k++) {
            row[k] = sh.fixed[3 * i + k][lane];
            Rr[k] = double_of(row[k], 62);
          }
          const double at[3] = {r1.x, r1.y, r1.z};
          if (spheres_fit(at, pos, P.m.qs + 38)) {
            spheres_row_fixed(row, comp(r1, i), pos, P.m.qs + 38, c4);
          } else {
            place_row(comp(r1, i), mk(Rr[0], Rr[1], Rr[2]), pos, c4);
          }
        } else {
          const Rows t = turn_rows<>(dO, mk(sh.col[0][lane], sh.col[1][lane], sh.col[2][lane]),
                                   mk(sh.col[3][lane], sh.col[4][lane], sh.col[5][lane]),
                                   mk(sh.col[6][lane], sh.col[7][lane], sh.col[8][lane]));
          const V3 row = i == 0 ? t.x : i == 1 ? t.y : t.z;
          Rr[0] = row.x; Rr[1] = row.y; Rr[2] = row.z;
          place_row(comp(r1, i), row, pos, c4);
        }
      }
    } else {
      // dR's row i, then column i of dR R renormalised, then row i of that (turn_rows' operations)
      double mag = 0.0, sn = 0.0, cs = 1.0;
      if (turns && w < 3) {
        const double mag2 = dO.x * dO.x + dO.y * dO.y + dO.z * dO.z;
        mag = sqrt_rn(mag2);
        double u = 0.0;
        if (positive_bits(mag)) {
          u = div_by(comp(dO, i), divisor_of(mag));
          sincos_step(mag, mag2, sn, cs);
        }
        sh.aux[w][lane] = u;
      }
      __syncthreads();
      if (turns && w < 3) {
        double e[3] = {i == 0 ? 1.0 : 0.0, i == 1 ? 1.0 : 0.0, i == 2 ? 1.0 : 0.0};
        if (positive_bits(mag)) {
          const double omc = 1.0 - cs, ui = sh.aux[i][lane], u1 = sh.aux[i1][lane], u2 = sh.aux[i2][lane];
          // (i, i): omc u_i u_i + c;  (i, i1): omc u_i u_i1 - sn u_i2;  (i, i2): omc u_i u_i2 + sn u_i1
          const double d0 = omc * ui * ui + cs, d1 = omc * ui * u1 - sn * u2, d2 = omc * ui * u2 + sn * u1;
          e[0] = i == 0 ? d0 : i1 == 0 ? d1 : d2;
          e[1] = i == 1 ? d0 : i1 == 1 ? d1 : d2;
          e[2] = i == 2 ? d0 : i1 == 2 ? d1 : d2;
        }
#pragma unroll
        for (int k = 0; k < 3; k++) sh.row[3 * i + k][lane] = e[k];
      }
      __syncthreads();
      if (turns && w < 3) {
        double t[3];
#pragma unroll
        for (int k = 0; k < 3; k++)
          t[k] = sh.row[3 * k][lane] * Rc[0] + sh.row[3 * k + 1][lane] * Rc[1] + sh.row[3 * k + 2][lane] * Rc[2];
        const Divisor by = divisor_of(sqrt_rn(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]));
#pragma unroll
        for (int k = 0; k < 3; k++) sh.col[3 * k + i][lane] = div_by(t[k], by);
      }
      __syncthreads();
      if (turns && w < 3) {
#pragma unroll
        for (int k = 0; k < 3; k++) Rr[k] = sh.col[3 * i + k][lane];
        place_row(comp(r1, i), mk(Rr[0], Rr[1], Rr[2]), pos, c4);
      }
    }
    if (w < 3) {
      double *o = sh.rec + lane * kRecStride;
      if (removed)
#pragma unroll
        for (int k = 0; k < 4; k++) c4[k] = me.s[3 * k + i];
      if (valid)
#pragma unroll
        for (int k = 0; k < 3; k++) P.p[RN00 + 3 * i + k][s] = Rr[k];
#pragma unroll
      for (int k = 0; k < 4; k++) o[9 + 3 * k + i] = c4[k];
    } else {
      double *o = sh.rec + lane * kRecStride;
      o[21] = rad;
      o[22] = P.p[MSPH][sv];
      o[23] = P.p[MWALL][sv];
    }
    __syncthreads();
    // the records: warp 3 forms the culling record and takes the clump's place, the others write
    // the neighbour records out
    if (w == 3) {
      if (valid) {
        const double *o = sh.rec + lane * kRecStride;
        NbrRec q;
        CullRec cr;
        V3 sp[4];
        for (int k = 0; k < 4; k++) sp[k] = mk(o[9 + 3 * k], o[10 + 3 * k], o[11 + 3 * k]);
        make_records(r1, mk(o[3], o[4], o[5]), mk(o[6], o[7], o[8]), sp, o[21], o[22], o[23], P.m, (int)key, q, cr);
        la.cull[s] = cr;
        if (la.build) {
          cells.rank_tmp[s] = arrive_in_bucket(cells, key);
        } else {
          int4 old[4];
          for (int k = 0; k < 4; k++) old[k] = cull[s].s[k];
          if (keep_place(s, old, cr, fl, d, cells.occ_next, ntags, near, cells.start, order, P.m, d->tick + 1, n))
            la.cull[s].away = 1;
        }
      }
    } else {
      const long cnt = n - bbase < kWide ? n - bbase : kWide;
      const int nw = (int)(cnt * kRecWords) / 2;
      double2 *b = reinterpret_cast<double2 *>(la.nbr + bbase);
      for (int k = tid; k < nw; k += 96) {
        const int w0 = 2 * k, q0 = w0 / kRecWords, k0 = w0 - q0 * kRecWords;
        b[k] = make_double2(sh.rec[q0 * kRecStride + k0], sh.rec[q0 * kRecStride + k0 + 1]);
      }
    }
    __syncthreads();
    if (tid == 0) {   // as in fused_body
      __threadfence();
      if (atomicInc(&d->ticket, gridDim.x - 1) == gridDim.x - 1) advance_clock(d);
    }
  };
  if constexpr (UNIFORM) body(kc);
  else body(fl.c);
}
