// edmd_lanes.cuh -- one event's arithmetic spread over the lanes of a group,
// shared by the engines that run an event per warp or part of a warp: lane
// roles (disk x axis), pair solves on two lanes, and the prediction of the one
// or two disks an event changes.
#pragma once
#include <cstddef>
#include "edmd_device.cuh"

namespace edmd {

constexpr int MAXC = 7;          // candidates buffered per cell list per lane (a count of three bits)

// candidate buffers of one lane group
struct LaneScratch {
  int32_t reg[2 * 9 * MAXC];     // walk buffers, one per (disk, cell) task
  int32_t comp[2 * 9 * MAXC];    // packed candidates
  int16_t ord[2 * 9 * MAXC];     // their scan order
};

// A group of GW lanes that works on one event: a whole warp (GW = 32) or a part
// of it.  Every collective goes through the group's mask and width, so the
// groups of a warp are independent and may diverge.
template <int GW>
struct Grp {
  int lane;                      // 0 .. GW-1
  unsigned mask;                 // the group's lanes within the warp
  __device__ __forceinline__ explicit Grp(int tid)
      : lane(tid & (GW - 1)), mask(GW == 32 ? 0xffffffffu : (((1u << GW) - 1u) << ((tid & 31) & ~(GW - 1)))) {}
  template <class T> __device__ __forceinline__ T shfl(T v, int src) const { return __shfl_sync(mask, v, src, GW); }
  template <class T> __device__ __forceinline__ T shfl_xor(T v, int o) const {
    return __shfl_xor_sync(mask, v, o, GW);
  }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  __device__ __forceinline__ bool any(bool p) const { return __any_sync(mask, p); }
  __device__ __forceinline__ uint32_t min_u32(uint32_t v) const { return __reduce_min_sync(mask, v); }
  // group-relative ballot
  __device__ __forceinline__ unsigned ballot(bool p) const {
    const unsigned m = __ballot_sync(mask, p) & mask;
    return GW == 32 ? m : m >> (__ffs(mask) - 1);
  }
  // group-relative index of the first lane where p holds, or -1
  __device__ __forceinline__ int first(bool p) const {
    const unsigned m = __ballot_sync(mask, p) & mask;
    return m ? ((__ffs(m) - 1) & (GW - 1)) : -1;
  }
};

// Lanes of the event handlers.  The (one or two) disks an event changes are
// spread over four lane roles, repeated over the group: disk `lane & 1` (the
// owner, or the partner of a collision) and axis `lane & 2` (x, or y).  Each
// lane holds its disk's coordinate, velocity and cell along its axis, so the
// scalar FP64 work of both disks and both axes shares its instructions: an
// FP64 instruction costs its ~76 issue cycles whatever the lanes it serves.
struct Own {
  double p, v, rad, vr;            // coordinate and velocity along the axis; radius, growth rate
  int c;                           // cell index along the axis
};

// a collision prediction of the lane's disk: time image, partner, its counter,
// the scan position (0..8) of the cell the partner was found in (4, the disk's
// own, when there is none), and the partner's tag (3 when there is none)
struct Next { uint64_t key; int32_t partner; uint32_t ca; int q, tag; };
constexpr int OVL_CORRUPT = -2;    // overlap marker: a cell list longer than N (EDMD_ERR_BUDGET)

// a disk record's coordinate or velocity along an axis (x, y, vx, vy lead it)
__device__ __forceinline__ double* axis_pos(Disk* d, bool y) { return &d->x + (y ? 1 : 0); }
__device__ __forceinline__ double* axis_vel(Disk* d, bool y) { return &d->vx + (y ? 1 : 0); }
static_assert(offsetof(Disk, y) == offsetof(Disk, x) + 8 && offsetof(Disk, vy) == offsetof(Disk, vx) + 8, "axis layout");

// nearest periodic image of a difference along an axis (PBC src/EDMD.c:5896)
__device__ __forceinline__ double near_image(double d, double hL, double L) {
  if (ge_pos(d, hL)) d -= L;
  else if (lt_neg(d, hL)) d += L;
  return d;
}

// candidate times compared as their order-preserving integer images: the
// same order as FP64 '<' (both zeros share one image; a NaN, which '<' never
// selects, maps above every number), on the integer pipe
__device__ __forceinline__ uint64_t cand_key(double d) {
  const uint64_t u = (uint64_t)__double_as_longlong(d);
  return (u & 0x7fffffffffffffffull) > 0x7ff0000000000000ull ? ~0ull : time_key(d);
}

__device__ __forceinline__ void best_merge(uint64_t& bk, int& bo, int& bp, uint32_t& bc,
                                           uint64_t k, int o, int p, uint32_t c) {
  if (k < bk || (k == bk && o < bo)) { bk = k; bo = o; bp = p; bc = c; }
}

// collisionTimeNormal (src/EDMD.c:2661-2723) and collisionTimeGrow (2598-2659)
// of an owner current at t and a candidate P, by the two lanes 2k, 2k + 1: one
// axis each (p1, v1 of the owner), the sums over the axes by shuffle.  A pair
// costs 16 FP64 instructions instead of the 24 of one lane, and the
// candidates of an event (about 6 per disk) still fit one pass of a warp.
// Same operations and roundings as coll_time_normal_i / coll_time_grow (the
// sums of two products commute).  Every lane of the group takes part; `act`
// marks the pairs that count.  The candidate comes flown to t: coordinate and
// velocity along the lane's axis, radius, growth rate.
template <int GW, bool ADD, bool GROW>
__device__ __forceinline__ double pair_time_flown(const Box& B, const Grp<GW>& G, bool act, double p1, double v1,
                                                  double rad1, double vr1, double p2, double vel, double rad2,
                                                  double vr2, bool* ovl) {
  const bool y = G.lane & 1;
  const double dv = vel - v1;
  const double d = near_image(p2 - p1, y ? B.hLy : B.hLx, y ? B.Ly : B.Lx);
  double b = d * dv, v2 = dv * dv, d2 = d * d;
  b += G.shfl_xor(b, 1);
  v2 += G.shfl_xor(v2, 1);
  d2 += G.shfl_xor(d2, 1);
  if constexpr (!GROW) {
    d2 -= contact2<ADD>(B, rad1, rad2);
    // b b on the y lane, v2 d2 on the x lane
    const double u = (y ? b : v2) * (y ? b : d2);
    const double w = G.shfl_xor(u, 1);
    const double det = (y ? u : w) - (y ? w : u);
    if (!act || is_pos(b)) return NEVER;
    if (lt_neg(d2, 0.01)) { *ovl = true; return NEVER; }
    if (is_neg(det)) return NEVER;
    return div_rn(-b - sqrt_rn(det), v2);
  } else {
  const double dvr = vr1 + vr2;
  const double dr = contact(B, rad1, rad2);
  b -= dvr * dr;
  const double den = v2 - dvr * dvr, gap = d2 - dr * dr;
  const double det = b * b - den * gap;
  const bool root = act && !(det < 0);
  // the two roots on the two lanes: -b - s on x, -b + s on y
  double r = 0;
  if (root) {
    const double s = sqrt_rn(det);
    r = div_rn(-b + flip(s, !y), den);
  }
  const double q = G.shfl_xor(r, 1);
  const double minus = y ? q : r, plus = y ? r : q;
  if (!root) return NEVER;
  if (((minus > 0) && (plus > 0) && (minus < plus)) || ((minus > 0) && (plus < 0))) return minus;
  else if (((minus > 0) && (plus > 0.000000001) && (plus < minus)) || ((minus < 0) && (plus > 0.000000001)))
    return plus;
  if (gap < -0.01) *ovl = true;
  return NEVER;
  }
}

// the same with the candidate's record, flown here
template <int GW, bool ADD, bool GROW>
__device__ __forceinline__ double pair_time_lanes(const Box& B, const Grp<GW>& G, bool act, double p1, double v1,
                                                  double rad1, double vr1, const Disk* P, const double* vr2p,
                                                  double t, bool* ovl) {
  const bool y = G.lane & 1;
  const double pos = (&P->x)[y ? 1 : 0], vel = (&P->vx)[y ? 1 : 0];
  const double lat2 = t - P->tl;
  double rad2 = P->rad, vr2 = 0;
  if constexpr (GROW) {
    vr2 = *vr2p;
    rad2 = rad2 + lat2 * vr2;
  }
  return pair_time_flown<GW, ADD, GROW>(B, G, act, p1, v1, rad1, vr1, pos + lat2 * vel, vel, rad2, vr2, ovl);
}

// group-relative lane of the least (time key, scan order), word by word like
// grp_argmin; a lane without a candidate has order -1, the largest word, and
// the least key only when no lane has a candidate
template <int GW>
__device__ __forceinline__ int best_lane(uint64_t k, int o, const Grp<GW>& G) {
  const uint32_t h = (uint32_t)(k >> 32);
  uint32_t m = G.min_u32(h);
  bool in = h == m;
  unsigned q = G.ballot(in);
  if (q & (q - 1)) {
    uint32_t v = in ? (uint32_t)k : 0xffffffffu;
    m = G.min_u32(v);                           // every lane of the group takes part
    in = in && v == m;
    v = in ? (uint32_t)o : 0xffffffffu;
    m = G.min_u32(v);
    in = in && v == m;
    q = G.ballot(in);
  }
  return __ffs(q) - 1;
}

// The candidates of the disks a0 at cell (X0, Y0) and a1 (may be -1) at
// (X1, Y1): the 3x3 neighbour cells, dy outer and dx inner, list order.  The
// (disk, cell) walks are tasks t = 0..8 (a0's cells in scan order) and 9..17
// (a1's): task t runs on lane t % GW, a lane with two tasks walks both lists
// at once.  The candidates are then packed over the group in task order, *tot
// of them, *tot0 for a0.  True when a list is longer than MAXC (nothing
// packed).  `on_cell(cell)` is called for every cell scanned, by the lane that
// walks it; *corrupt is set on a lane whose list is longer than the system.
template <int GW, class F>
__device__ __forceinline__ bool gather(const SysDev& S, int a0, int a1, int X0, int X1, int Y0, int Y1,
                                       const Grp<GW>& G, LaneScratch* sm, int* tot, int* tot0, bool* corrupt,
                                       F&& on_cell) {
  const Box& B = S.B;
  const int lane = G.lane;
  const int ntask = a1 >= 0 ? 18 : 9;
  // the tasks of this lane: t = lane + k GW, k < NT (a warp: one task per
  // lane; 16 lanes: two; 8 lanes: three; 4 lanes: five)
  constexpr int NT = (18 + GW - 1) / GW;
  int pt[NT], ct[NT], ot[NT], qt[NT], hc[NT];
#pragma unroll
  for (int k = 0; k < NT; k++) {
    const int u = lane + k * GW;
    const bool second = u >= 9;
    ot[k] = second ? a1 : a0;
    const int q = second ? u - 9 : u;
    qt[k] = q;
    hc[k] = pbc_cy(B, (second ? Y1 : Y0) + q / 3 - 1) * B.Nxc + pbc_cx(B, (second ? X1 : X0) + q % 3 - 1);
    pt[k] = u < ntask ? S.head[hc[k]] : NIL;
    if (u < ntask) on_cell(hc[k]);
    ct[k] = 0;
  }
  {
    int guard = 0;                   // the lists hold N disks in all
    bool more = true;
    while (more && guard++ < 2 * B.N) {
      more = false;
#pragma unroll
      for (int k = 0; k < NT; k++) {
        if (pt[k] != NIL) {
          const int u = lane + k * GW;
          if (pt[k] != ot[k]) { if (ct[k] < MAXC) sm->reg[u * MAXC + ct[k]] = pt[k]; ct[k]++; }
          pt[k] = S.d[pt[k]].nxt;
          more |= pt[k] != NIL;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NT; k++)
      if (pt[k] != NIL) *corrupt = true;
  }
  bool over = false;
#pragma unroll
  for (int k = 0; k < NT; k++) over |= ct[k] > MAXC;
  if (G.any(over)) return true;
  // exclusive prefix of the counts (at most 7) in task order, bit by bit
  int ex[NT];
  int base = 0;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < NT; k++) {
    const unsigned c0 = G.ballot(ct[k] & 1), c1 = G.ballot(ct[k] & 2), c2 = G.ballot(ct[k] & 4);
    ex[k] = base + __popc(c0 & below) + 2 * __popc(c1 & below) + 4 * __popc(c2 & below);
    base += __popc(c0) + 2 * __popc(c1) + 4 * __popc(c2);
  }
  // a0's candidates are tasks 0..8: their count is the prefix at task 9
  *tot0 = G.shfl(ex[9 / GW], 9 % GW);
  *tot = base;
#pragma unroll
  for (int k = 0; k < NT; k++) {
    const int u = lane + k * GW;
    for (int m = 0; m < ct[k]; m++) {
      sm->comp[ex[k] + m] = sm->reg[u * MAXC + m];
      sm->ord[ex[k] + m] = (int16_t)(qt[k] * MAXC + m);
    }
  }
  G.sync();
  return false;
}

// Candidates found and flown to the event's time by another warp (gather): the
// prediction is then left with the pair solves.
struct Flown { double p[2], v[2], rad, vr; uint32_t coll; int32_t id; };
struct Flock : LaneScratch {
  Flown cand[2 * 9 * MAXC];
  int tot, tot0;
  bool spill, corrupt;
};

// collisionEventNormal / Grow (src/EDMD.c:2829 / 3104) for disks a0 and a1
// (a1 may be -1), both current at t, whose lane roles hold `own`: of the
// candidates (gather) keep the first strict minimum, each solved by two lanes.
// `tag_of(p)` gives 0..3 for a candidate, loaded beside its record.
// ORD: lanes the naming order of overlapping pairs refers to.
// FLOWN: the candidates come from `flock`.
template <int GW, bool ADD, bool GROW, int ORD, bool FLOWN = false, class F, class T>
__device__ __forceinline__ Next predict2(const SysDev& S, double t, int a0, int a1, const Own& own,
                                         uint64_t* npair, const Grp<GW>& G, LaneScratch* sm, bool* ovl, int* ovl_a,
                                         int* ovl_b, F&& on_cell, T&& tag_of, const Flock* flock = nullptr) {
  const Box& B = S.B;
  const int lane = G.lane;
  const double dinit = GROW ? 10000000 : NEVER;
  const uint32_t coll0 = S.d[0].coll;
  const int ntask = a1 >= 0 ? 18 : 9;
  const int X0 = G.shfl(own.c, 0), X1 = G.shfl(own.c, 1), Y0 = G.shfl(own.c, 2), Y1 = G.shfl(own.c, 3);
  // a list longer than N is corrupt: reported like an overlap, with the
  // marker OVL_CORRUPT in place of the first disk (EDMD_ERR_BUDGET)
  bool lcorrupt = false, spill;
  int tot = 0, tot0 = 0;
  if constexpr (FLOWN) {
    tot = flock->tot; tot0 = flock->tot0; spill = flock->spill; lcorrupt = flock->corrupt;
  } else {
    spill = gather(S, a0, a1, X0, X1, Y0, Y1, G, sm, &tot, &tot0, &lcorrupt, on_cell);
  }
  uint64_t bd0 = cand_key(dinit), bd1 = bd0;
  int bo0 = -1, bo1 = -1, bp0 = 0, bp1 = 0;
  uint32_t bc0 = 0, bc1 = 0;
  // of several overlapping pairs the one named is fixed by the order the
  // candidates have when each takes a lane of its own
  uint32_t lk = 0xffffffffu;
  int la = -1, lb = -1;
  if (!spill) {
    for (int f0 = 0; f0 < tot; f0 += GW / 2) {
      const int f = f0 + (lane >> 1);
      const bool act = f < tot;
      const bool g1 = act && f >= tot0;
      const int src = (g1 ? 1 : 0) | ((lane & 1) << 1);
      const double p1 = G.shfl(own.p, src), v1 = G.shfl(own.v, src), rad1 = G.shfl(own.rad, src);
      const double vr1 = GROW ? G.shfl(own.vr, src) : 0.0;
      int p, o;
      uint32_t pc;
      double dt;
      bool ov = false;
      if constexpr (FLOWN) {
        const Flown& P = flock->cand[act ? f : 0];
        p = P.id; o = (int)flock->ord[act ? f : 0] << 2; pc = P.coll;
        dt = pair_time_flown<GW, ADD, GROW>(B, G, act, p1, v1, rad1, vr1, P.p[lane & 1], P.v[lane & 1], P.rad, P.vr, &ov);
      } else {
        p = act ? sm->comp[f] : a0;
        o = act ? (int)sm->ord[f] << 2 | tag_of(p) : 0;
        const Disk* P = S.d + p;
        pc = P->coll;
        dt = pair_time_lanes<GW, ADD, GROW>(B, G, act, p1, v1, rad1, vr1, P, S.vr + p, t, &ov);
      }
      const uint64_t kd = cand_key(dt);
      if (ov) {
        const uint32_t k = ((uint32_t)(f % ORD) << 16) | (0xffffu - (uint32_t)f);
        if (k < lk) { lk = k; la = g1 ? a1 : a0; lb = p; }
      }
      if (g1) best_merge(bd1, bo1, bp1, bc1, kd, o, p, pc);
      else if (act) best_merge(bd0, bo0, bp0, bc0, kd, o, p, pc);
    }
    G.sync();
  } else {
    // a cell list longer than MAXC: the lists are walked again, one after the
    // other, every pair by the first two lanes
    tot = 0;
#pragma unroll 1
    for (int u = 0; u < ntask; u++) {
      const bool g1 = u >= 9;
      const int q = g1 ? u - 9 : u, a = g1 ? a1 : a0;
      const int src = (g1 ? 1 : 0) | ((lane & 1) << 1);
      const double p1 = G.shfl(own.p, src), v1 = G.shfl(own.v, src), rad1 = G.shfl(own.rad, src);
      const double vr1 = GROW ? G.shfl(own.vr, src) : 0.0;
      int p = S.head[pbc_cy(B, (g1 ? Y1 : Y0) + q / 3 - 1) * B.Nxc + pbc_cx(B, (g1 ? X1 : X0) + q % 3 - 1)];
      int k = 0, guard = 0;
      while (p != NIL && guard++ < B.N) {
        const Disk* P = S.d + p;
        const int nx = P->nxt;
        if (p != a) {
          bool ov = false;
          const uint64_t kd =
              cand_key(pair_time_lanes<GW, ADD, GROW>(B, G, true, p1, v1, rad1, vr1, P, S.vr + p, t, &ov));
          if (ov) {
            const uint32_t w = ((uint32_t)(u % ORD) << 16) | (0xffffu - (uint32_t)(u * 2048 + min(k, 2047)));
            if (w < lk) { lk = w; la = a; lb = p; }
          }
          if (g1) best_merge(bd1, bo1, bp1, bc1, kd, (q * (1 << 20) + k) << 2 | tag_of(p), p, P->coll);
          else best_merge(bd0, bo0, bp0, bc0, kd, (q * (1 << 20) + k) << 2 | tag_of(p), p, P->coll);
          k++;
        }
        p = nx;
      }
      if (p != NIL) lcorrupt = true;
      tot += k;
    }
  }
  *npair += (uint64_t)tot;
  // lexicographic (dt, scan order) minimum over the group
  Next r;
  {
    const int w0 = best_lane(bd0, bo0, G);
    bd0 = G.shfl(bd0, w0); bo0 = G.shfl(bo0, w0); bp0 = G.shfl(bp0, w0); bc0 = G.shfl(bc0, w0);
  }
  if (a1 >= 0) {
    const int w1 = best_lane(bd1, bo1, G);
    bd1 = G.shfl(bd1, w1); bo1 = G.shfl(bo1, w1); bp1 = G.shfl(bp1, w1); bc1 = G.shfl(bc1, w1);
    if (lane & 1) { bd0 = bd1; bo0 = bo1; bp0 = bp1; bc0 = bc1; }
  }
  if (bo0 < 0) bc0 = coll0;         // no partner: partner 0 (src/EDMD.c:2830)
  r.key = bd0; r.partner = bp0; r.ca = bc0;
  r.q = bo0 < 0 ? 4 : spill ? bo0 >> 22 : (bo0 >> 2) / MAXC;
  r.tag = bo0 & 3;
  if (G.any(lk != 0xffffffffu || lcorrupt)) {
    const uint32_t least = G.min_u32(lk);
    const int src = G.first(lk == least && lk != 0xffffffffu);
    *ovl = true;
    if (src >= 0) { *ovl_a = G.shfl(la, src); *ovl_b = G.shfl(lb, src); }
    if (G.any(lcorrupt)) { *ovl_a = OVL_CORRUPT; *ovl_b = a0; }
  }
  return r;
}

// a contact from its lanes: r_j - r_i (nearest image) and v_j - v_i along the
// lane's axis, the same on both disks' lanes; the other disk's mass and radius
struct Meet { double d, dv, mo, ro; };
template <int GW>
__device__ __forceinline__ Meet meet_lanes(const Box& B, const Grp<GW>& G, const Own& own, double m) {
  const bool odd = G.lane & 1, y = G.lane & 2;
  const double po = G.shfl_xor(own.p, 1), vo = G.shfl_xor(own.v, 1);
  Meet c;
  c.mo = G.shfl_xor(m, 1);
  c.ro = G.shfl_xor(own.rad, 1);
  c.d = near_image((odd ? own.p : po) - (odd ? po : own.p), y ? B.hLy : B.hLx, y ? B.Ly : B.Lx);
  c.dv = (odd ? own.v : vo) - (odd ? vo : own.v);
  return c;
}

// The elastic rule (src/EDMD.c:3802-3827) on a contact's lanes: own.v becomes
// the new velocity, ctl gains virial term lane % 4 (collTermX, Y, XY, YX; on
// quad 1, lanes 4..7, where the group has one), f and r = (dx, dy) come back.
// inv = (1 / (m_i + m_j)) (1 + res).  Independent products share one FP64
// instruction over quads of lanes; operations and roundings are the
// reference's (a - x as a + (-x), 4 r and x / 4 are exact, products commute).
template <int GW, bool ADD>
__device__ __forceinline__ double elastic_lanes(const Box& B, const Grp<GW>& G, Own& own, double m, const Meet& c,
                                                double inv, double& ctl, double* dxo, double* dyo) {
  const int lane = G.lane, quad = (lane >> 2) & 3;
  const bool odd = lane & 1, y = lane & 2;
  // r . v by axis, sigma^2, m_i m_j
  double sa = times4(own.rad), sb = c.ro;
  if (ADD && B.additive) sa = sb = own.rad + c.ro;
  double pr, sig2, mm;
  if constexpr (GW >= 16) {
    const double r = (quad == 0 ? c.d : quad == 1 ? sa : m) * (quad == 0 ? c.dv : quad == 1 ? sb : c.mo);
    sig2 = G.shfl(r, 4);
    mm = G.shfl(r, 8);
    pr = G.shfl(r, 0) + G.shfl(r, 2);
  } else if constexpr (GW == 8) {
    const double r = (quad & 1 ? sa : c.d) * (quad & 1 ? sb : c.dv);
    sig2 = G.shfl(r, 4);
    mm = m * c.mo;
    pr = G.shfl(r, 0) + G.shfl(r, 2);
  } else {
    sig2 = sa * sb;
    mm = m * c.mo;
    pr = c.d * c.dv;
    pr += G.shfl_xor(pr, 2);
  }
  const double kernel = inv * pr;
  const double f = __double_as_longlong(sig2) == 0x4010000000000000ll ? kernel * 0.25 : div_rn(kernel, sig2);
  const double od = G.shfl_xor(c.d, 2);
  const double dx = y ? od : c.d, dy = y ? c.d : od;
  const double ra = odd ? dy : dx, rb = y == odd ? dx : dy;
  if constexpr (GW >= 8) {
    const bool vir = (lane >> 2) == 1;
    const double w1 = f * (vir ? mm : c.mo);
    const double w2 = w1 * (vir ? ra : c.d);
    const double w3 = w2 * rb;
    const double s = (vir ? ctl : own.v) + (vir ? w3 : flip(w2, odd));
    if (vir) ctl = s;
    else own.v = s;
  } else {
    ctl += mm * f * ra * rb;
    own.v += flip(f * c.mo * c.d, odd);
  }
  *dxo = dx;
  *dyo = dy;
  return f;
}
// the lane that holds virial term k after elastic_lanes
template <int GW>
__device__ __forceinline__ constexpr int virial_lane(int k) { return GW >= 8 ? 4 + k : k; }

}  // namespace edmd
