// edmd_engine.cu -- serial-exact event engine (one or two warps per system) and the C ABI.
//
// Each system is advanced by a warp (with a second one beside it in contexts of
// few systems) that pops events in exactly the order of the reference's queue
// (src/EDMD.c:2144-2327: a calendar of N buckets of width 5/N plus an overflow
// bucket, feeding an unbalanced BST whose in-order ties go to the later
// insertion).  That order is emulated by the key
//     (b, t, tie)
// b   = absolute calendar bucket in which the event enters the BST,
// t   = event time,
// tie = class and counter reproducing the BST insertion order inside a bucket:
//       class 0  re-added directly into the BST by an overflow wrap (inserted
//                before the bucket's own list is loaded), ascending counter;
//       class 1  pushed onto a bucket list (LIFO: loaded last-pushed-first),
//                descending counter;
//       class 2  inserted directly because it falls in the current bucket,
//                ascending counter.
// The keys live in a 32-ary tournament tree (level 0 = one leaf per disk, the
// minimum of its crossing and collision events, plus three special events);
// each tree level is fixed by one coalesced load and hardware reductions.
// Collision prediction packs the candidates of the 3x3 neighbour cells of the
// (up to two) disks that changed into the lanes of the warp.
#include "edmd_lanes.cuh"
#include "../../include/edmd_gpu.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <vector>

using namespace edmd;

namespace edmd {
cudaError_t lane_build(const SysDev* ds, int nsys, cudaStream_t st);
cudaError_t lane_run_launch(const SysDev* ds, const RunArgs& A, int threads_per_block, cudaStream_t st);
}

#define FULL 0xffffffffu

namespace {

constexpr int WARPS_PER_BLOCK = 4;

// scratch of one lane group (one system)
struct WarpSmem : LaneScratch {
  long long msum[2];             // last two mass sums of the collision rule (bits) ...
  double inv[2];                 // ... and (1 / msum) (1 + res), the same operations' result
};


__device__ __forceinline__ Node empty_node(int idx) {
  Node n; n.tk = ~0ull; n.tie = ~0ull; n.b = BINF; n.idx = idx;
  return n;
}

__device__ __forceinline__ bool node_less(const Node& a, const Node& b) {
  return key_less(a.b, a.tk, a.tie, a.idx, b.b, b.tk, b.tie, b.idx);
}

// Group-relative lane of the least node: word by word from the top of the key
// (b, time, tie, idx), each word's minimum by one redux instruction.  The
// first two words (bucket and the upper half of the time) decide almost
// always.  A butterfly that moves whole 24-byte nodes takes five steps of six
// shuffles and a four-word compare; a redux takes 28 cycles where one shuffle
// takes 42.
template <int GW>
__device__ __forceinline__ int grp_argmin(const Node& n, const Grp<GW>& G) {
  const uint32_t mb = G.min_u32(n.b);
  bool in = n.b == mb;
  auto next = [&](uint32_t w) {
    const uint32_t v = in ? w : 0xffffffffu;
    const uint32_t m = G.min_u32(v);            // every lane of the group takes part
    in = in && v == m;
  };
  next((uint32_t)(n.tk >> 32));
  unsigned q = G.ballot(in);
  if (q & (q - 1)) {
    next((uint32_t)n.tk);
    next((uint32_t)(n.tie >> 32));
    next((uint32_t)n.tie);
    next((uint32_t)n.idx);
    q = G.ballot(in);
  }
  return __ffs(q) - 1;
}

// this lane's child of node `par` of level h-1 (the least of its 32 / GW
// children), with the nodes at ia and ib taken from na and nb (T, cnt: that level)
template <int GW>
__device__ __forceinline__ Node child_node(const Node* __restrict__ T, int cnt, int par, int ia, const Node& na, int ib,
                                           const Node& nb, const Grp<GW>& G) {
  Node c = empty_node(0x7fffffff);
#pragma unroll
  for (int k = 0; k < 32; k += GW) {
    const int ch = (par << 5) + k + G.lane;
    Node m = empty_node(0x7fffffff);
    if (ch == ia) m = na;
    else if (ch == ib) m = nb;
    else if (ch < cnt) m = T[ch];
    if (GW == 32 || node_less(m, c)) c = m;
  }
  return c;
}
template <int GW>
__device__ __forceinline__ Node child_node(const SysDev& S, int h, int par, int ia, const Node& na, int ib,
                                           const Node& nb, const Grp<GW>& G) {
  return child_node(S.tree + S.lev_off[h - 1], S.lev_cnt[h - 1], par, ia, na, ib, nb, G);
}

__device__ __forceinline__ Node ev_node(const Ev& e, int idx) {
  Node n; n.tk = time_key(e.t); n.tie = e.tie; n.b = e.b; n.idx = idx;
  return n;
}

// a leaf's node: the earlier of its events, with that event's slot
__device__ __forceinline__ Node leaf_node(const SysDev& S, int leaf) {
  const int N = S.B.N;
  const int slot = leaf < N ? leaf : N + leaf;           // disk: crossing slot; special: 2N + (leaf - N)
  Node n = empty_node(slot);
  const Ev e0 = S.ev[slot];
  if (e0.st == ST_QUEUED) n = ev_node(e0, slot);
  if (leaf < N) {
    const Ev e1 = S.ev[N + leaf];
    if (e1.st == ST_QUEUED) { const Node m = ev_node(e1, N + leaf); if (node_less(m, n)) n = m; }
  }
  return n;
}

template <int GW>
__device__ __forceinline__ Node shfl_node(const Node& n, int src, const Grp<GW>& G) {
  Node r;
  r.tk = G.shfl(n.tk, src); r.tie = G.shfl(n.tie, src);
  r.b = G.shfl(n.b, src); r.idx = G.shfl(n.idx, src);
  return r;
}

// the leaves la and lb (lb < 0: none) become na and nb: fix their paths to
// the root, both paths level by level.  A parent they share is reduced once,
// and a node just changed is carried in registers, so no level waits for the
// stores of the one below it.
template <int GW>
__device__ __forceinline__ void path_update(const SysDev& S, int la, int lb, Node na, Node nb, const Grp<GW>& G) {
  const int lane = G.lane;
  if (lane == 0) S.tree[la] = na;
  if (lane == 1 && lb >= 0) S.tree[lb] = nb;
  int ia = la, ib = lb;
#pragma unroll 1
  for (int h = 1; h < S.nlev; h++) {
    Node* T = S.tree + S.lev_off[h];
    const int pa = ia >> 5, pb = ib >> 5;       // pb = -1: one path (left)
    const Node ca = child_node(S, h, pa, ia, na, ib, nb, G);
    Node cb = ca;
    if (pb >= 0 && pb != pa) cb = child_node(S, h, pb, ib, nb, -1, nb, G);
    int src = grp_argmin(ca, G);
    if (lane == src) T[pa] = ca;
    na = shfl_node(ca, src, G);
    ia = pa;
    ib = -1;
    if (pb >= 0 && pb != pa) {
      src = grp_argmin(cb, G);
      if (lane == src) T[pb] = cb;
      nb = shfl_node(cb, src, G);
      ib = pb;
    }
  }
  G.sync();
}

// one leaf recomputed from its events
template <int GW>
__device__ __forceinline__ void leaf_update(const SysDev& S, int leaf, const Grp<GW>& G) {
  const Node n = leaf_node(S, leaf);
  path_update(S, leaf, -1, n, n, G);
}

// rebuild every level of the tree (after init or the growth stop)
template <int GW>
__device__ __noinline__ void tree_rebuild(const SysDev& S, const Grp<GW>& G) {
  const int lane = G.lane;
  for (int l = lane; l < S.L; l += GW) S.tree[l] = leaf_node(S, l);
  G.sync();
#pragma unroll
  for (int h = 1; h < MAXLEV; h++) {
    if (h >= S.nlev) break;
    for (int par = 0; par < S.lev_cnt[h]; par++) {
      const Node none = empty_node(0x7fffffff);
      const Node c = child_node(S, h, par, -1, none, -1, none, G);
      if (lane == grp_argmin(c, G)) S.tree[S.lev_off[h] + par] = c;
    }
    G.sync();
  }
}

// ---------------------------------------------------------------- queue

// the queue's scalar state; out-of-line functions take and return it by value,
// so that the event loop's copy stays in registers
struct Queue {
  double P;                      // paulTime of the current bucket
  uint64_t C, k, next_wrap;      // insertion counter, current bucket, next overflow wrap
  int32_t ovf;                   // head of the overflow list
};
__device__ __forceinline__ Queue queue_of(const SysState& R) {
  Queue q;
  q.P = R.P; q.C = R.C; q.k = R.k; q.next_wrap = R.next_wrap; q.ovf = R.ovf;
  return q;
}
__device__ __forceinline__ void queue_to(SysState& R, const Queue& q) {
  R.P = q.P; R.C = q.C; R.k = q.k; R.next_wrap = q.next_wrap; R.ovf = q.ovf;
}

// addEventToQueue (src/EDMD.c:2144) in key form, in two parts: where the
// event goes (FP64: its offset from paulTime; -1 current bucket, -2
// overflow, else the bucket offset), and the insertion (integer work).
__device__ __forceinline__ int sched_place(const SysDev& S, const Queue& R, double T) {
  const Box& B = S.B;
  const double dt = T - R.P;
  if (!ge_pos(dt, B.dtP)) return -1;           // dt < dtPaul
  if (ge_pos(dt, B.dtPN)) return -2;           // dt >= dtPaul * N
  return bucket_offset(dt, B.dtP, S.rdtP);
}

// queue key and state of an event placed at `place` with insertion counter C;
// `cls_direct` is 2 for a schedule from an event handler and 0 for the
// re-add done by a wrap
__device__ __forceinline__ void sched_key(const Queue& R, uint64_t C, uint64_t cls_direct, int place, Ev& ev) {
  if (place == -1) {
    ev.b = (uint32_t)R.k; ev.tie = (cls_direct << 62) | C; ev.st = ST_QUEUED;
  } else if (place == -2) {
    ev.b = BINF; ev.tie = C; ev.st = ST_OVF;
  } else {
    ev.b = (uint32_t)(R.k + (uint64_t)place); ev.tie = (1ull << 62) | (TIE_MAX - C); ev.st = ST_QUEUED;
  }
}

template <int GW>
__device__ __forceinline__ void sched_insert(const SysDev& S, Queue& R, int e, double T, int32_t j,
                                             uint32_t ca, uint64_t cls_direct, int place, const Grp<GW>& G) {
  const int lane = G.lane;
  Ev ev;
  ev.t = T; ev.j = j; ev.ca = ca;
  sched_key(R, R.C, cls_direct, place, ev);
  if (place == -2) {
    if (lane == 0) {
      S.on[e] = R.ovf; S.op[e] = NIL;
      if (R.ovf != NIL) S.op[R.ovf] = e;
    }
    R.ovf = e;
  }
  R.C++;
  if (lane == 0) S.ev[e] = ev;
  G.sync();
}

template <int GW>
__device__ void schedule(const SysDev& S, Queue& R, int e, double T, int32_t j, uint32_t ca,
                         uint64_t cls_direct, const Grp<GW>& G) {
  sched_insert(S, R, e, T, j, ca, cls_direct, sched_place(S, R, T), G);
}

// removeEventFromQueue (src/EDMD.c:2209) in key form
template <int GW>
__device__ void unqueue(const SysDev& S, Queue& R, int e, const Grp<GW>& G) {
  const int lane = G.lane;
  uint32_t st = S.ev[e].st;
  if (st == ST_OVF) {
    int p = S.op[e], n = S.on[e];
    if (lane == 0) {
      if (p != NIL) S.on[p] = n;
      if (n != NIL) S.op[n] = p;
    }
    if (p == NIL) R.ovf = n;
  }
  if (lane == 0) S.ev[e].st = ST_NONE;
  G.sync();
}

// the overflow bucket is redistributed when the calendar wraps
// (addNextPaulEvent src/EDMD.c:2287-2300)
// (head OVF_CORRUPT: the list is longer than it can be, i.e. corrupt)
constexpr int32_t OVF_CORRUPT = -2;
template <int GW>
__device__ __noinline__ Queue do_wrap(const SysDev& S, Queue R, Grp<GW> G) {
  const int N = S.B.N;
  int e = R.ovf;
  R.ovf = NIL;
  G.sync();
  int guard = 0;                       // the overflow list holds at most 2N + 3 events
  while (e != NIL && guard++ <= 2 * N + NSPECIAL) {
    int n = S.on[e];
    double T = S.ev[e].t;
    int32_t j = S.ev[e].j;
    uint32_t ca = S.ev[e].ca;
    schedule(S, R, e, T, j, ca, 0ull, G);
    G.sync();
    int leaf = e < 2 * N ? (e < N ? e : e - N) : N + (e - 2 * N);
    leaf_update(S, leaf, G);
    e = n;
  }
  R.next_wrap += (uint64_t)N;
  if (e != NIL) R.ovf = OVF_CORRUPT;
  return R;
}

// ---------------------------------------------------------------- prediction

__device__ __forceinline__ void grow_fly(const SysDev& S, Disk& p, int i, double t, bool grow) {
  double dt = t - p.tl;
  free_fly_i(S.B, p, t);
  if (grow) p.rad += dt * S.vr[i];
}

// ---------------------------------------------------------------- handlers


// sequential sum over disks, in index order, identical in all lanes
template <int GW, class F>
__device__ __forceinline__ void seq_sums(const SysDev& S, const Grp<GW>& G, int nval, double* out, F f) {
  const int lane = G.lane;
  const int N = S.B.N;
  for (int k = 0; k < nval; k++) out[k] = 0;
  for (int base = 0; base < N; base += GW) {
    double v[4] = {0, 0, 0, 0};
    int i = base + lane;
    if (i < N) f(i, v);
    int lim = min(GW, N - base);
    for (int s = 0; s < lim; s++)
      for (int k = 0; k < nval; k++) out[k] += G.shfl(v[k], s);
  }
}

// physicalQ (src/EDMD.c:5968-6013): px, py, E
template <int GW>
__device__ __noinline__ void physical_q(const SysDev& S, const Grp<GW>& G, double* E, double* px, double* py) {
  double o[3];
  seq_sums(S, G, 3, o, [&](int i, double* v) {
    Disk p = S.d[i];
    v[0] = p.vx * p.m;
    v[1] = p.vy * p.m;
    double vx = p.vx;
    v[2] = 0.5 * p.m * (vx * vx + p.vy * p.vy);
  });
  *px = o[0]; *py = o[1]; *E = o[2];
}

// takeAThermo + saveThermo (src/EDMD.c:4679, 5232-5697) with Nthermo = 1
template <int GW>
__device__ void do_thermo(const SysDev& S, SysState& R, const Grp<GW>& G) {
  const int lane = G.lane;
  const int N = S.B.N;
  double E, px, py;
  physical_q(S, G, &E, &px, &py);
  double area = S.B.Lx * S.B.Ly;
  double dT = R.t - R.lastThermo;
  R.lastThermo = R.t;
  double e4[4];
  seq_sums(S, G, 4, e4, [&](int i, double* v) {
    Disk p = S.d[i];
    v[0] = p.m * p.vx * p.vx; v[1] = p.m * p.vy * p.vy;
    v[2] = p.m * p.vx * p.vy; v[3] = p.m * p.vy * p.vx;
  });
  double row[9];
  row[0] = R.t; row[1] = (double)R.ncol; row[2] = E / N;
  row[4] = -1 * R.collT[0] / (area * dT) + e4[0] / area;
  row[5] = -1 * R.collT[1] / (area * dT) + e4[1] / area;
  row[6] = -1 * R.collT[2] / (area * dT) + e4[2] / area;
  row[7] = -1 * R.collT[3] / (area * dT) + e4[3] / area;
  row[3] = (-1 / (dT)) * (R.collT[0] + R.collT[1]) / (2 * area) + E / area;
  R.collT[0] = R.collT[1] = R.collT[2] = R.collT[3] = 0;
  double vxa;
  seq_sums(S, G, 1, &vxa, [&](int i, double* v) { v[0] = S.d[i].vx; });
  vxa /= N;
  double v24[2];
  seq_sums(S, G, 2, v24, [&](int i, double* v) {
    double d = S.d[i].vx - vxa; double d2 = d * d; v[0] = d2; v[1] = d2 * d2;
  });
  v24[0] /= N; v24[1] /= N;
  row[8] = (v24[0] > 0.0) ? v24[1] / (3.0 * v24[0] * v24[0]) - 1.0 : 0.0;
  if (R.t != 0) {
    if (R.nrows < S.rows_cap && lane == 0)
      for (int k = 0; k < 9; k++) S.rows[(int64_t)R.nrows * 9 + k] = row[k];
    R.nrows++;
  }
}

// stopGrow (src/EDMD.c:4740-4800)
template <int GW, bool ADD>
__device__ void do_growstop(const SysDev& S, SysState& R, const Grp<GW>& G, WarpSmem* sm,
                            bool* ovl, int* oa, int* ob) {
  const int lane = G.lane;
  const int N = S.B.N;
  for (int i = lane; i < N; i += GW) {
    Disk p = S.d[i];
    grow_fly(S, p, i, R.t, true);
    p.coll = 0;
    S.d[i] = p;
    S.crossX[i] = 0; S.crossY[i] = 0;
  }
  R.ncol = 0; R.ncross = 0;
  R.grow = 0;
  G.sync();
  // normalizePhysicalQ (src/EDMD.c:5723-5764)
  double E, px, py;
  physical_q(S, G, &E, &px, &py);
  for (int i = lane; i < N; i += GW) {
    Disk p = S.d[i];
    p.vx -= px / (N * p.m);
    p.vy -= py / (N * p.m);
    S.d[i] = p;
  }
  G.sync();
  physical_q(S, G, &E, &px, &py);
  for (int i = lane; i < N; i += GW) {
    Disk p = S.d[i];
    p.vx /= sqrt(E / N / S.Einit);
    p.vy /= sqrt(E / N / S.Einit);
    S.d[i] = p;
  }
  G.sync();
  Queue Q = queue_of(R);
  for (int i = 0; i < N; i++) {
    uint32_t c = S.d[i].coll + 1;
    if (lane == 0) S.d[i].coll = c;
    G.sync();
    unqueue(S, Q, N + i, G);
    Own own;
    own.p = *axis_pos(S.d + i, lane & 2); own.v = *axis_vel(S.d + i, lane & 2); own.rad = S.d[i].rad;
    own.vr = 0;
    own.c = (lane & 2 ? S.cy : S.cx)[i];
    R.npred++;
    const Next r = predict2<GW, ADD, false, GW>(S, R.t, i, -1, own, &R.npair, G, sm, ovl, oa, ob, [](int) {}, [](int) { return 0; });
    schedule(S, Q, N + i, R.t + key_time(r.key), r.partner, r.ca, 2ull, G);
    unqueue(S, Q, i, G);
    int dir;
    Disk p = S.d[i];
    double tc = crossing_time_i(S.B, p, S.cx[i], S.cy[i], R.t, &dir);
    schedule(S, Q, i, tc, dir, 0, 2ull, G);
    G.sync();
  }
  queue_to(R, Q);
  tree_rebuild(S, G);
}

// offset of the next crossing of the lane's disk and its direction
// (src/EDMD.c:2405-2482), one axis per lane
template <int GW>
__device__ __forceinline__ double next_crossing(const Box& B, const Grp<GW>& G, int c, double p, double v, int* dir) {
  const bool ydim = G.lane & 2;
  const bool neg = is_neg(v);
  const double a = near_image((neg ? c : 1 + c) * (ydim ? B.cys : B.cxs) - p, ydim ? B.hLy : B.hLx,
                              ydim ? B.Ly : B.Lx);
  const double ta = div_rn(a, v);
  const int da = (ydim ? 3 : 1) + (neg ? 0 : 1);
  const double tb = G.shfl_xor(ta, 2);
  const int db = G.shfl_xor(da, 2);
  const bool ux = lt_i(ydim ? tb : ta, ydim ? ta : tb);
  *dir = ux == ydim ? db : da;
  return ux == ydim ? tb : ta;
}

// ---------------------------------------------------------------- two warps on one system

// What the two warps of a system exchange (k_run_pair): the first runs the
// event loop, the second does beside it whatever does not need the outcome of
// the event, or is not needed before the next one.
struct Aside : Flock {
  // the event (first warp): disk i (or an order below), disk j of a collision
  // or the direction of a crossing, the partner's counter, the time, and the
  // calendar: paulTime of bucket k, the event's bucket b
  int i, j;
  bool coll, grow;
  uint32_t ca, b;
  double t, P;
  uint64_t k;
  double p[4], v[4];             // outcome (first warp): coordinate and velocity of the lane roles
  Node leaf[2];                  // the changed leaves (first warp)
  double tc[2];                  // next crossings (second warp): offset from t, direction
  int dir[2];
  double Pb;                     // paulTime of bucket b (second warp)
  Node rest;                     // least of the leaves that the event leaves alone (second warp)
  int self[2];                   // where disk i's candidates hold j, and j's hold i (-1: they don't); one place
                                 // each, since a 3x3 scan of at least three cells an axis meets a disk once
  Node sibs[MAXLEV][2];          // least sibling of each path node, by level
  int off[MAXLEV], cnt[MAXLEV];  // the tree's levels
};
constexpr int ASIDE_END = -1, ASIDE_FLUSH = -2;

// Both warps of a block meet here, three times an event: [A] the event is
// known, [B] its outcome is, and the candidates are flown, [C] the crossings
// and the rest of the tree are.  Neither leaves the event loop between A and C.
__device__ __forceinline__ void pair_barrier() {
  __syncwarp();
  asm volatile("barrier.sync 1, 64;" ::: "memory");
}

// after this the tree in memory is up to date (first warp)
__device__ __forceinline__ void pair_flush(Aside* as, int lane) {
  if (lane == 0) as->i = ASIDE_FLUSH;
  pair_barrier();
  pair_barrier();                             // i has been read
}

// The second warp.  Between A and B: the candidates of the disks that change,
// flown to the event's time.  It reads the state before the event, into which
// the first warp stores nothing until B; what the event changes is known: a
// crossing disk's cell, and the colliding disks' own records, which the first
// warp fills in (self).  Between B and C, while the first warp solves the pairs:
// the next crossings, the calendar's walk to the event, the paths of the last
// event's leaves in the tree, and the least siblings along this event's paths.
// Their minimum and the new leaves are all the first warp needs for the next
// event, so the tree itself is one event late (pair_flush).
__device__ __forceinline__ void run_aside(const SysDev& S, Grp<32> G, Aside* as) {
  const int lane = G.lane;
  const bool odd = lane & 1, ydim = lane & 2;
  const Box& B = S.B;
  int li = -1, lj = -1;                       // the last event's leaves
  const int nlev = S.nlev;
  for (int h = lane; h < nlev; h += 32) { as->off[h] = S.lev_off[h]; as->cnt[h] = S.lev_cnt[h]; }
  G.sync();
  auto fix_paths = [&]() {
    if (li < 0) return;
    Node na = as->leaf[0], nb = as->leaf[1];
    if (lane == 0) S.tree[li] = na;
    if (lane == 1 && lj >= 0) S.tree[lj] = nb;
    int ia = li, ib = lj;
#pragma unroll 1
    for (int h = 1; h < nlev; h++) {
      Node* T = S.tree + as->off[h];
      const Node sa = as->sibs[h][0], sb = as->sibs[h][1];
      ia >>= 5;
      ib >>= 5;                               // -1: one path (left)
      if (ib == ia) {
        if (node_less(nb, na)) na = nb;
        ib = -1;
      }
      if (node_less(sa, na)) na = sa;
      if (ib >= 0 && node_less(sb, nb)) nb = sb;
      if (lane == 0) T[ia] = na;
      if (lane == 1 && ib >= 0) T[ib] = nb;
    }
    li = -1;
    G.sync();
  };
  for (;;) {
    pair_barrier();                                                    // A
    const int i = as->i;
    if (i < 0) {
      fix_paths();
      if (i == ASIDE_END) break;
      pair_barrier();
      continue;
    }
    const bool coll = as->coll, grow = as->grow;
    const double t = as->t;
    const int w = as->j;
    const bool stale = coll && S.d[w].coll != as->ca;
    const int j = coll && !stale ? w : -1;
    const int my = odd && j >= 0 ? j : i;
    int c = (ydim ? S.cy : S.cx)[my];
    if (!coll && ydim == (w >= 3)) {
      const int n = ydim ? B.Nyc : B.Nxc;
      c = w & 1 ? (c == 0 ? n - 1 : c - 1) : (c + 1 == n ? 0 : c + 1);
    }
    int tot = 0, tot0 = 0;
    bool corrupt = false;
    const bool spill = gather(S, i, j, G.shfl(c, 0), G.shfl(c, 1), G.shfl(c, 2), G.shfl(c, 3), G, as, &tot, &tot0,
                              &corrupt, [](int) {});
    corrupt = G.any(corrupt);
    if (lane < 2) as->self[lane] = -1;
    if (lane == 0) { as->tot = tot; as->tot0 = tot0; as->spill = spill; as->corrupt = corrupt; }
    G.sync();
    if (!spill)
      for (int f = lane >> 1; f < tot; f += 16) {
        const int p = as->comp[f], y = lane & 1;
        const Disk* P = S.d + p;
        Flown& F = as->cand[f];
        const double vel = (&P->vx)[y], lat = t - P->tl;
        F.p[y] = (&P->x)[y] + lat * vel;
        F.v[y] = vel;
        double rad = P->rad, vr = 0;
        if (grow) { vr = S.vr[p]; rad = rad + lat * vr; }
        if (!y) {
          F.rad = rad; F.vr = vr; F.coll = P->coll; F.id = p;
          if (p == (f < tot0 ? j : i)) as->self[f < tot0 ? 0 : 1] = f;
        }
      }
    pair_barrier();                                                    // B
    if (!stale) {
      int dir;
      const double tc = next_crossing(B, G, c, as->p[lane & 3], as->v[lane & 3], &dir);
      if (lane < 2) { as->tc[lane] = tc; as->dir[lane] = dir; }
    }
    double P = as->P;
    for (uint64_t k = as->k; k < as->b; k++) P += B.dtP;
    if (lane == 0) as->Pb = P;
    fix_paths();
    // a level's nodes are loaded while those of the level below are compared
    Node rest = empty_node(0x7fffffff);
    const Node none = rest;
    int ia = i, ib = j;
    auto load = [&](int h, Node& ca, Node& cb) {
      const Node* T = S.tree + as->off[h - 1];
      const int cnt = as->cnt[h - 1], pa = ia >> 5, pb = ib >> 5;
      ca = child_node(T, cnt, pa, ia, none, ib, none, G);
      const bool apart = pb >= 0 && pb != pa;
      if (apart) cb = child_node(T, cnt, pb, ib, none, -1, none, G);
      ia = pa;
      ib = apart ? pb : -1;
      return apart;
    };
    Node ca, cb = none, da, db = none;
    bool apart = load(1, ca, cb), next = false;
#pragma unroll 1
    for (int h = 1; h < nlev; h++) {
      if (h + 1 < nlev) next = load(h + 1, da, db);
      int src = grp_argmin(ca, G);
      if (lane == src) as->sibs[h][0] = ca;
      if (node_less(ca, rest)) rest = ca;
      if (apart) {
        src = grp_argmin(cb, G);
        if (lane == src) as->sibs[h][1] = cb;
        if (node_less(cb, rest)) rest = cb;
      }
      ca = da; cb = db; apart = next;
    }
    if (lane == grp_argmin(rest, G)) as->rest = rest;
    li = i; lj = j;
    pair_barrier();                                                    // C
  }
}

// ---------------------------------------------------------------- run loop

// what ends a stretch of disk events
enum { END_STOP, END_SPECIAL, END_SHARE };

// A stretch of disk events of one system: until a stop, or a special event
// (screenshot, thermo, growth stop), which is taken off the queue and left in
// *special.  One event is one chain of dependent instructions, so its latency
// is what counts (a single system), and its FP64 instructions and code size (a
// full GPU).  Both disks and both axes share the scalar FP64 work (struct
// Own), the two or four events an event schedules are placed and stored by one
// lane each, a changed leaf of the tree is built from those lanes' registers,
// and the scalar state is held in registers: the growth phase has its own copy
// of the loop, and everything rare is left to serve_special.
// ADD = false: a context without additive-contact systems (the rule's
// switch compiled out of the pair solves and the collision rule)
// PAIR: a second warp works beside this one (run_aside).
template <int GW, bool ADD, bool GROW, bool PAIR>
__device__ __forceinline__ int run_events(const SysDev& S, const RunArgs& A, int64_t max_coll, const Grp<GW>& G,
                                          WarpSmem* sm, Aside* as, int64_t& logged, int64_t& nev, int64_t share_end,
                                          int* special) {
  const int lane = G.lane;
  const bool odd = lane & 1, ydim = lane & 2;
  const Box& B = S.B;
  const int N = B.N;
  SysState* const st = S.st;
  double t = st->t;
  Queue Q = queue_of(*st);
  // the four virial sums: lane l accumulates term l % 4 (see elastic_lanes)
  double ctl = st->collT[lane & 3];
  const double tmax = S.tmax;
  const double onepr = 1 + S.res;
  // (1 + res) / (m_i + m_j) of the last two mass sums: a repeated quotient and
  // product give the same bits.  2 is first (1 / 2 is exact); no sum is +0
  if (lane == 0) {
    sm->msum[0] = 0x4000000000000000ll; sm->inv[0] = 0.5 * onepr;
    sm->msum[1] = 0; sm->inv[1] = 0;
  }
  G.sync();
  const int root = S.lev_off[S.nlev - 1];
  Node top;                                   // PAIR: the root
  if constexpr (PAIR) top = S.tree[root];
  uint64_t ncoll = 0, nstale = 0, npair = 0, nlog = st->nlog;
  const uint64_t ntrace0 = st->ntrace;
  const int64_t nev0 = nev;
  int stop = 0, status = EDMD_OK, end = END_STOP;
  bool ovl = false;
  int oa = -1, ob = -1;
  for (;;) {
    if (!le_i(t, tmax)) { stop = EDMD_STOP_TMAX; break; }
    if (logged >= max_coll) { stop = EDMD_STOP_COLL; break; }
    if (nev >= share_end) {
      if (nev >= A.max_events) status = EDMD_ERR_BUDGET;
      else end = END_SHARE;
      break;
    }
    Node r = top;
    int guard = 0;
    for (;;) {
      if constexpr (!PAIR) r = S.tree[root];
      if (r.b == BINF || (uint64_t)r.b >= Q.next_wrap) {
        if (r.b == BINF && Q.ovf == NIL) { status = EDMD_ERR_BUDGET; break; }
        while (Q.k < Q.next_wrap) { Q.P += B.dtP; Q.k++; }
        if constexpr (PAIR) pair_flush(as, lane);
        Q = do_wrap(S, Q, G);
        if constexpr (PAIR) r = S.tree[root];
        if (Q.ovf == OVF_CORRUPT) { Q.ovf = NIL; status = EDMD_ERR_BUDGET; break; }
        if (++guard > (1 << 20)) { status = EDMD_ERR_BUDGET; break; }
        continue;
      }
      break;
    }
    if (status != EDMD_OK) break;
    const int e = r.idx;
    const Ev E = S.ev[e];
    // the calendar's walk to the event: by the second warp if that runs it
    if (!PAIR || e >= 2 * N || le_i(A.t_stop, E.t))
      while (Q.k < (uint64_t)r.b) { Q.P += B.dtP; Q.k++; }
    if (le_i(A.t_stop, E.t)) { stop = EDMD_STOP_TIME; break; }
    t = E.t;
    nev++;
    if (e >= 2 * N) {
      *special = e;
      end = END_SPECIAL;
      break;
    }
    {
      const bool coll = e >= N;
      const int i = coll ? e - N : e, j = coll ? E.j : i;
      if constexpr (PAIR) {
        if (lane == 0) {
          as->i = i; as->j = E.j; as->coll = coll; as->grow = GROW; as->ca = E.ca; as->t = t;
          as->P = Q.P; as->k = Q.k; as->b = r.b;
        }
        if (Q.k < (uint64_t)r.b) Q.k = r.b;
        pair_barrier();                                                // A
      }
      const int my = odd ? j : i;
      Disk* const D = S.d + my;
      Own own;
      own.p = *axis_pos(D, ydim); own.v = *axis_vel(D, ydim); own.rad = D->rad;
      own.c = (ydim ? S.cy : S.cx)[my];
      own.vr = GROW ? S.vr[my] : 0.0;
      const double m = D->m;
      const uint32_t hits = D->coll;
      // events replaced by this one's, beside the popped one: the crossings of
      // both disks and the partner's collision, or a crossing disk's collision
      const int old = coll ? (lane == 0 ? i : lane == 1 ? j : lane == 3 ? N + j : -1) : (lane == 2 ? N + i : -1);
      const uint32_t old_st = old >= 0 ? S.ev[old].st : ST_NONE;
      {
        // freeFlyNormal / Grow (src/EDMD.c:4954 / 4992) of the lane's coordinate
        const double L = ydim ? B.Ly : B.Lx;
        const double dt = t - D->tl;
        own.p += dt * own.v;
        if (is_neg(own.p)) own.p += L;
        else if (ge_pos(own.p, L)) own.p -= L;
        if (GROW) own.rad += dt * own.vr;
      }
      const bool stale = coll && E.ca != G.shfl(hits, 1);
      const bool two = coll && !stale;       // a second disk changes
      // the state is stored only after the second warp has read it
      auto outcome = [&]() {
        if constexpr (PAIR) {
          if (lane < 4) { as->p[lane] = own.p; as->v[lane] = own.v; }
          pair_barrier();                                              // B
        }
      };
      if (two) {
        // ---------------- collision (doTheCollisionNormal 3542 / Grow 3465)
        if ((A.flags & EDMD_F_TRACE) && S.trace && (int64_t)(ntrace0 + ncoll) < S.trace_cap) {
          const int ci = G.shfl(own.c, 2) * B.Nxc + G.shfl(own.c, 0), cj = G.shfl(own.c, 3) * B.Nxc + G.shfl(own.c, 1);
          if (lane == 0) {
            edmd_collision* tr = (edmd_collision*)S.trace + (ntrace0 + ncoll);
            tr->i = i; tr->j = j; tr->cell_i = ci; tr->cell_j = cj; tr->t = t;
          }
        }
        ncoll++;
        if (!GROW || !(A.flags & EDMD_F_COUNT_NORMAL)) logged++;
        const Meet c = meet_lanes(B, G, own, m);
        const double d = c.d, dv = c.dv, mo = c.mo;
        const double msum = m + mo;
        const long long mk = __double_as_longlong(msum);
        if constexpr (!GROW) {   // elastic branch src/EDMD.c:3802-3827
          double inv;
          if (mk == sm->msum[0]) inv = sm->inv[0];
          else if (mk == sm->msum[1]) inv = sm->inv[1];
          else {
            inv = div_rn(1.0, msum) * onepr;
            G.sync();
            if (lane == 0) {
              sm->msum[1] = sm->msum[0]; sm->inv[1] = sm->inv[0];
              sm->msum[0] = mk; sm->inv[0] = inv;
            }
            G.sync();
          }
          double dx, dy;
          const double f = elastic_lanes<GW, ADD>(B, G, own, m, c, inv, ctl, &dx, &dy);
          if (A.flags & EDMD_F_LOG) {
            const double dvo = G.shfl_xor(dv, 2);
            if (S.log && (int64_t)nlog < S.log_cap && lane == 0) {
              edmd_log_entry* lg = (edmd_log_entry*)S.log + nlog;
              lg->i = i; lg->j = j; lg->t = t; lg->dx = dx; lg->dy = dy;
              lg->dvx = dv; lg->dvy = dvo; lg->f = f;
            }
            nlog++;
          }
        } else {       // growth rule src/EDMD.c:3479-3520, with its res = 1 and delta = 0
          const double dvr = own.vr + G.shfl_xor(own.vr, 1);
          double s2 = d * d;
          s2 += G.shfl_xor(s2, 2);
          const double dist = sqrt_rn(s2);
          const double dr = div_rn(d, dist);
          double pr = dr * dv;
          pr += G.shfl_xor(pr, 2);
          const double inv = mk == 0x4000000000000000ll ? 0.5 : div_rn(1.0, msum);
          const double collKernel = inv * 2.0 * (pr - dvr);
          // the rule's second term, 2 m inv delta r, is a zero of r's sign
          const double delta = 0;
          own.v += flip(collKernel * mo * dr - 2 * mo * inv * delta * dr, odd);
        }
        outcome();
        if (lane < 4) {
          *axis_pos(D, ydim) = own.p;
          *axis_vel(D, ydim) = own.v;
          if (!ydim) {
            D->tl = t;
            D->coll = hits + 1;
            if (GROW) D->rad = own.rad;
          }
        }
      } else if (stale) {
        outcome();
        if (lane == 0 || lane == 2) *axis_pos(D, ydim) = own.p;
        if (lane == 0) {
          D->tl = t;
          if (GROW) D->rad = own.rad;
        }
        nstale++;
      } else {
        // ---------------- cell crossing (doTheCrossing 2501)
        const int from = G.shfl(own.c, 2) * B.Nxc + G.shfl(own.c, 0);
        int wrap = 0;
        if (ydim == (E.j >= 3)) {
          const int n = ydim ? B.Nyc : B.Nxc;
          if (E.j & 1) { if (own.c - 1 == -1) { own.c = n - 1; wrap = -1; } else own.c -= 1; }
          else { if (own.c + 1 == n) { own.c = 0; wrap = 1; } else own.c += 1; }
        }
        const int to = G.shfl(own.c, 2) * B.Nxc + G.shfl(own.c, 0);
        outcome();
        if (lane == 0 || lane == 2) {
          *axis_pos(D, ydim) = own.p;
          (ydim ? S.cy : S.cx)[i] = own.c;
          if (wrap) (ydim ? S.crossY : S.crossX)[i] += wrap;
        }
        if (lane == 0) {
          const int pv = S.prv[i], nx = D->nxt;
          if (pv == NIL) S.head[from] = nx;
          else S.d[pv].nxt = nx;
          if (nx != NIL) S.prv[nx] = pv;
          const int h = S.head[to];
          S.prv[i] = NIL;
          D->nxt = h;
          D->tl = t;
          if (GROW) D->rad = own.rad;
          S.head[to] = i;
          if (h != NIL) S.prv[h] = i;
        }
      }
      // removeEventFromQueue (src/EDMD.c:2209) of the replaced events: every
      // slot is written again below, so only the overflow list needs work
      // (lane 0 alone touches its links)
      unsigned gone = G.ballot(!stale && old_st == ST_OVF);
      while (gone) {
        const int q = __ffs(gone) - 1;
        gone &= gone - 1;
        const int x = G.shfl(old, q);
        int first = Q.ovf;
        if (lane == 0) {
          const int p = S.op[x], n = S.on[x];
          if (p != NIL) S.on[p] = n;
          if (n != NIL) S.op[n] = p;
          if (p == NIL) first = n;
        }
        Q.ovf = G.shfl(first, 0);
      }
      // the next crossing and collision
      double tc = 0;
      int dir = 0;
      Next nx;
      if constexpr (PAIR) {
        if (two && lane < 4) {                  // the colliding disks as each other's candidates
          const int f = as->self[odd ? 0 : 1];
          if (f >= 0) {
            Flown& F = as->cand[f];
            F.p[ydim ? 1 : 0] = own.p; F.v[ydim ? 1 : 0] = own.v;
            if (!ydim) { F.rad = own.rad; F.coll = hits + 1; }
          }
        }
        G.sync();
        nx = predict2<GW, ADD, GROW, GW, true>(S, t, i, two ? j : -1, own, &npair, G, sm, &ovl, &oa, &ob, [](int) {}, [](int) { return 0; }, as);
        pair_barrier();                                                // C
        tc = as->tc[lane & 1];
        dir = as->dir[lane & 1];
        Q.P = as->Pb;
      } else {
        if (!stale) tc = next_crossing(B, G, own.c, own.p, own.v, &dir);
        G.sync();
        nx = predict2<GW, ADD, GROW, GW>(S, t, i, two ? j : -1, own, &npair, G, sm, &ovl, &oa, &ob, [](int) {}, [](int) { return 0; });
      }
      // addEventToQueue (src/EDMD.c:2144): lanes 0 and 1 take the crossings of
      // the two disks, lanes 2 and 3 their collisions; in that order they get
      // the insertion counters and join the overflow list
      const unsigned who = stale ? 4u : two ? 15u : 5u;
      const bool mine = lane < 4 && ((who >> lane) & 1u);
      Ev ev;
      ev.t = t + (ydim ? key_time(nx.key) : tc);
      ev.j = ydim ? nx.partner : dir;
      ev.ca = ydim ? nx.ca : 0;
      const int slot = (ydim ? N : 0) + my;
      const uint64_t C = Q.C + __popc(who & ((1u << lane) - 1u));
      const int place = mine ? sched_place(S, Q, ev.t) : 0;
      sched_key(Q, C, 2ull, place, ev);
      Q.C += __popc(who);
      unsigned over = G.ballot(mine && place == -2);
      while (over) {
        const int q = __ffs(over) - 1;
        over &= over - 1;
        const int x = G.shfl(slot, q);
        if (lane == 0) {
          S.on[x] = Q.ovf; S.op[x] = NIL;
          if (Q.ovf != NIL) S.op[Q.ovf] = x;
        }
        Q.ovf = x;
      }
      if (mine) S.ev[slot] = ev;
      else if (stale && lane == 0) ev = S.ev[slot];      // the crossing that stays
      // the leaves: the earlier of a disk's two events
      Node n = empty_node(slot);
      if (ev.st == ST_QUEUED) n = ev_node(ev, slot);
      {
        Node o;
        o.tk = G.shfl_xor(n.tk, 2); o.tie = G.shfl_xor(n.tie, 2);
        o.b = G.shfl_xor(n.b, 2); o.idx = G.shfl_xor(n.idx, 2);
        if (node_less(o, n)) n = o;
      }
      if constexpr (PAIR) {
        // the root: the changed leaves (lanes 0 and 1) and all others (lane 2)
        if (lane < 2) as->leaf[lane] = n;
        if (lane == 2) n = as->rest;
        if (lane > 2 || (lane == 1 && !two)) n = empty_node(0x7fffffff);
        top = shfl_node(n, grp_argmin(n, G), G);
      } else {
        path_update(S, i, two ? j : -1, shfl_node(n, 0, G), shfl_node(n, 1, G), G);
      }
    }
    if (ovl) { status = oa == OVL_CORRUPT ? EDMD_ERR_BUDGET : EDMD_ERR_OVERLAP; break; }
  }
  if constexpr (PAIR) pair_flush(as, lane);
  const double vir = G.shfl(ctl, virial_lane<GW>(lane & 3));
  if (lane < 4) st->collT[lane] = vir;
  if (lane == 0) {
    const uint64_t n = (uint64_t)(nev - nev0) - (end == END_SPECIAL ? 1 : 0);   // disk events
    const uint64_t cross = n - ncoll - nstale;
    st->t = t;
    queue_to(*st, Q);
    st->ncol += ncoll; st->ncol_total += ncoll; st->ntrace = ntrace0 + ncoll;
    st->ncross += cross; st->nstale += nstale;
    st->npair += npair; st->npred += 2 * ncoll + cross + nstale;
    st->nevents += (uint64_t)(nev - nev0);
    st->nlog = nlog;
    st->stop_reason = stop;
    st->status = status;
    if (ovl) { st->err_a = oa; st->err_b = ob; }
  }
  G.sync();
  return end;
}

// a special event e just popped, on the system's state in memory; false when
// the run ends with it
template <int GW, bool ADD>
__device__ __noinline__ bool serve_special(const SysDev& S, uint32_t flags, int e, Grp<GW> G, WarpSmem* sm) {
  const int lane = G.lane;
  const int N = S.B.N;
  SysState R = *S.st;
  const bool grow = R.grow != 0;
  int stop = 0, oa = -1, ob = -1;
  bool ovl = false;
  if (lane == 0) S.ev[e].st = ST_NONE;
  G.sync();
  if (e == 2 * N + SP_GROW) {
    do_growstop<GW, ADD>(S, R, G, sm, &ovl, &oa, &ob);
    if (flags & EDMD_F_STOP_AT_GROW) stop = EDMD_STOP_GROW;
  } else {
    double next;
    if (e == 2 * N + SP_SCREEN) {
      // ---------------- screenshot (takeAScreenshot 4657): free-fly everything
      for (int i = lane; i < N; i += GW) {
        Disk p = S.d[i];
        grow_fly(S, p, i, R.t, grow);
        S.d[i] = p;
      }
      G.sync();
      next = R.t + S.dtime;
      if (flags & EDMD_F_STOP_AT_SCREEN) stop = EDMD_STOP_SCREEN;
    } else {
      do_thermo(S, R, G);
      next = R.t + S.dtimeTh;
    }
    Queue Q = queue_of(R);
    schedule(S, Q, e, next, 0, 0, 2ull, G);
    queue_to(R, Q);
    leaf_update(S, e - N, G);
  }
  if (ovl) {
    R.status = oa == OVL_CORRUPT ? EDMD_ERR_BUDGET : EDMD_ERR_OVERLAP;
    R.err_a = oa; R.err_b = ob;
  }
  R.stop_reason = stop;
  G.sync();
  if (lane == 0) *S.st = R;
  G.sync();
  return !ovl && !stop;
}

// the event loop of one system, at most `share` events of it; true when the
// call is done with the system
template <int GW, bool ADD = true, bool PAIR = false>
__device__ bool run_system(const SysDev& S, const RunArgs& A, const Grp<GW>& G, WarpSmem* sm, RunProgress& pr,
                           int64_t share, Aside* as = nullptr) {
  if (S.st->status != EDMD_OK) return true;
  const int64_t share_end = A.max_events - pr.nev > share ? pr.nev + share : A.max_events;
  for (;;) {
    int special = 0, end;
    if (S.st->grow) end = run_events<GW, ADD, true, PAIR>(S, A, A.max_coll, G, sm, as, pr.logged, pr.nev, share_end, &special);
    else end = run_events<GW, ADD, false, PAIR>(S, A, A.max_coll, G, sm, as, pr.logged, pr.nev, share_end, &special);
    if (end == END_SHARE) return false;
    if (end != END_SPECIAL || !serve_special<GW, ADD>(S, A.flags, special, G, sm)) return true;
  }
}

// Events a system runs before it makes room for a waiting one.  Turns of 256 are
// ~5 ms and leave little of the launch's end to a part of the groups; measured
// against 1024 (ms): 3100 systems of 64-1024 disks, 257 / 400 / 1200 collisions
// 6.4 / 9.3 / 24.8 against 6.9 / 11.1 / 28.7; 4096 of 256-1024 disks 7.6 / 11.6 /
// 31.7 against 8.5 / 13.3 / 33.6; 16384 of 96 disks 24.1 / 36.8 / 111.3 against
// 25.2 / 38.7 / 111.0; for one unit of time 37.8, 45.2 and 19.3 against 37.9, 46.9
// and 19.7.  A call of at most 256 collisions takes turns of 1024, in which most
// systems end (1.7 events a collision at phi 0.55): 16384 of 96 disks, 150
// collisions 16.1 ms against 18.2 in turns of 256.
__device__ __forceinline__ int64_t share_of(int64_t max_coll) { return max_coll <= 256 ? 1024 : 256; }

// The place whose system a lane group runs next, -1 when there is none.  A
// group leaves its own place `mine` (-1: its system is done) in the waiting slot
// that the ticket names and takes what waited there; slots are only exchanged
// whole, so no group ever waits for another.  ticket[1] counts the waiting
// places and is never below their number: raised before a place goes into a
// slot, lowered after one came out.  The last group to finish looks through
// slots that no one fills any more, so no place is left behind.
template <int GW>
__device__ __noinline__ int next_place(const RunArgs& A, int mine, Grp<GW> G) {
  const unsigned nw = (unsigned)A.nwait;
  int got = -1;
  unsigned at = 0;
  if (G.lane == 0) {
    __threadfence();                                  // the system's state before its place
    at = atomicAdd(&A.ticket[0], 1u) % nw;
    if (mine >= 0) {
      atomicAdd(&A.ticket[1], 1u);
      got = atomicExch(&A.waiting[at], mine);
      if (got < 0) got = atomicExch(&A.waiting[at], -1);   // a hole: back out (or take what came in since)
      if (got >= 0) atomicAdd(&A.ticket[1], ~0u);
    }
  }
  got = G.shfl(got, 0);
  at = (unsigned)G.shfl((int)at, 0);
  // nothing yet (this system is done, or another group took it from the hole):
  // any waiting place from the ticket's slot on
  for (unsigned k = 0; k < nw && got < 0; k += GW) {
    int left = 0;
    if (G.lane == 0) left = (int)atomicAdd(&A.ticket[1], 0u);
    if (G.shfl(left, 0) <= 0) break;
    const unsigned q = (at + k + G.lane) % nw;
    unsigned here = G.ballot(k + G.lane < nw && *(volatile int32_t*)&A.waiting[q] >= 0);
    while (here && got < 0) {
      const int l = __ffs(here) - 1;
      here &= here - 1;
      int v = -1;
      if (G.lane == l) {
        v = atomicExch(&A.waiting[q], -1);
        if (v >= 0) atomicAdd(&A.ticket[1], ~0u);
      }
      got = G.shfl(v, l);
    }
  }
  __threadfence();                                    // and the place before the system's state
  G.sync();
  return got;
}

// Lane groups (GW lanes, one system each), all resident.  With more systems
// than groups the others wait, and after every share of events a group changes
// its system for a waiting one: the systems advance together and the launch
// ends with all groups busy.  Whole systems, longest first by the last call's
// times, left the last ones to a nearly empty GPU: 4096 systems of 256-1024
// disks 9.5e7 coll/s, 1.2e8 in turns.
// MINB: blocks of four warps per SM the registers allow for (run_shape).
template <int GW, bool ADD, int MINB>
__global__ void __launch_bounds__(32 * WARPS_PER_BLOCK, MINB)
k_run(const SysDev* __restrict__ sys, RunArgs A) {
  __shared__ WarpSmem smem[WARPS_PER_BLOCK * (32 / GW)];
  const Grp<GW> G(threadIdx.x);
  WarpSmem* sm = &smem[threadIdx.x / GW];
  int p = (int)((blockIdx.x * blockDim.x + threadIdx.x) / GW);
  if (p >= A.nrun) return;
  while (p >= 0) {
    const int s = A.order ? A.order[p] : p;
    RunProgress pr{0, 0};
    if (A.nwait) pr = A.progress[p];
    const bool done = run_system<GW, ADD>(sys[s], A, G, sm, pr, A.nwait ? share_of(A.max_coll) : A.max_events);
    if (!A.nwait) break;
    if (G.lane == 0) A.progress[p] = pr;
    G.sync();
    p = next_place(A, done ? -1 : p, G);
  }
}

// Two warps per system, one system per block.  An event is one chain of
// dependent instructions (64 cycles for each FP64 one, 106 for a load that hits
// L1), so a context of few systems leaves the GPU idle whatever its lanes do;
// run_aside takes ~40 % of the chain off it: of ~10.5k cycles per event the
// neighbour lists and candidates were 2.4k, the crossings 1.0k, the tree 1.4k to
// 2.0k and the calendar 0.2k.  Measured, one warp / two (600 collisions a
// system, ms): 1 system of 1000 disks 6.2 / 4.9, 304 of 128-512 7.1 / 5.7, 912
// 8.2 / 6.9, 1064 of 64-1024 8.9 / 7.4, 1216 8.4 / 7.5; with registers for 10
// blocks per SM 1520 of 128-512 9.1 / 8.7 but 304 6.0, and 1824 10.1 / 10.1.
constexpr int PAIR_PER_SM = 8;
template <bool ADD>
__global__ void __launch_bounds__(64, PAIR_PER_SM) k_run_pair(const SysDev* __restrict__ sys, RunArgs A) {
  __shared__ WarpSmem smem;
  __shared__ Aside as;
  const Grp<32> G(threadIdx.x);
  const int p = blockIdx.x;
  if (p >= A.nrun) return;                    // both warps
  const SysDev& S = sys[A.order ? A.order[p] : p];
  if (threadIdx.x < 32) {
    RunProgress pr{0, 0};
    run_system<32, ADD, true>(S, A, G, &smem, pr, A.max_events, &as);
    if (G.lane == 0) as.i = ASIDE_END;
    pair_barrier();                           // A, the last
  } else {
    run_aside(S, G, &as);
  }
}

__global__ void k_waiting(RunArgs A) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < A.nwait) A.waiting[k] = A.nrun + k;
  if (k < A.nrun + A.nwait) A.progress[k] = RunProgress{0, 0};
  if (k == 0) { A.ticket[0] = 0; A.ticket[1] = (unsigned)A.nwait; }
}

// How nsys systems are run with gw lanes each: kernel, warps and systems of a
// block.  With 32 lanes up to eight systems per SM get two warps each
// (k_run_pair; `pair`: unless they would not all be resident, or one has fewer
// than three cells along an axis: its 3x3 scans meet a colliding partner more
// than once, and the second warp's list holds one place for it, while the
// one-warp loop reads every candidate after the collision).  One warp each,
// measured (203 disks alone / 192 growth starts / 1824 < 2600 mixed systems,
// ms; every build has the same event loop):
//   3 blocks per SM, 168 registers: 1.41 / 15.2 / 36
//   4 blocks, 128 registers:        1.45 / 15.5 / 40.5 (2432 warps, a second wave)
//   5 blocks, 96 registers:         1.50 / 16.4 / 30.2 (3040 warps)
//   6 blocks, 80 registers:         1.58 / 17.6 / 32.2
// so systems that all find a warp at three blocks per SM run there (8 bytes of
// spill stores), and larger batches at five (476 bytes).
bool few_cells(const Box& B) { return B.Nxc < 3 || B.Nyc < 3; }
using RunKernel = void (*)(const SysDev*, RunArgs);
struct RunShape { RunKernel kernel; int warps, systems; };   // a block's warps and systems
RunShape run_shape(int gw, bool additive, int nsys, int nsm, bool pair) {
  const int W = WARPS_PER_BLOCK;
  if (gw == 4) return {k_run<4, true, 4>, W, W * 8};
  if (gw == 8) return {k_run<8, true, 4>, W, W * 4};
  if (gw == 16) return {k_run<16, true, 4>, W, W * 2};
  if (pair && nsys <= PAIR_PER_SM * nsm) return {additive ? k_run_pair<true> : k_run_pair<false>, 2, 1};
  if (nsys <= 3 * W * nsm) return {additive ? k_run<32, true, 3> : k_run<32, false, 3>, W, W};
  return {additive ? k_run<32, true, 5> : k_run<32, false, 5>, W, W};
}

// ---------------------------------------------------------------- shared-memory kernel

// where one system's engine state sits in a block's dynamic shared memory:
// disk records, event slots, tree, cell coordinates and links, cell heads and
// overflow links; the scalar state, growth rates, trace, log and thermo rows
// stay in global memory
struct SmemLayout {
  size_t d, ev, tree, cx, cy, prv, crossX, crossY, head, on, op, total;
};

__host__ __device__ inline SmemLayout smem_layout(const SysDev& S) {
  const size_t N = (size_t)S.B.N, E = 2 * N + NSPECIAL, C = (size_t)S.B.Nxc * S.B.Nyc;
  size_t nodes = 0;
  for (int h = 0; h < S.nlev; h++) nodes += (size_t)S.lev_cnt[h];
  SmemLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t r = o; o += (bytes + 63) & ~(size_t)63; return r; };
  L.d = take(N * sizeof(Disk));
  L.ev = take(E * sizeof(Ev));
  L.tree = take(nodes * sizeof(Node));
  L.cx = take(N * 4); L.cy = take(N * 4); L.prv = take(N * 4);
  L.crossX = take(N * 4); L.crossY = take(N * 4);
  L.head = take(C * 4);
  L.on = take(E * 4); L.op = take(E * 4);
  L.total = o;
  return L;
}

// words of one array between global and shared memory, over the warp
__device__ __forceinline__ void warp_copy(void* dst, const void* src, size_t bytes, int lane) {
  uint32_t* d = (uint32_t*)dst;
  const uint32_t* s = (const uint32_t*)src;
  for (size_t k = lane; k < bytes / 4; k += 32) d[k] = s[k];
}

// One warp per block: each system of `list` is copied into the block's
// shared memory, run by the same event loop as k_run through a descriptor
// whose arrays point there (every access in it is a generic-address access),
// and copied back.  Dependent accesses then cost shared-memory latency
// instead of L2/HBM latency, at the price of one resident system per ~100 KB.
__global__ void __launch_bounds__(32) k_run_smem(const SysDev* __restrict__ sys, RunArgs A,
                                                 const int32_t* __restrict__ list, int nlist,
                                                 int32_t* __restrict__ work) {
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ WarpSmem wsm;
  const Grp<32> G(threadIdx.x);
  const int lane = G.lane;
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(work, 1);
    it = G.shfl(it, 0);
    if (it >= nlist) break;
    const int s = list[it];
    const SysDev& S = sys[s];
    const SmemLayout Y = smem_layout(S);
    const size_t N = (size_t)S.B.N, E = 2 * N + NSPECIAL, C = (size_t)S.B.Nxc * S.B.Nyc;
    size_t nodes = 0;
    for (int h = 0; h < S.nlev; h++) nodes += (size_t)S.lev_cnt[h];
    SysDev L = S;
    L.d = (Disk*)(dyn + Y.d); L.ev = (Ev*)(dyn + Y.ev); L.tree = (Node*)(dyn + Y.tree);
    L.cx = (int32_t*)(dyn + Y.cx); L.cy = (int32_t*)(dyn + Y.cy); L.prv = (int32_t*)(dyn + Y.prv);
    L.crossX = (int32_t*)(dyn + Y.crossX); L.crossY = (int32_t*)(dyn + Y.crossY);
    L.head = (int32_t*)(dyn + Y.head); L.on = (int32_t*)(dyn + Y.on); L.op = (int32_t*)(dyn + Y.op);
    warp_copy(L.d, S.d, N * sizeof(Disk), lane);
    warp_copy(L.ev, S.ev, E * sizeof(Ev), lane);
    warp_copy(L.tree, S.tree, nodes * sizeof(Node), lane);
    warp_copy(L.cx, S.cx, N * 4, lane); warp_copy(L.cy, S.cy, N * 4, lane);
    warp_copy(L.prv, S.prv, N * 4, lane);
    warp_copy(L.crossX, S.crossX, N * 4, lane); warp_copy(L.crossY, S.crossY, N * 4, lane);
    warp_copy(L.head, S.head, C * 4, lane);
    warp_copy(L.on, S.on, E * 4, lane); warp_copy(L.op, S.op, E * 4, lane);
    G.sync();
    RunProgress pr{0, 0};
    run_system(L, A, G, &wsm, pr, A.max_events);
    G.sync();
    warp_copy(S.d, L.d, N * sizeof(Disk), lane);
    warp_copy(S.ev, L.ev, E * sizeof(Ev), lane);
    warp_copy(S.tree, L.tree, nodes * sizeof(Node), lane);
    warp_copy(S.cx, L.cx, N * 4, lane); warp_copy(S.cy, L.cy, N * 4, lane);
    warp_copy(S.prv, L.prv, N * 4, lane);
    warp_copy(S.crossX, L.crossX, N * 4, lane); warp_copy(S.crossY, L.crossY, N * 4, lane);
    warp_copy(S.head, L.head, C * 4, lane);
    warp_copy(S.on, L.on, E * 4, lane); warp_copy(S.op, L.op, E * 4, lane);
    G.sync();
  }
}

// ---------------------------------------------------------------- init kernels

// initial predictions of eventListInit (src/EDMD.c:2007-2012): all disks are
// current at t = 0 and the calendar sits at bucket 0, so every key is known
// without serialising: the k-th scheduled event has counter k.
// grid.y = system, grid.x covers the disks of the largest system + 1.
__global__ void k_init_events(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const Box& B = S.B;
  const int N = B.N;
  const bool grow = S.st->grow != 0;
  const int nspec = grow ? 3 : 2;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  auto key = [&](Ev& ev, double T, uint64_t C) {
    double dt = T - 0.0;
    if (dt < B.dtP) { ev.b = 0; ev.tie = (2ull << 62) | C; ev.st = ST_QUEUED; }
    else if (dt >= B.dtPN) { ev.b = BINF; ev.tie = C; ev.st = ST_OVF; }
    else { int d = (int)(dt / B.dtP); ev.b = (uint32_t)d; ev.tie = (1ull << 62) | (TIE_MAX - C); ev.st = ST_QUEUED; }
  };
  if (i < N) {
    Disk A = S.d[i];
    int dir;
    Ev ec; ec.t = crossing_time(B, A, S.cx[i], S.cy[i], 0.0, &dir); ec.j = dir; ec.ca = 0;
    key(ec, ec.t, (uint64_t)nspec + 2ull * i);
    S.ev[i] = ec;
    double bd = grow ? 10000000 : NEVER;
    int bp = 0;
    bool ov = false;
    int ovp = -1;                     // first partner found overlapping
    int X = S.cx[i], Y = S.cy[i];
    uint64_t np = 0;
    for (int q = 0; q < 9; q++) {
      int cell = pbc_cy(B, Y + q / 3 - 1) * B.Nxc + pbc_cx(B, X + q % 3 - 1);
      for (int p = S.head[cell]; p != NIL; p = S.d[p].nxt) {
        if (p == i) continue;
        Disk P = S.d[p];
        bool o2 = false;
        double d = grow ? coll_time_grow(B, A, S.vr[i], P, S.vr[p], 0.0, &o2)
                        : coll_time_normal(B, A, P, 0.0, &o2);
        if (o2 && ovp < 0) ovp = p;
        ov |= o2;
        np++;
        if (bd > d) { bd = d; bp = p; }
      }
    }
    Ev el; el.t = 0.0 + bd; el.j = bp; el.ca = 0;
    key(el, el.t, (uint64_t)nspec + 2ull * i + 1);
    S.ev[N + i] = el;
    atomicAdd((unsigned long long*)&S.st->npair, (unsigned long long)np);
    // one thread (the first to claim the status) names the pair
    if (ov && atomicCAS(&S.st->status, EDMD_OK, EDMD_ERR_OVERLAP) == EDMD_OK) {
      S.st->err_a = i;
      S.st->err_b = ovp;
    }
  } else if (i == N) {
    // thermo, [growth stop], screenshot in eventListInit order
    Ev e; e.j = 0; e.ca = 0;
    e.t = S.st->lastThermo;   // holds first_thermo + 1e-9 on entry
    key(e, e.t, 0);
    S.ev[2 * N + SP_THERMO] = e;
    uint64_t C = 1;
    Ev g; g.j = 0; g.ca = 0; g.t = S.st->collT[0];  // holds t_growstop on entry
    if (grow) { key(g, g.t, C); C++; } else { g.st = ST_NONE; g.b = BINF; g.tie = 0; }
    S.ev[2 * N + SP_GROW] = g;
    Ev sc; sc.j = 0; sc.ca = 0; sc.t = S.st->collT[1];  // holds first_screen on entry
    key(sc, sc.t, C);
    S.ev[2 * N + SP_SCREEN] = sc;
  }
}

// link the initial overflow bucket in LIFO order and finish the scalar state.
// The reference pushes the initial events in the order
// thermo, [growth stop], screenshot, then crossing i and collision i for
// i = 0..N-1 (eventListInit, src/EDMD.c:1935-2019); an overflow event's `on`
// link is the previous overflow event in that order and `op` the next one, so
// both follow from a running maximum over the push positions.
__device__ __forceinline__ int init_slot(int p, int N, bool grow) {
  const int nspec = grow ? 3 : 2;
  if (p < nspec) {
    if (p == 0) return 2 * N + SP_THERMO;
    if (grow && p == 1) return 2 * N + SP_GROW;
    return 2 * N + SP_SCREEN;
  }
  const int k = p - nspec;
  return (k & 1) ? N + (k >> 1) : (k >> 1);
}

// The running maximum goes chunk by chunk: k_init_last leaves each chunk's
// last overflow position in the tree's array (built after it), k_init_finish
// takes the nearest one before its chunk.  One block walked a whole system
// before: 4x10^6 disks took 31,000 block steps.
constexpr int INIT_CHUNK = 4096;

__global__ void __launch_bounds__(256) k_init_last(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const int N = S.B.N;
  const bool grow = S.st->grow != 0;
  const int P = (grow ? 3 : 2) + 2 * N, p0 = blockIdx.x * INIT_CHUNK;
  if (p0 >= P) return;
  int last = -1;
  for (int p = p0 + threadIdx.x; p < min(P, p0 + INIT_CHUNK); p += 256)
    if (S.ev[init_slot(p, N, grow)].st == ST_OVF) last = p;
  __shared__ int m[8];
  last = __reduce_max_sync(FULL, last);
  if ((threadIdx.x & 31) == 0) m[threadIdx.x >> 5] = last;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) last = max(last, m[w]);
    ((int*)S.tree)[blockIdx.x] = last;
  }
}

__global__ void __launch_bounds__(256) k_init_finish(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const int N = S.B.N;
  const bool grow = S.st->grow != 0;
  const int P = (grow ? 3 : 2) + 2 * N, p0 = blockIdx.x * INIT_CHUNK;
  if (p0 >= P) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int* last_of = (const int*)S.tree;
  __shared__ int wmax[8];
  __shared__ int carry;
  // the last overflow position before this chunk
  if (w == 0) {
    int before = -1;
    for (int c = blockIdx.x - 1; c >= 0 && before < 0; c -= 32) {
      const int l = c - lane >= 0 ? last_of[c - lane] : -1;
      before = __reduce_max_sync(FULL, l);
    }
    if (lane == 0) carry = before;
  }
  __syncthreads();
  for (int base = p0; base < min(P, p0 + INIT_CHUNK); base += blockDim.x) {
    const int p = base + threadIdx.x;
    const int e = p < P ? init_slot(p, N, grow) : -1;
    const bool ovf = e >= 0 && S.ev[e].st == ST_OVF;
    // exclusive running maximum of the overflow positions: the previous one
    int v = ovf ? p : -1;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(FULL, incl, o);
      if (lane >= o && u > incl) incl = u;
    }
    if (lane == 31) wmax[w] = incl;
    __syncthreads();
    int before = carry;
    for (int k = 0; k < w; k++) before = wmax[k] > before ? wmax[k] : before;
    int excl = __shfl_up_sync(FULL, incl, 1);
    if (lane == 0) excl = -1;
    const int prev = excl > before ? excl : before;
    if (ovf) {
      // every overflow event but the last gets its `op` from its successor
      const int pe = prev >= 0 ? init_slot(prev, N, grow) : NIL;
      S.on[e] = pe;
      if (pe != NIL) S.op[pe] = e;
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) {
      const int last = incl > before ? incl : before;
      carry = last;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && p0 + INIT_CHUNK >= P) {         // the system's last chunk
    SysState& R = *S.st;
    R.ovf = carry >= 0 ? init_slot(carry, N, grow) : NIL;
    if (R.ovf != NIL) S.op[R.ovf] = NIL;
    R.C = (uint64_t)(grow ? 3 : 2) + 2ull * N;
    R.npred = (uint64_t)N;
    R.lastThermo = 0;
    R.collT[0] = R.collT[1] = 0;
  }
}

// levels 0, 1 and 2 of the tree, 1024 leaves per block: a warp's leaves are
// one parent's children, a block's parents another's
__global__ void __launch_bounds__(1024) k_tree_leaves(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const int l = blockIdx.x * 1024 + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.x * 1024 >= S.L) return;
  const Grp<32> G(threadIdx.x);
  __shared__ Node up[32];
  Node n = empty_node(0x7fffffff);
  if (l < S.L) S.tree[l] = n = leaf_node(S, l);
  const int src = grp_argmin(n, G);
  if (lane == src) {
    up[w] = n;
    if ((l >> 5) < S.lev_cnt[1]) S.tree[S.lev_off[1] + (l >> 5)] = n;     // a system has at least two leaves
  }
  if (S.nlev < 3) return;
  __syncthreads();
  if (w == 0) {
    const Node m = up[lane];
    if (lane == grp_argmin(m, G)) S.tree[S.lev_off[2] + blockIdx.x] = m;
  }
}

// the levels above, for systems of more than 1024 leaves: one block per
// system, a warp per parent, level by level
__global__ void __launch_bounds__(256) k_tree_build(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.x];
  const Grp<32> G(threadIdx.x);
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int h = 3; h < S.nlev; h++) {
    for (int par = w; par < S.lev_cnt[h]; par += nw) {
      const Node none = empty_node(0x7fffffff);
      const Node c = child_node(S, h, par, -1, none, -1, none, G);
      if (G.lane == grp_argmin(c, G)) S.tree[S.lev_off[h] + par] = c;
    }
    __syncthreads();
  }
}

// event set, overflow list and (warp engine) tree of nsys systems of at most
// maxN disks whose disks and cell lists are in place
cudaError_t init_queues(const SysDev* sys, int nsys, int maxN, bool tree, cudaStream_t st) {
  k_init_events<<<dim3((maxN + 1 + 127) / 128, nsys), 128, 0, st>>>(sys);
  const dim3 g((3 + 2 * maxN + INIT_CHUNK - 1) / INIT_CHUNK, nsys);
  k_init_last<<<g, 256, 0, st>>>(sys);
  k_init_finish<<<g, 256, 0, st>>>(sys);
  if (tree) {
    k_tree_leaves<<<dim3((maxN + NSPECIAL + 1023) / 1024, nsys), 1024, 0, st>>>(sys);
    if (maxN + NSPECIAL > 1024) k_tree_build<<<nsys, 256, 0, st>>>(sys);
  }
  return cudaGetLastError();
}

// freeFly of every disk to its system's time: blocks of 256 disks
__global__ void __launch_bounds__(256) k_sync(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= S.B.N) return;
  Disk p = S.d[i];
  grow_fly(S, p, i, S.st->t, S.st->grow != 0);
  S.d[i] = p;
}

// ---- a system's disks and cell lists from host arrays

// a disk the engine cannot take: its position (after the periodic wrap of a
// restart), then its radius
__host__ __device__ __forceinline__ void wrap_restart(double& x, double& y, double Lx, double Ly) {
  if (x < 0) x += Lx; else if (x >= Lx) x -= Lx;     // PBCpostX/Y (src/EDMD.c:1405-1406)
  if (y < 0) y += Ly; else if (y >= Ly) y -= Ly;
}
// 0: good, 1: position outside the box, 2: radius not zero or normal positive
__host__ __device__ __forceinline__ int bad_disk(double x, double y, double rad, double Lx, double Ly, bool restart) {
  if (restart) wrap_restart(x, y, Lx, Ly);
  if (!(x >= 0 && x < Lx && y >= 0 && y < Ly)) return 1;
  return radius_ok(rad) ? 0 : 2;
}

// SoA staging arrays (x y vx vy rad m of all disks, `total` each) of the
// systems; doff[s]: first disk of system s
__global__ void k_check(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff,
                        const double* __restrict__ in, int64_t total, bool restart, unsigned long long* bad) {
  const SysDev& S = sys[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.B.N) return;
  const int64_t g = doff[blockIdx.y] + i;
  const int b = bad_disk(in[g], in[total + g], in[4 * total + g], S.B.Lx, S.B.Ly, restart);
  if (b) atomicMin(bad, 2ull * (unsigned long long)g + (unsigned long long)(b - 1));
}

// records and cells (src/EDMD.c:1906 cellListInit); each disk also joins a
// chain of its cell, in any order, through the overflow links (not yet in use)
__global__ void k_stage(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff,
                        const double* __restrict__ in, int64_t total, bool restart) {
  const SysDev& S = sys[blockIdx.y];
  const Box& B = S.B;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B.N) return;
  const int64_t g = doff[blockIdx.y] + i;
  Disk q;
  q.x = in[g]; q.y = in[total + g]; q.vx = in[2 * total + g]; q.vy = in[3 * total + g];
  q.rad = in[4 * total + g]; q.m = in[5 * total + g];
  if (restart) wrap_restart(q.x, q.y, B.Lx, B.Ly);
  q.tl = 0; q.nxt = NIL; q.coll = 0;
  int X = (int)(q.x * B.cxf), Y = (int)(q.y * B.cyf);
  if (X >= B.Nxc) X = B.Nxc - 1;
  if (Y >= B.Nyc) Y = B.Nyc - 1;
  S.d[i] = q;
  S.cx[i] = X; S.cy[i] = Y;
  S.crossX[i] = 0; S.crossY[i] = 0;
  S.on[i] = atomicExch(&S.head[Y * B.Nxc + X], i);
}

// the reference pushes disks onto their cells' lists in index order (addToCell
// src/EDMD.c:2053, push-front), so a list runs from the largest index down:
// each disk finds its neighbours in that order on its cell's chain
__global__ void k_links(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.B.N) return;
  int below = NIL, above = NIL;
  for (int j = S.head[S.cy[i] * S.B.Nxc + S.cx[i]]; j != NIL; j = S.on[j]) {
    if (j < i && j > below) below = j;
    if (j > i && (above == NIL || j < above)) above = j;
  }
  S.d[i].nxt = below;
  S.prv[i] = above;
}

__global__ void k_heads(const SysDev* __restrict__ sys) {
  const SysDev& S = sys[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < S.B.N && S.prv[i] == NIL) S.head[S.cy[i] * S.B.Nxc + S.cx[i]] = i;
}

// disk records of every system -> concatenated SoA staging (x y vx vy rad m)
__global__ void k_gather(const Disk* __restrict__ d, int64_t total, double* __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  Disk p = d[i];
  out[i] = p.x; out[total + i] = p.y; out[2 * total + i] = p.vx;
  out[3 * total + i] = p.vy; out[4 * total + i] = p.rad; out[5 * total + i] = p.m;
}

}  // namespace

// ==================================================================== C ABI

#include "edmd_ctx.h"

static int g_engine = EDMD_ENGINE_AUTO;
static int g_lane_threads = 32;
static int g_group = 32;                        // warp engine: lanes per system

extern "C" int edmd_set_engine(int32_t kind) {
  if (kind < EDMD_ENGINE_AUTO || kind > EDMD_ENGINE_LANE) return EDMD_ERR_ARG;
  g_engine = kind;
  return EDMD_OK;
}

extern "C" int edmd_set_lane_threads(int32_t threads_per_block) {
  if (threads_per_block < 1 || threads_per_block > 1024) return EDMD_ERR_ARG;
  g_lane_threads = threads_per_block;
  return EDMD_OK;
}

extern "C" int edmd_set_warp_group(int32_t lanes) {
  if (lanes != 4 && lanes != 8 && lanes != 16 && lanes != 32) return EDMD_ERR_ARG;
  g_group = lanes;
  return EDMD_OK;
}

extern "C" int edmd_device_info(char* name, int32_t cap, int32_t* sm_count) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) return EDMD_ERR_NODEV;
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, 0) != cudaSuccess) return EDMD_ERR_CUDA;
  if (name && cap > 0) { strncpy(name, p.name, cap - 1); name[cap - 1] = 0; }
  if (sm_count) *sm_count = p.multiProcessorCount;
  return EDMD_OK;
}



constexpr int64_t PIN_BYTES = (int64_t)4 << 20;      // one staging buffer
// Smaller lists are copied directly; below PIN_THREADS the calling thread moves
// the pieces itself, since starting threads costs ~0.4 ms.  10^5 disks (4.8 MB)
// back: 0.2 ms direct into arrays the device has used before, 3.2 ms into
// others (a program that takes new arrays every time alternates); staged 0.4 ms.
constexpr int64_t PIN_LEAST = (int64_t)1 << 20, PIN_THREADS = (int64_t)16 << 20;

cudaError_t host_copies(edmd_ctx* ctx, const std::vector<HostCopy>& list, bool to_device) {
  const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  int64_t total = 0;
  for (const HostCopy& c : list) total += c.bytes;
  // pieces of at most one buffer; page-locked arrays directly
  std::vector<HostCopy> pieces;
  cudaError_t e = cudaSuccess;
  for (const HostCopy& c : list) {
    cudaPointerAttributes at;
    const bool pageable = total >= PIN_LEAST && cudaPointerGetAttributes(&at, c.host) == cudaSuccess &&
                          at.type == cudaMemoryTypeUnregistered;
    if (!pageable) {
      e = to_device ? cudaMemcpyAsync(c.dev, c.host, c.bytes, kind, ctx->stream)
                    : cudaMemcpyAsync(c.host, c.dev, c.bytes, kind, ctx->stream);
      if (e != cudaSuccess) return e;
      continue;
    }
    for (int64_t o = 0; o < c.bytes; o += PIN_BYTES)
      pieces.push_back({(char*)c.host + o, (char*)c.dev + o, std::min(PIN_BYTES, c.bytes - o)});
  }
  if (pieces.empty()) return cudaStreamSynchronize(ctx->stream);
  if (!ctx->pin) {
    e = cudaMallocHost((void**)&ctx->pin, 2 * PIN_BYTES);
    if (e != cudaSuccess) {                          // no page-locked memory left: copy directly
      ctx->pin = nullptr;
      cudaGetLastError();
      e = cudaSuccess;
      for (const HostCopy& c : pieces)
        if (e == cudaSuccess)
          e = to_device ? cudaMemcpyAsync(c.dev, c.host, c.bytes, kind, ctx->stream)
                        : cudaMemcpyAsync(c.host, c.dev, c.bytes, kind, ctx->stream);
      const cudaError_t es = cudaStreamSynchronize(ctx->stream);
      return e != cudaSuccess ? e : es;
    }
  }
  for (cudaEvent_t& ev : ctx->pin_ev)
    if (e == cudaSuccess && !ev) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  if (e != cudaSuccess) return e;
  const int n = (int)pieces.size();
  // host threads move slices of piece after piece as `open` lets them; `moved`
  // counts the slices done
  std::atomic<int> open{0}, quit{0};
  std::atomic<int64_t> moved{0};
  auto slice = [&](int p, int k, int of) {
    const int64_t lo = pieces[p].bytes * k / of, hi = pieces[p].bytes * (k + 1) / of;
    char* pin = ctx->pin + (p & 1) * PIN_BYTES;
    if (to_device) memcpy(pin + lo, (char*)pieces[p].host + lo, hi - lo);
    else memcpy((char*)pieces[p].host + lo, pin + lo, hi - lo);
  };
  std::vector<std::thread> pool;
  const int want = total < PIN_THREADS ? 0 : host_threads(total, PIN_THREADS) / 2;
  std::atomic<int> workers{0};                       // fixed before the first piece opens
  for (int k = 0; k < want; k++) {
    try {
      pool.emplace_back([&, k] {
        for (int p = 0; p < n; p++) {
          while (open.load(std::memory_order_acquire) <= p)
            if (quit.load()) return;
            else std::this_thread::yield();
          slice(p, k, workers.load());
          moved.fetch_add(1, std::memory_order_release);
        }
      });
    } catch (...) {
      break;
    }
  }
  const int nw = (int)pool.size();
  workers = nw;
  auto move = [&](int p) {                           // piece p between its buffer and the host array
    if (!nw) { slice(p, 0, 1); return; }
    open.store(p + 1, std::memory_order_release);
    while (moved.load(std::memory_order_acquire) < (int64_t)nw * (p + 1)) std::this_thread::yield();
  };
  for (int p = 0; p <= n && e == cudaSuccess; p++) {
    if (to_device) {
      if (p == n) break;
      if (p >= 2) e = cudaEventSynchronize(ctx->pin_ev[p & 1]);          // its buffer is free again
      if (e != cudaSuccess) break;
      move(p);
      e = cudaMemcpyAsync(pieces[p].dev, ctx->pin + (p & 1) * PIN_BYTES, pieces[p].bytes, kind, ctx->stream);
      if (e == cudaSuccess) e = cudaEventRecord(ctx->pin_ev[p & 1], ctx->stream);
    } else {
      if (p < n) {
        e = cudaMemcpyAsync(ctx->pin + (p & 1) * PIN_BYTES, pieces[p].dev, pieces[p].bytes, kind, ctx->stream);
        if (e == cudaSuccess) e = cudaEventRecord(ctx->pin_ev[p & 1], ctx->stream);
      }
      if (p > 0 && e == cudaSuccess) e = cudaEventSynchronize(ctx->pin_ev[(p - 1) & 1]);
      if (p > 0 && e == cudaSuccess) move(p - 1);
    }
  }
  quit = 1;
  for (auto& th : pool) th.join();
  const cudaError_t es = cudaStreamSynchronize(ctx->stream);
  return e != cudaSuccess ? e : es;
}

// (Re)initialise every system from host arrays: the arrays go to the device
// as they are, the records, the cell lists in index order (cellListInit
// src/EDMD.c:1906 -> addToCell 2053, push-front) and the event set
// (eventListInit 1935) are made there.  Measured on 4x10^6 disks: 83 ms with
// records and lists made on 16 host threads and the overflow list and tree
// walked by one block; on 10^6 disks 18.9 ms.
// first_screen/first_thermo/t_growstop per system come from `desc` unless
// `restart`, which follows the -l load path: normal phase, firstScreen 1,
// firstThermo 1000 (src/EDMD.c:244-247; eventListInit 1958 skips the growth
// shift when load != 0).
static int stage_all(edmd_ctx* ctx, const double* x, const double* y, const double* vx,
                     const double* vy, const double* rad, const double* m, const double* vr,
                     bool restart) {
  ctx->round_dirty = false;
  const int64_t TN = ctx->total_N;
  const int nsys = ctx->nsys;
  cudaStream_t sm = ctx->stream;
  const double* const in[6] = {x, y, vx, vy, rad, m};
  const dim3 gd((ctx->maxN + 255) / 256, nsys);
  // the first bad disk in index order (2 g: position, 2 g + 1: radius), found
  // before any state changes: a small context on the host, without waiting
  // for the device
  unsigned long long first_bad = ~0ull;
  const bool on_device = TN >= ((int64_t)1 << 14);
  if (!on_device)
    for (int s = 0; s < nsys && first_bad == ~0ull; s++)
      for (int64_t g = ctx->disk_off[s]; g < ctx->disk_off[s] + ctx->desc[s].N; g++)
        if (const int b = bad_disk(x[g], y[g], rad[g], ctx->desc[s].Lx, ctx->desc[s].Ly, restart)) {
          first_bad = 2ull * g + (b - 1);
          break;
        }
  if (first_bad == ~0ull) {
    std::vector<HostCopy> list;
    for (int k = 0; k < 6; k++) list.push_back({(void*)in[k], ctx->stage + k * TN, TN * 8});
    CK(host_copies(ctx, list, true));
  }
  if (on_device) {
    CK(cudaMemcpyAsync(ctx->bad, &first_bad, 8, cudaMemcpyHostToDevice, sm));
    k_check<<<gd, 256, 0, sm>>>(ctx->ds, ctx->doff, ctx->stage, TN, restart, ctx->bad);
    CK(cudaGetLastError());
    CK(sync_copy(ctx, &first_bad, ctx->bad, 8, cudaMemcpyDeviceToHost));
  }
  if (first_bad != ~0ull) {
    const int64_t g = (int64_t)(first_bad / 2);
    const int s = (int)(std::upper_bound(ctx->disk_off.begin(), ctx->disk_off.end(), g) - ctx->disk_off.begin()) - 1;
    return set_err(ctx, EDMD_ERR_ARG, std::string(first_bad % 2 ? "radius not zero or normal positive"
                                                                  : "position outside the box") +
                                          " (system " + std::to_string(s) + ")");
  }
  std::vector<SysState> hst(nsys);
  for (int s = 0; s < nsys; s++) {
    const SysDev& S = ctx->hs[s];
    const Box& B = S.B;
    const edmd_system_desc& D = ctx->desc[s];
    SysState& st = hst[s];
    memset(&st, 0, sizeof(st));
    st.k = 0; st.next_wrap = (uint64_t)B.N; st.ovf = NIL;
    st.grow = (!restart && D.t_growstop > 0) ? 1 : 0;
    double fs = restart ? 1.0 : D.first_screen, ft = restart ? 1000.0 : D.first_thermo;
    st.lastThermo = ft + 0.000000001;   // addEventThermo(firstThermo + 1e-9), read by k_init_events
    st.collT[0] = st.grow ? D.t_growstop : -1;
    st.collT[1] = fs;
  }
  CK(cudaMemcpyAsync(ctx->st, hst.data(), nsys * sizeof(SysState), cudaMemcpyHostToDevice, sm));
  if (vr && !restart) CK(cudaMemcpyAsync(ctx->vr, vr, TN * 8, cudaMemcpyHostToDevice, sm));
  else if (!vr && !restart) CK(cudaMemsetAsync(ctx->vr, 0, TN * 8, sm));
  CK(cudaMemsetAsync(ctx->head, 0xff, ctx->total_C * 4, sm));      // NIL
  k_stage<<<gd, 256, 0, sm>>>(ctx->ds, ctx->doff, ctx->stage, TN, restart);
  k_links<<<gd, 256, 0, sm>>>(ctx->ds);
  k_heads<<<gd, 256, 0, sm>>>(ctx->ds);
  CK(cudaGetLastError());
  CK(init_queues(ctx->ds, nsys, ctx->maxN, ctx->engine == EDMD_ENGINE_WARP, sm));
  if (ctx->engine == EDMD_ENGINE_LANE) CK(lane_build(ctx->ds, nsys, sm));
  return report_status(ctx, "initial configuration");
}

extern "C" int edmd_create(int32_t nsys, const edmd_system_desc* desc, const double* x,
                           const double* y, const double* vx, const double* vy,
                           const double* rad, const double* m, const double* vr,
                           int64_t trace_cap, edmd_ctx** out) {
  if (!out || nsys <= 0 || !desc || !x || !y || !vx || !vy || !rad || !m || trace_cap < 0)
    return EDMD_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return EDMD_ERR_NODEV;
  edmd_ctx* ctx = new edmd_ctx();
  *out = ctx;
  ctx->nsys = nsys;
  ctx->hs.resize(nsys);
  ctx->desc.assign(desc, desc + nsys);
  ctx->disk_off.resize(nsys);
  ctx->cell_off.resize(nsys);
  const int rows_cap = 1024;
  std::vector<int64_t> ev_off(nsys), node_off(nsys);
  int64_t TN = 0, TC = 0, TE = 0, TT = 0;
  for (int s = 0; s < nsys; s++) {
    const edmd_system_desc& D = desc[s];
    if (D.N < 2 || !(D.Lx > 0) || !(D.Ly > 0) || (D.contact != EDMD_CONTACT_NONADDITIVE &&
                                                     D.contact != EDMD_CONTACT_ADDITIVE))
      return set_err(ctx, EDMD_ERR_ARG, "bad system descriptor");
    SysDev& S = ctx->hs[s];
    memset(&S, 0, sizeof(S));
    Box& B = S.B;
    B.N = D.N; B.Lx = D.Lx; B.Ly = D.Ly;
    B.additive = D.contact == EDMD_CONTACT_ADDITIVE;
    if (B.additive) ctx->any_additive = true;
    B.hLx = D.Lx / 2; B.hLy = D.Ly / 2;                      // boxConstantHelper 679-714
    B.Nyc = (int)(B.hLy); B.Nxc = (int)(B.hLx);
    if (B.Nxc < 1 || B.Nyc < 1) return set_err(ctx, EDMD_ERR_ARG, "box smaller than one cell");
    if (few_cells(B)) ctx->any_few_cells = true;
    B.cxs = D.Lx / B.Nxc; B.cys = D.Ly / B.Nyc;
    B.cxf = 1 / B.cxs; B.cyf = 1 / B.cys;
    B.dtP = 5.0 / (double)D.N;
    B.dtPN = B.dtP * D.N;
    S.rdtP = 1.0 / B.dtP;
    S.res = D.res; S.Einit = D.Einit; S.dtime = D.dtime; S.dtimeTh = D.dtime_thermo; S.tmax = D.tmax;
    S.L = D.N + NSPECIAL;
    int c = S.L;
    S.nlev = 0;
    int64_t nodes = 0;
    for (;;) {
      if (S.nlev >= MAXLEV) return set_err(ctx, EDMD_ERR_ARG, "system too large");
      S.lev_off[S.nlev] = (int32_t)nodes; S.lev_cnt[S.nlev] = c; nodes += c; S.nlev++;
      if (c == 1) break;
      c = (c + 31) / 32;
    }
    ctx->disk_off[s] = TN; ctx->cell_off[s] = TC; ev_off[s] = TE; node_off[s] = TT;
    TN += D.N; TC += (int64_t)B.Nxc * B.Nyc; TE += 2 * (int64_t)D.N + NSPECIAL; TT += nodes;
    if (D.N > ctx->maxN) ctx->maxN = D.N;
  }
  ctx->total_N = TN; ctx->total_C = TC;
  ctx->engine = g_engine;
  if (ctx->engine == EDMD_ENGINE_AUTO) {
    // One thread per system issues each FP64 instruction for up to 32 systems,
    // but needs enough of them to hide its dependent loads; the warp loop is
    // full from ~3000 systems on.  Hex starts at phi 0.55, 1000 collisions a
    // call, one warp / one thread per system in 1e8 coll/s:
    //   systems   96 disks     256          1024         64-1024 mixed
    //   16384     1.77 / 1.25  1.70 / 1.20  1.50 / 1.14  1.66 / 1.18
    //   24576     1.77 / 1.70  1.68 / 1.63  1.50 / 1.54  1.65 / 1.62
    //   28672     1.77 / 1.89  1.65 / 1.85  -            1.64 / 1.83
    //   32768     1.77 / 2.03  1.64 / 2.03  -            1.63 / 1.98
    // (150 collisions after a restart, whose calendars take longer to build:
    // 24576 x 256 46.7 / 51.6 ms, 28672 54.3 / 56.8, 32768 61.3 / 61.8).  The
    // calendars cost 1 KB per disk.
    const bool many = nsys >= 28672 && 2 * (int64_t)ctx->maxN + NSPECIAL <= 65535 &&
                      TN * (int64_t)(CAL_SUB * CAL_LINE * 2 + 2) <= ((int64_t)32 << 30);
    ctx->engine = many ? EDMD_ENGINE_LANE : EDMD_ENGINE_WARP;
  }
  if (ctx->engine == EDMD_ENGINE_LANE && 2 * (int64_t)ctx->maxN + NSPECIAL > 65535)
    return set_err(ctx, EDMD_ERR_ARG, "thread-per-system engine supports N <= 32766");
  CK(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
  CK(cudaEventCreate(&ctx->e0));
  CK(cudaEventCreate(&ctx->e1));
  // one allocation for the context's arrays (twenty of them: 203 disks 251 us,
  // 20000 disks 500, 192 growth starts 1340; one: 230, 389, 1127)
  size_t bytes = 0;
  auto take = [&](auto** p, size_t n) {
    if (ctx->slab) *p = (std::remove_reference_t<decltype(*p)>)(ctx->slab + bytes);
    bytes += (std::max<size_t>(n, 1) * sizeof(**p) + 255) & ~(size_t)255;
  };
  auto arrays = [&]() {
    bytes = 0;
    take(&ctx->d, TN); take(&ctx->vr, TN);
    take(&ctx->cx, TN); take(&ctx->cy, TN); take(&ctx->prv, TN);
    take(&ctx->crossX, TN); take(&ctx->crossY, TN);
    take(&ctx->head, TC);
    take(&ctx->ev, TE); take(&ctx->on, TE); take(&ctx->op, TE);
    take(&ctx->tree, TT);
    take(&ctx->st, nsys);
    take(&ctx->trace, (size_t)nsys * trace_cap);
    take(&ctx->rows, (size_t)nsys * rows_cap * 9);
    take(&ctx->stage, 6 * TN);
    take(&ctx->order, nsys);
    take(&ctx->ds, nsys);
    take(&ctx->doff, nsys);
    take(&ctx->bad, 1);
  };
  arrays();
  CK(dalloc(&ctx->slab, bytes));
  arrays();
  if (ctx->engine == EDMD_ENGINE_LANE) {
    CK(dalloc(&ctx->cal, (size_t)TN * CAL_SUB * CAL_LINE));
    CK(dalloc(&ctx->mask, (size_t)TN));
  }
  for (int s = 0; s < nsys; s++) {
    SysDev& S = ctx->hs[s];
    int64_t o = ctx->disk_off[s];
    S.d = ctx->d + o; S.vr = ctx->vr + o;
    S.cx = ctx->cx + o; S.cy = ctx->cy + o; S.prv = ctx->prv + o;
    S.crossX = ctx->crossX + o; S.crossY = ctx->crossY + o;
    S.head = ctx->head + ctx->cell_off[s];
    S.ev = ctx->ev + ev_off[s]; S.on = ctx->on + ev_off[s]; S.op = ctx->op + ev_off[s];
    S.tree = ctx->tree + node_off[s];
    S.st = ctx->st + s;
    S.trace = trace_cap > 0 ? (void*)(ctx->trace + (size_t)s * trace_cap) : nullptr;
    S.trace_cap = trace_cap;
    S.rows = ctx->rows + (size_t)s * rows_cap * 9;
    S.rows_cap = rows_cap;
    if (ctx->engine == EDMD_ENGINE_LANE) {
      S.cal = ctx->cal + (size_t)o * CAL_SUB * CAL_LINE;
      S.mask = ctx->mask + o;
      S.invw = CAL_SUB / S.B.dtP;
    }
  }
  CK(cudaMemcpyAsync(ctx->ds, ctx->hs.data(), nsys * sizeof(SysDev), cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(ctx->doff, ctx->disk_off.data(), nsys * 8, cudaMemcpyHostToDevice, ctx->stream));
  return stage_all(ctx, x, y, vx, vy, rad, m, vr, false);
}

extern "C" int edmd_load_state(edmd_ctx* ctx, const double* x, const double* y, const double* vx,
                               const double* vy, const double* rad, const double* m) {
  if (!ctx || !x || !y || !vx || !vy || !rad || !m) return EDMD_ERR_ARG;
  return stage_all(ctx, x, y, vx, vy, rad, m, nullptr, true);
}

// the event loop on `nsys` places on the context's stream, with the tables of
// waiting systems when they exceed the resident lane groups
static int run_launch(edmd_ctx* ctx, RunArgs A, int nsys, int gw, int nsm) {
  RunShape shape = run_shape(gw, ctx->any_additive, nsys, nsm, !ctx->any_few_cells);
  int per_sm = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shape.kernel, 32 * shape.warps, 0));
  if (shape.systems == 1 && per_sm * nsm < nsys) {
    shape = run_shape(gw, ctx->any_additive, nsys, nsm, false);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shape.kernel, 32 * shape.warps, 0));
  }
  const int per_block = shape.systems;
  const int grid = std::max(1, std::min(per_sm * nsm, (nsys + per_block - 1) / per_block));
  A.nrun = std::min(nsys, grid * per_block);
  A.nwait = nsys - A.nrun;
  if (A.nwait) {
    if (!ctx->waiting) {
      CK(dalloc(&ctx->waiting, ctx->nsys)); CK(dalloc(&ctx->ticket, 2)); CK(dalloc(&ctx->progress, ctx->nsys));
    }
    A.waiting = ctx->waiting; A.ticket = ctx->ticket; A.progress = ctx->progress;
    k_waiting<<<(nsys + 255) / 256, 256, 0, ctx->stream>>>(A);
    ctx->last_launches++;
  }
  shape.kernel<<<grid, 32 * shape.warps, 0, ctx->stream>>>(ctx->ds, A);
  CK(cudaGetLastError());
  ctx->last_launches++;
  return EDMD_OK;
}

// EDMD_F_SMEM: the systems whose engine state fits one block's shared memory
// go to k_run_smem on a second stream, the others to k_run on the context's
// stream; both start after e0 and the context's stream waits for the second
// one before e1.
static int advance_smem_split(edmd_ctx* ctx, RunArgs A, int nsm) {
  int dev = 0, optin = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t limit = (size_t)optin - sizeof(WarpSmem) - 1024;
  std::vector<int32_t> fit, rest;
  size_t need = 0;
  for (int s = 0; s < ctx->nsys; s++) {
    const size_t b = smem_layout(ctx->hs[s]).total;
    if (b <= limit) { fit.push_back(s); need = b > need ? b : need; }
    else rest.push_back(s);
  }
  if (!ctx->smem_list) {
    CK(dalloc(&ctx->smem_list, ctx->nsys));
    CK(dalloc(&ctx->smem_work, 1));
    CK(cudaEventCreateWithFlags(&ctx->e2, cudaEventDisableTiming));
  }
  if (!ctx->stream2) CK(cudaStreamCreateWithFlags(&ctx->stream2, cudaStreamNonBlocking));
  if (!rest.empty())
    CK(cudaMemcpyAsync(ctx->order, rest.data(), rest.size() * sizeof(int32_t), cudaMemcpyHostToDevice,
                       ctx->stream));
  if (!fit.empty())
    CK(cudaMemcpyAsync(ctx->smem_list, fit.data(), fit.size() * sizeof(int32_t), cudaMemcpyHostToDevice,
                       ctx->stream));
  CK(cudaMemsetAsync(ctx->smem_work, 0, sizeof(int32_t), ctx->stream));
  CK(cudaEventRecord(ctx->e0, ctx->stream));
  if (!fit.empty()) {
    CK(cudaFuncSetAttribute(k_run_smem, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need));
    int per = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_run_smem, 32, need));
    int g = per * nsm;
    if (g > (int)fit.size()) g = (int)fit.size();
    if (g < 1) g = 1;
    CK(cudaStreamWaitEvent(ctx->stream2, ctx->e0, 0));
    k_run_smem<<<g, 32, need, ctx->stream2>>>(ctx->ds, A, ctx->smem_list, (int)fit.size(), ctx->smem_work);
    CK(cudaGetLastError());
    ctx->last_launches++;
    CK(cudaEventRecord(ctx->e2, ctx->stream2));
  }
  if (!rest.empty()) {
    RunArgs B = A;
    B.order = ctx->order;
    const int rc = run_launch(ctx, B, (int)rest.size(), 32, nsm);
    if (rc) return rc;
  }
  if (!fit.empty()) CK(cudaStreamWaitEvent(ctx->stream, ctx->e2, 0));
  return EDMD_OK;
}

extern "C" int edmd_advance(edmd_ctx* ctx, int64_t max_coll, double t_stop, uint32_t flags,
                            int64_t max_events, float* elapsed_ms) {
  if (!ctx) return EDMD_ERR_ARG;
  if (max_coll < 0 || max_events <= 0) return set_err(ctx, EDMD_ERR_ARG, "bad advance limits");
  if (ctx->round_dirty)
    return set_err(ctx, EDMD_ERR_ARG, "advanced by the round engine: reload the state with edmd_load_state");
  RunArgs A;
  A.max_coll = max_coll; A.t_stop = t_stop; A.flags = flags; A.max_events = max_events;
  A.nsys = ctx->nsys;
  A.order = nullptr; A.waiting = nullptr; A.ticket = nullptr; A.progress = nullptr;
  A.nwait = 0; A.nrun = ctx->nsys;
  ctx->last_launches = 0;
  if (ctx->engine == EDMD_ENGINE_LANE) {
    CK(cudaEventRecord(ctx->e0, ctx->stream));
    CK(lane_run_launch(ctx->ds, A, g_lane_threads, ctx->stream));
    ctx->last_launches = 1;
  } else {
    int dev = 0, nsm = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int gw = g_group;                     // lanes per system: 4, 8, 16 or 32
    int rc;
    if ((flags & EDMD_F_SMEM) && gw == 32) {
      rc = advance_smem_split(ctx, A, nsm);
    } else {
      CK(cudaEventRecord(ctx->e0, ctx->stream));
      rc = run_launch(ctx, A, ctx->nsys, gw, nsm);
    }
    if (rc) return rc;
  }
  CK(cudaGetLastError());
  CK(cudaEventRecord(ctx->e1, ctx->stream));
  CK(cudaEventSynchronize(ctx->e1));
  CK(cudaEventElapsedTime(&ctx->last_ms, ctx->e0, ctx->e1));
  if (elapsed_ms) *elapsed_ms = ctx->last_ms;
  return report_status(ctx, "advance");
}

extern "C" int edmd_sync(edmd_ctx* ctx) {
  if (!ctx) return EDMD_ERR_ARG;
  k_sync<<<dim3((ctx->maxN + 255) / 256, ctx->nsys), 256, 0, ctx->stream>>>(ctx->ds);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(ctx->stream));
  return EDMD_OK;
}

extern "C" int edmd_get_state(edmd_ctx* ctx, int32_t s, double* x, double* y, double* vx,
                              double* vy, double* rad, double* m, int32_t* cell, uint32_t* coll) {
  if (!ctx || s < 0 || s >= ctx->nsys) return EDMD_ERR_ARG;
  const SysDev& S = ctx->hs[s];
  int N = S.B.N;
  std::vector<Disk> hd(N);
  std::vector<int32_t> hcx(N), hcy(N);
  CK(sync_copy(ctx, hd.data(), S.d, N * sizeof(Disk), cudaMemcpyDeviceToHost));
  CK(sync_copy(ctx, hcx.data(), S.cx, N * 4, cudaMemcpyDeviceToHost));
  CK(sync_copy(ctx, hcy.data(), S.cy, N * 4, cudaMemcpyDeviceToHost));
  for (int i = 0; i < N; i++) {
    if (x) x[i] = hd[i].x;
    if (y) y[i] = hd[i].y;
    if (vx) vx[i] = hd[i].vx;
    if (vy) vy[i] = hd[i].vy;
    if (rad) rad[i] = hd[i].rad;
    if (m) m[i] = hd[i].m;
    if (cell) cell[i] = hcy[i] * S.B.Nxc + hcx[i];
    if (coll) coll[i] = hd[i].coll;
  }
  return EDMD_OK;
}

extern "C" int edmd_get_states(edmd_ctx* ctx, double* x, double* y, double* vx, double* vy,
                               double* rad, double* m) {
  if (!ctx) return EDMD_ERR_ARG;
  const int64_t TN = ctx->total_N;
  k_gather<<<(unsigned)((TN + 255) / 256), 256, 0, ctx->stream>>>(ctx->d, TN, ctx->stage);
  CK(cudaGetLastError());
  double* outs[6] = {x, y, vx, vy, rad, m};
  std::vector<HostCopy> list;
  for (int k = 0; k < 6; k++)
    if (outs[k]) list.push_back({outs[k], ctx->stage + k * TN, TN * 8});
  CK(host_copies(ctx, list, false));
  return EDMD_OK;
}

extern "C" int edmd_get_counters(edmd_ctx* ctx, int32_t s, edmd_counters* out) {
  if (!ctx || s < 0 || s >= ctx->nsys || !out) return EDMD_ERR_ARG;
  SysState R;
  CK(sync_copy(ctx, &R, ctx->hs[s].st, sizeof(R), cudaMemcpyDeviceToHost));
  out->ncol = R.ncol; out->ncol_total = R.ncol_total; out->ncross = R.ncross;
  out->nstale = R.nstale; out->npair = R.npair; out->npred = R.npred; out->nevents = R.nevents;
  out->nscreen = R.nscreen;
  out->t = R.t; out->growing = R.grow; out->stop_reason = R.stop_reason;
  return EDMD_OK;
}

extern "C" int edmd_get_all_counters(edmd_ctx* ctx, edmd_counters* out) {
  if (!ctx || !out) return EDMD_ERR_ARG;
  std::vector<SysState> R(ctx->nsys);
  CK(sync_copy(ctx, R.data(), ctx->st, ctx->nsys * sizeof(SysState), cudaMemcpyDeviceToHost));
  for (int s = 0; s < ctx->nsys; s++) {
    edmd_counters& o = out[s];
    o.ncol = R[s].ncol; o.ncol_total = R[s].ncol_total; o.ncross = R[s].ncross;
    o.nstale = R[s].nstale; o.npair = R[s].npair; o.npred = R[s].npred; o.nevents = R[s].nevents;
    o.nscreen = R[s].nscreen;
    o.t = R[s].t; o.growing = R[s].grow; o.stop_reason = R[s].stop_reason;
  }
  return EDMD_OK;
}

extern "C" int edmd_get_virial(edmd_ctx* ctx, int32_t s, double out[4], int32_t reset) {
  if (!ctx || s < 0 || s >= ctx->nsys || !out) return EDMD_ERR_ARG;
  SysState* p = ctx->hs[s].st;
  CK(sync_copy(ctx, out, p->collT, 4 * sizeof(double), cudaMemcpyDeviceToHost));
  if (reset) CK(sync_set(ctx, p->collT, 0, 4 * sizeof(double)));
  return EDMD_OK;
}

extern "C" int edmd_get_thermo(edmd_ctx* ctx, int32_t s, double* rows, int32_t cap, int32_t* n) {
  if (!ctx || s < 0 || s >= ctx->nsys || !n) return EDMD_ERR_ARG;
  const SysDev& S = ctx->hs[s];
  int32_t nr = 0;
  CK(sync_copy(ctx, &nr, &S.st->nrows, 4, cudaMemcpyDeviceToHost));
  *n = nr;
  int k = nr < cap ? nr : cap;
  if (k > S.rows_cap) k = S.rows_cap;
  if (rows && k > 0) CK(sync_copy(ctx, rows, S.rows, (size_t)k * 9 * 8, cudaMemcpyDeviceToHost));
  return nr > S.rows_cap ? EDMD_ERR_CAPACITY : EDMD_OK;
}

extern "C" int edmd_take_thermo(edmd_ctx* ctx, int32_t s, double* rows, int32_t cap, int32_t* n) {
  const int rc = edmd_get_thermo(ctx, s, rows, cap, n);
  if (rc != EDMD_OK && rc != EDMD_ERR_CAPACITY) return rc;
  const int32_t zero = 0;
  CK(sync_copy(ctx, &ctx->hs[s].st->nrows, &zero, 4, cudaMemcpyHostToDevice));
  return rc;
}

extern "C" int edmd_get_trace(edmd_ctx* ctx, int32_t s, edmd_collision* out, int64_t cap, int64_t* n) {
  if (!ctx || s < 0 || s >= ctx->nsys || !n) return EDMD_ERR_ARG;
  const SysDev& S = ctx->hs[s];
  uint64_t nt = 0;
  CK(sync_copy(ctx, &nt, &S.st->ntrace, 8, cudaMemcpyDeviceToHost));
  *n = (int64_t)nt;
  int64_t k = (int64_t)nt < cap ? (int64_t)nt : cap;
  if (k > S.trace_cap) k = S.trace_cap;
  if (out && k > 0) CK(sync_copy(ctx, out, S.trace, k * sizeof(edmd_collision), cudaMemcpyDeviceToHost));
  return (int64_t)nt > S.trace_cap ? EDMD_ERR_CAPACITY : EDMD_OK;
}

extern "C" int edmd_set_device(int32_t dev) {
  return cudaSetDevice(dev) == cudaSuccess ? EDMD_OK : EDMD_ERR_CUDA;
}

extern "C" int edmd_host_alloc(void** p, int64_t bytes) {
  if (!p || bytes <= 0) return EDMD_ERR_ARG;
  return cudaMallocHost(p, (size_t)bytes) == cudaSuccess ? EDMD_OK : EDMD_ERR_CUDA;
}

extern "C" int edmd_host_free(void* p) {
  return cudaFreeHost(p) == cudaSuccess ? EDMD_OK : EDMD_ERR_CUDA;
}

extern "C" int edmd_destroy(edmd_ctx* ctx) {
  if (!ctx) return EDMD_OK;
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  round_free(ctx);
  void* ptrs[] = {ctx->slab, ctx->waiting, ctx->ticket, ctx->progress, ctx->cal, ctx->mask};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  for (void* p : ctx->ckpt)
    if (p) cudaFree(p);
  if (ctx->logbuf) cudaFree(ctx->logbuf);
  if (ctx->pcf) cudaFree(ctx->pcf);
  if (ctx->pin) cudaFreeHost(ctx->pin);
  for (cudaEvent_t e : ctx->pin_ev)
    if (e) cudaEventDestroy(e);
  if (ctx->e0) cudaEventDestroy(ctx->e0);
  if (ctx->e1) cudaEventDestroy(ctx->e1);
  if (ctx->c0) cudaEventDestroy(ctx->c0);
  if (ctx->e2) cudaEventDestroy(ctx->e2);
  if (ctx->stream2) cudaStreamDestroy(ctx->stream2);
  if (ctx->smem_list) cudaFree(ctx->smem_list);
  if (ctx->smem_work) cudaFree(ctx->smem_work);
  if (ctx->c1) cudaEventDestroy(ctx->c1);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
  return EDMD_OK;
}

extern "C" int edmd_get_engine(const edmd_ctx* ctx) {
  return ctx ? ctx->engine : -1;
}

extern "C" int edmd_get_last_ms(const edmd_ctx* ctx, float* ms) {
  if (!ctx || !ms) return EDMD_ERR_ARG;
  *ms = ctx->last_ms;
  return EDMD_OK;
}

extern "C" int edmd_get_last_launches(const edmd_ctx* ctx, int64_t* n) {
  if (!ctx || !n) return EDMD_ERR_ARG;
  *n = ctx->last_launches;
  return EDMD_OK;
}

// ==================================================================== allocation-free entry point
//
// edmd_run_noalloc serves callers that must not allocate device memory, for
// example code that runs inside a latency-critical loop or a host framework
// that owns every device buffer and forbids cudaMalloc/cudaFree after start-up.
// The caller passes its own device arrays (the state in and out); everything
// the engine needs besides them -- the system descriptor, cell lists, event
// records, the tournament tree and the scalar state -- lives
// in the file-scope array below, which every GPU that loads this library keeps
// until the process exits.
namespace {
constexpr int64_t NOALLOC_MAX_N = 8192;        // disks per call
constexpr int64_t NOALLOC_MAX_CELLS = 65536;   // Nxcells * Nycells per call
constexpr size_t NOALLOC_BYTES = (size_t)4 << 20;
constexpr int NOALLOC_MAX_DEVICES = 64;
// event budget of one call (see edmd_run_noalloc)
constexpr int64_t NOALLOC_EVENTS_PER_COLL = 256, NOALLOC_EVENTS_PER_DISK = 256, NOALLOC_EVENTS_BASE = 1 << 20;
}

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];
static unsigned char* g_noalloc_addr[NOALLOC_MAX_DEVICES];   // device address, per device
static thread_local std::string g_noalloc_err;

namespace {

__global__ void k_noalloc_put(SysDev s, SysDev* dst) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *dst = s;
}

// disk records, cell lists (index order, push-front as addToCell) and the
// scalar state from the caller's device arrays; one thread, N <= 8192.
// A position outside [0, Lx) x [0, Ly) (or a NaN), or a radius that is not
// zero or normal positive, is an argument error, as in edmd_create: the
// scalar state gets status EDMD_ERR_ARG with the first such
// disk in err_a, the event loop then does nothing, and the host reports it.
// The cell index is still clamped into the grid so that the initial
// predictions that run before the loop stay inside the arrays.
__global__ void k_noalloc_stage(const SysDev* __restrict__ sys, const double* x, const double* y,
                                const double* vx, const double* vy, const double* rad,
                                const double* m, double first_screen, double first_thermo) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const SysDev& S = sys[0];
  const Box& B = S.B;
  const int N = B.N;
  int bad = -1;
  for (int c = 0; c < B.Nxc * B.Nyc; c++) S.head[c] = NIL;
  for (int i = 0; i < N; i++) {
    Disk q;
    q.x = x[i]; q.y = y[i]; q.vx = vx[i]; q.vy = vy[i]; q.tl = 0; q.rad = rad[i]; q.m = m[i];
    q.coll = 0;
    if (bad < 0 && !(q.x >= 0 && q.x < B.Lx && q.y >= 0 && q.y < B.Ly && radius_ok(q.rad))) bad = i;
    int X = (int)(q.x * B.cxf), Y = (int)(q.y * B.cyf);
    if (!(X < B.Nxc)) X = B.Nxc - 1;
    if (!(Y < B.Nyc)) Y = B.Nyc - 1;
    if (!(X >= 0)) X = 0;
    if (!(Y >= 0)) Y = 0;
    S.cx[i] = X; S.cy[i] = Y; S.prv[i] = NIL;
    S.crossX[i] = 0; S.crossY[i] = 0;
    S.vr[i] = 0;
    q.nxt = S.head[Y * B.Nxc + X];
    S.head[Y * B.Nxc + X] = i;
    if (q.nxt != NIL) S.prv[q.nxt] = i;
    S.d[i] = q;
  }
  SysState st;
  memset(&st, 0, sizeof(st));
  st.k = 0; st.next_wrap = (uint64_t)N; st.ovf = NIL; st.grow = 0;
  st.lastThermo = first_thermo + 0.000000001;   // read by k_init_events
  st.collT[0] = -1;
  st.collT[1] = first_screen;
  if (bad >= 0) { st.status = EDMD_ERR_ARG; st.err_a = bad; }
  *S.st = st;
}

__global__ void k_noalloc_out(const SysDev* __restrict__ sys, double* x, double* y, double* vx,
                              double* vy) {
  const SysDev& S = sys[0];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.B.N; i += gridDim.x * blockDim.x) {
    Disk p = S.d[i];
    x[i] = p.x; y[i] = p.y; vx[i] = p.vx; vy[i] = p.vy;
  }
}

int noalloc_fail(int code, const char* m) {
  g_noalloc_err = m;
  return code;
}

}  // namespace

extern "C" int edmd_run_noalloc(const edmd_system_desc* desc, double* x, double* y, double* vx,
                                double* vy, const double* rad, const double* m, int64_t max_coll,
                                double t_stop, int64_t* ncol_out, double* t_out, void* stream) {
  if (!desc || !x || !y || !vx || !vy || !rad || !m || max_coll < 0)
    return noalloc_fail(EDMD_ERR_ARG, "edmd_run_noalloc: null argument or negative max_coll");
  const edmd_system_desc& D = *desc;
  if (D.t_growstop > 0)
    return noalloc_fail(EDMD_ERR_ARG, "edmd_run_noalloc: growth starts are not supported");
  if (D.N < 2 || D.N > NOALLOC_MAX_N)
    return noalloc_fail(EDMD_ERR_CAPACITY, "edmd_run_noalloc: N must be in [2, 8192]");
  if (D.contact != EDMD_CONTACT_NONADDITIVE && D.contact != EDMD_CONTACT_ADDITIVE)
    return noalloc_fail(EDMD_ERR_ARG, "edmd_run_noalloc: bad contact rule");
  SysDev S;
  memset(&S, 0, sizeof(S));
  Box& B = S.B;
  B.N = D.N; B.Lx = D.Lx; B.Ly = D.Ly;
  B.additive = D.contact == EDMD_CONTACT_ADDITIVE;
  B.hLx = D.Lx / 2; B.hLy = D.Ly / 2;                      // boxConstantHelper 679-714
  B.Nyc = (int)(B.hLy); B.Nxc = (int)(B.hLx);
  if (!(D.Lx > 0) || !(D.Ly > 0) || B.Nxc < 1 || B.Nyc < 1)
    return noalloc_fail(EDMD_ERR_ARG, "edmd_run_noalloc: box smaller than one cell");
  if ((int64_t)B.Nxc * B.Nyc > NOALLOC_MAX_CELLS)
    return noalloc_fail(EDMD_ERR_CAPACITY, "edmd_run_noalloc: more than 65536 cells");
  B.cxs = D.Lx / B.Nxc; B.cys = D.Ly / B.Nyc;
  B.cxf = 1 / B.cxs; B.cyf = 1 / B.cys;
  B.dtP = 5.0 / (double)D.N;
  B.dtPN = B.dtP * D.N;
  S.rdtP = 1.0 / B.dtP;
  S.res = D.res; S.Einit = D.Einit; S.dtime = D.dtime; S.dtimeTh = D.dtime_thermo; S.tmax = D.tmax;
  S.L = D.N + NSPECIAL;
  int c = S.L;
  size_t nodes = 0;
  for (;;) {
    S.lev_off[S.nlev] = (int32_t)nodes; S.lev_cnt[S.nlev] = c; nodes += c; S.nlev++;
    if (c == 1) break;
    c = (c + 31) / 32;
  }
  // once per device, with that device current: the device address of the array
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES)
    return noalloc_fail(EDMD_ERR_CUDA, "edmd_run_noalloc: no current CUDA device");
  if (!g_noalloc_addr[dev]) {
    void* a = nullptr;
    cudaError_t ce = cudaGetSymbolAddress(&a, g_noalloc_scratch);
    if (ce != cudaSuccess || !a) return noalloc_fail(EDMD_ERR_CUDA, cudaGetErrorString(ce));
    g_noalloc_addr[dev] = (unsigned char*)a;
  }
  unsigned char* base = g_noalloc_addr[dev];
  size_t off = 0;
  auto take = [&](size_t bytes) { unsigned char* r = base + off; off += align_up(bytes, 256); return r; };
  size_t N = D.N, E = 2 * N + NSPECIAL, C = (size_t)B.Nxc * B.Nyc;
  SysDev* dsys = (SysDev*)take(sizeof(SysDev));
  S.st = (SysState*)take(sizeof(SysState));
  S.d = (Disk*)take(N * sizeof(Disk));
  S.vr = (double*)take(N * 8);
  S.cx = (int32_t*)take(N * 4); S.cy = (int32_t*)take(N * 4); S.prv = (int32_t*)take(N * 4);
  S.crossX = (int32_t*)take(N * 4); S.crossY = (int32_t*)take(N * 4);
  S.head = (int32_t*)take(C * 4);
  S.ev = (Ev*)take(E * sizeof(Ev));
  S.on = (int32_t*)take(E * 4); S.op = (int32_t*)take(E * 4);
  S.tree = (Node*)take(nodes * sizeof(Node));
  S.rows = (double*)take(64 * 9 * 8);
  S.rows_cap = 64;
  S.trace = nullptr; S.trace_cap = 0;
  if (off > NOALLOC_BYTES)
    return noalloc_fail(EDMD_ERR_CAPACITY, "edmd_run_noalloc: system does not fit the 4 MiB scratch array");
  cudaStream_t st = (cudaStream_t)stream;
  RunArgs A;
  // a finite event budget: NOALLOC_EVENTS_PER_COLL events per requested
  // collision plus NOALLOC_EVENTS_PER_DISK per disk (saturating), so that a
  // loop whose clock stops advancing ends with EDMD_ERR_BUDGET
  const int64_t cap = (int64_t)1 << 60;
  const int64_t per_coll = max_coll > cap / NOALLOC_EVENTS_PER_COLL ? cap : max_coll * NOALLOC_EVENTS_PER_COLL;
  const int64_t budget = std::min(cap, per_coll + (int64_t)N * NOALLOC_EVENTS_PER_DISK + NOALLOC_EVENTS_BASE);
  A.max_coll = max_coll; A.t_stop = t_stop; A.flags = 0; A.max_events = budget;
  A.nsys = 1; A.order = nullptr; A.waiting = nullptr; A.ticket = nullptr; A.progress = nullptr;
  A.nwait = 0; A.nrun = 1;
  k_noalloc_put<<<1, 1, 0, st>>>(S, dsys);
  k_noalloc_stage<<<1, 32, 0, st>>>(dsys, x, y, vx, vy, rad, m, D.first_screen, D.first_thermo);
  if (cudaError_t qe = init_queues(dsys, 1, N, true, st); qe != cudaSuccess)
    return noalloc_fail(EDMD_ERR_CUDA, cudaGetErrorString(qe));
  const RunShape shape = run_shape(32, B.additive != 0, 1, 1, !few_cells(B));
  shape.kernel<<<1, 32 * shape.warps, 0, st>>>(dsys, A);
  k_sync<<<dim3((N + 255) / 256, 1), 256, 0, st>>>(dsys);
  k_noalloc_out<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(dsys, x, y, vx, vy);
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return noalloc_fail(EDMD_ERR_CUDA, cudaGetErrorString(ce));
  SysState R;
  ce = cudaMemcpyAsync(&R, S.st, sizeof(R), cudaMemcpyDeviceToHost, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  if (ce != cudaSuccess) return noalloc_fail(EDMD_ERR_CUDA, cudaGetErrorString(ce));
  if (ncol_out) *ncol_out = (int64_t)R.ncol;
  if (t_out) *t_out = R.t;
  if (R.status == EDMD_ERR_ARG)
    return noalloc_fail(R.status, ("edmd_run_noalloc: position of disk " + std::to_string(R.err_a) +
                                   " outside the box").c_str());
  if (R.status == EDMD_ERR_OVERLAP)
    return noalloc_fail(R.status, ("edmd_run_noalloc: overlapping disks " + std::to_string(R.err_a) + " and " +
                                   std::to_string(R.err_b)).c_str());
  if (R.status == EDMD_ERR_BUDGET)
    return noalloc_fail(R.status, "edmd_run_noalloc: event budget exhausted (the state at the stop is written back)");
  if (R.status != EDMD_OK) return noalloc_fail(R.status, "edmd_run_noalloc: event loop stopped");
  g_noalloc_err.clear();
  return EDMD_OK;
}

extern "C" const char* edmd_last_error(const edmd_ctx* ctx) {
  return ctx ? ctx->err.c_str() : g_noalloc_err.c_str();
}
