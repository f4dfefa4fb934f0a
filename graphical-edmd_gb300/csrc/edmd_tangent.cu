// edmd_tangent.cu -- tangent-linear and adjoint dynamics of the hard-disk system,
// engine checkpoints, and the collision-geometry log that feeds them.
//
// The reference has no derivatives; this is the differentiation pattern built on
// top of its dynamics.  Between collisions a disk flies freely,
//     dr(t) = dr(t0) + dv (t - t0),   dv constant,
// and at an elastic collision of i and j (src/EDMD.c:3587-3827: r = r_j - r_i at
// contact, v = v_j - v_i before it, f = (1+res)/(m_i+m_j) (r.v)/sigma^2,
// v_i += f m_j r, v_j -= f m_i r) the tangent map is that of Dellago, Posch and
// Hoover (Phys. Rev. E 53, 1485 (1996)), re-derived here:
//     dt_c = -(r . dr_ij) / (r . v)                  shift of the collision time
//     drc  = dr_ij + v dt_c                          relative position at contact
//     df   = (f / (r . v)) (v . drc + r . dv_ij)
//     w    = df r + f drc
//     dr_i' = dr_i - Dv_i dt_c,  dr_j' = dr_j - Dv_j dt_c     (Dv = velocity jumps)
//     dv_i' = dv_i + m_j w,      dv_j' = dv_j - m_i w
// The adjoint applies the transpose of the same map backwards over the log.
#include "edmd_ctx.h"

#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>

namespace {

// ---------------------------------------------------------------- tangent kernels

// A collision of the log with what its maps need beside it, 32 at a time in
// shared memory: the masses and the quotient come for all 32 in one pass, so
// the chain from collision to collision waits for none of them.
struct Coll {
  double t, dx, dy, dvx, dvy, f, mi, mj, rv, frv;
  int32_t i, j;
};
__device__ __forceinline__ Coll coll_of(const edmd_log_entry& L, const Disk* __restrict__ d) {
  Coll c;
  c.i = L.i; c.j = L.j; c.t = L.t;
  c.dx = L.dx; c.dy = L.dy; c.dvx = L.dvx; c.dvy = L.dvy; c.f = L.f;
  c.mi = d[L.i].m; c.mj = d[L.j].m;
  c.rv = L.dx * L.dvx + L.dy * L.dvy;
  c.frv = div_rn(L.f, c.rv);
  return c;
}

// T is row-major [4N][K]: row 4i+c holds component c (dx, dy, dvx, dvy) of disk
// i for the K tangent vectors, so lane k of a warp reads one coalesced row.
// One warp, bound by the chain from collision to collision: the rows of the
// next collision are loaded while this one is computed, unless they share a
// disk.  1024 disks, 32 vectors: 3.1 -> 1.2 us a collision.
__device__ __forceinline__ void tangent_apply_warp(const edmd_log_entry* __restrict__ log, int64_t M,
                                                   const Disk* __restrict__ d, double* T, double* tl, int K, int k,
                                                   Coll* tile) {
  const bool on = k < K;
  double xi = 0, yi = 0, vxi = 0, vyi = 0, xj = 0, yj = 0, vxj = 0, vyj = 0, ti = 0, tj = 0;
  auto load = [&](int i, double& x, double& y, double& vx, double& vy, double& t) {
    const double* R = T + (size_t)4 * i * K + k;
    if (on) { x = R[0]; y = R[K]; vx = R[2 * K]; vy = R[3 * K]; }
    t = tl[i];
  };
  for (int64_t n0 = 0; n0 < M; n0 += 32) {
    __syncwarp();
    if (n0 + k < M) tile[k] = coll_of(log[n0 + k], d);
    __syncwarp();
    const int cnt = (int)(M - n0 < 32 ? M - n0 : 32);
    load(tile[0].i, xi, yi, vxi, vyi, ti);
    load(tile[0].j, xj, yj, vxj, vyj, tj);
    for (int n = 0; n < cnt; n++) {
      const Coll& L = tile[n];
      const int i = L.i, j = L.j;
      const int ni = n + 1 < cnt ? tile[n + 1].i : -1, nj = n + 1 < cnt ? tile[n + 1].j : -1;
      const bool si = ni == i || ni == j, sj = nj == i || nj == j;      // written below
      double axi = 0, ayi = 0, avxi = 0, avyi = 0, axj = 0, ayj = 0, avxj = 0, avyj = 0, ati = 0, atj = 0;
      if (ni >= 0 && !si) load(ni, axi, ayi, avxi, avyi, ati);
      if (nj >= 0 && !sj) load(nj, axj, ayj, avxj, avyj, atj);
      {
        double* Ri = T + (size_t)4 * i * K + k;
        double* Rj = T + (size_t)4 * j * K + k;
        // free flight to the collision
        xi += vxi * (L.t - ti); yi += vyi * (L.t - ti);
        xj += vxj * (L.t - tj); yj += vyj * (L.t - tj);
        const double drx = xj - xi, dry = yj - yi, dvx = vxj - vxi, dvy = vyj - vyi;
        const double dtc = div_rn(-(L.dx * drx + L.dy * dry), L.rv);
        const double rcx = drx + L.dvx * dtc, rcy = dry + L.dvy * dtc;
        const double df = L.frv * (L.dvx * rcx + L.dvy * rcy + L.dx * dvx + L.dy * dvy);
        const double wx = df * L.dx + L.f * rcx, wy = df * L.dy + L.f * rcy;
        const double Dvix = L.f * L.mj * L.dx, Dviy = L.f * L.mj * L.dy;
        const double Dvjx = -L.f * L.mi * L.dx, Dvjy = -L.f * L.mi * L.dy;
        if (on) {
          Ri[0] = xi - Dvix * dtc;           Ri[K] = yi - Dviy * dtc;
          Rj[0] = xj - Dvjx * dtc;           Rj[K] = yj - Dvjy * dtc;
          Ri[2 * K] = vxi + L.mj * wx;       Ri[3 * K] = vyi + L.mj * wy;
          Rj[2 * K] = vxj - L.mi * wx;       Rj[3 * K] = vyj - L.mi * wy;
        }
      }
      if (k == 0) { tl[i] = L.t; tl[j] = L.t; }
      __syncwarp();
      if (si) load(ni, axi, ayi, avxi, avyi, ati);
      if (sj) load(nj, axj, ayj, avxj, avyj, atj);
      xi = axi; yi = ayi; vxi = avxi; vyi = avyi; ti = ati;
      xj = axj; yj = ayj; vxj = avxj; vyj = avyj; tj = atj;
    }
  }
}

__global__ void __launch_bounds__(32) k_tangent_apply(const edmd_log_entry* __restrict__ log, int64_t M,
                                                      const Disk* __restrict__ d, double* T, double* tl, int K) {
  __shared__ Coll tile[32];
  tangent_apply_warp(log, M, d, T, tl, K, threadIdx.x, tile);
}

// value of row e at the common time tq (virtual free flight, T itself unchanged)
__device__ __forceinline__ double row_at(const double* T, const double* tl, int e, int k, int K,
                                         double tq) {
  int c = e & 3;
  double v = T[(size_t)e * K + k];
  if (c < 2) v += T[(size_t)(e + 2) * K + k] * (tq - tl[e >> 2]);
  return v;
}

// per-block partial Gram matrices of the tangent vectors flown to tq; summed
// over the blocks in a fixed order by k_gram_sum, so the result is
// reproducible run to run
__global__ void k_gram(const double* __restrict__ T, const double* __restrict__ tl, int N, int K,
                       const double* __restrict__ tqp, double* __restrict__ Gp) {
  const double tq = *tqp;
  __shared__ double rows[32][33];
  const int k = threadIdx.x & 31, l = threadIdx.x >> 5;   // 32 x 32 threads
  double acc = 0;
  for (int e0 = blockIdx.x * 32; e0 < 4 * N; e0 += gridDim.x * 32) {
    int e = e0 + l;
    rows[l][k] = (e < 4 * N && k < K) ? row_at(T, tl, e, k, K, tq) : 0.0;
    __syncthreads();
    if (k < K && l < K)
      for (int r = 0; r < 32; r++) acc += rows[r][k] * rows[r][l];
    __syncthreads();
  }
  if (k < K && l < K) Gp[(size_t)blockIdx.x * K * K + k * K + l] = acc;
}

__global__ void k_gram_sum(const double* __restrict__ Gp, int nblocks, int K, double* __restrict__ G) {
  const int e = threadIdx.x;
  if (e >= K * K) return;
  double s = 0;
  for (int b = 0; b < nblocks; b++) s += Gp[(size_t)b * K * K + e];
  G[e] = s;
}

// Cholesky G = R^T R (R upper) of one K x K Gram matrix by one warp, logs of
// diag(R) accumulated, Rinv = R^-1.  Right-looking on the warp's shared copy
// M: step j takes the square root of the pivot, scales row j, and lane c
// updates column c of the trailing upper triangle; then lane c solves
// R x = e_c by back substitution into column c of Q.
__device__ void chol_warp(const double* __restrict__ G, int K, double* __restrict__ Rinv,
                          double* __restrict__ logdiag, int accumulate, int* __restrict__ fail,
                          double (*M)[33], double (*Q)[33], int lane) {
  for (int a = 0; a < K; a++)
    if (lane < K) M[a][lane] = G[a * K + lane];
  __syncwarp();
  for (int j = 0; j < K; j++) {
    const double s = M[j][j];
    if (!(s > 0)) {                                 // the same value in every lane
      if (lane == 0) *fail = 1;
      return;
    }
    const double d = sqrt(s);
    __syncwarp();
    if (lane > j && lane < K) M[j][lane] /= d;
    if (lane == j) M[j][j] = d;
    __syncwarp();
    if (lane > j && lane < K) {
      const double rjc = M[j][lane];
      for (int a2 = j + 1; a2 <= lane; a2++) M[a2][lane] -= M[j][a2] * rjc;
    }
    __syncwarp();
  }
  if (accumulate && lane < K) logdiag[lane] += log(M[lane][lane]);
  if (lane < K) {
    for (int a2 = K - 1; a2 >= 0; a2--) {
      double v = (a2 == lane) ? 1.0 : 0.0;
      for (int p = a2 + 1; p < K; p++) v -= M[a2][p] * Q[p][lane];
      Q[a2][lane] = v / M[a2][a2];
    }
    for (int a2 = 0; a2 < K; a2++) Rinv[a2 * K + lane] = Q[a2][lane];
  }
  __syncwarp();
}

__global__ void __launch_bounds__(32) k_chol(const double* __restrict__ G, int K, double* __restrict__ Rinv,
                                             double* __restrict__ logdiag, int accumulate, int* __restrict__ fail) {
  __shared__ double M[32][33], Q[32][33];
  chol_warp(G, K, Rinv, logdiag, accumulate, fail, M, Q, threadIdx.x);
}

// T <- T' Rinv at the common time tq (every disk's tangent clock set to tq), one
// thread per row: its K values in registers (KM: their number rounded up), Rinv
// from shared memory, column k the sum over l <= k in order.  FP64 issue bounds
// it, so the lanes are 32 rows and the sums stop at the triangle.  (One thread
// per disk kept 128 values in local memory, and 1024 disks gave eight blocks:
// 200 us a pass, 22 so.)
constexpr int RINV_THREADS = 128;               // rows per block: whole disks to a warp
template <int KM>
__device__ __forceinline__ void apply_rinv_rows(double* T, double* tl, int N, int e, int K, double tq,
                                                const double* __restrict__ Rinv) {
  __shared__ double Rs[KM][KM];
  for (int q = threadIdx.x; q < KM * KM; q += RINV_THREADS)
    Rs[q / KM][q % KM] = q / KM < K && q % KM < K ? Rinv[(q / KM) * K + q % KM] : 0.0;
  __syncthreads();
  const bool on = e < 4 * N;
  double v[KM];
#pragma unroll
  for (int k = 0; k < KM; k++) v[k] = on && k < K ? row_at(T, tl, e, k, K, tq) : 0.0;
  __syncwarp();                                 // the disk's rows are read
#pragma unroll
  for (int k = 0; k < KM; k++) {
    double s = 0;
#pragma unroll
    for (int l = 0; l <= k; l++) s += v[l] * Rs[l][k];
    if (on && k < K) T[(size_t)e * K + k] = s;
  }
  if (on && (e & 3) == 0) tl[e >> 2] = tq;
}

template <int KM>
__global__ void __launch_bounds__(RINV_THREADS) k_apply_rinv(double* T, double* tl, int N, int K,
                                                             const double* __restrict__ tqp,
                                                             const double* __restrict__ Rinv) {
  apply_rinv_rows<KM>(T, tl, N, blockIdx.x * RINV_THREADS + threadIdx.x, K, *tqp, Rinv);
}

// ---------------------------------------------------------------- adjoint kernels

// One warp sweeps a log backwards, applying the transpose of the collision map
// and of the free flights between collisions.  A is [N][4]: (g_x, g_y, g_vx,
// g_vy) of each disk at its time ta[i].  Lanes hold the disk `lane & 1` and the
// axis `lane & 2` of a collision, so its chain of FP64 operations is one axis
// of one disk; masses and quotients come 32 collisions at a time.  (One thread
// per system: 3.5 us a collision; so 0.9.)
__device__ __forceinline__ void adjoint_warp(const edmd_log_entry* __restrict__ log, int64_t M,
                                             const Disk* __restrict__ d, double* A, double* ta, int lane, Coll* tile) {
  const bool odd = lane & 1, y = lane & 2;
  auto over_axes = [](double v) { return v + __shfl_xor_sync(0xffffffffu, v, 2); };
  for (int64_t n1 = M; n1 > 0; n1 -= 32) {
    const int cnt = (int)(n1 < 32 ? n1 : 32);
    __syncwarp();
    if (lane < cnt) tile[lane] = coll_of(log[n1 - 1 - lane], d);
    __syncwarp();
    for (int n = 0; n < cnt; n++) {
      const Coll& L = tile[n];
      const int me = odd ? L.j : L.i;
      const double r = y ? L.dy : L.dx, v = y ? L.dvy : L.dvx, mo = odd ? L.mi : L.mj;
      double* a = A + 4 * (size_t)me + (y ? 1 : 0);
      const double g = a[0];
      // transpose of the free flight from the collision to the disk's adjoint time
      const double gv = a[2] + g * (ta[me] - L.t);
      // w enters dv_i' with +m_j and dv_j' with -m_i
      const double pw = mo * gv, po = __shfl_xor_sync(0xffffffffu, pw, 1);
      const double gw = odd ? po - pw : pw - po;
      // dt_c enters the positions through -Dv dt_c
      const double D = (odd ? -L.f : L.f) * mo * r;
      const double q = over_axes(D * g), qo = __shfl_xor_sync(0xffffffffu, q, 1);
      double gdt = -(odd ? qo : q) - (odd ? q : qo);
      // w = df r + f drc, df = (f/rv) (v . drc + r . dv_ij)
      const double gdf = over_axes(r * gw);
      const double s = L.frv * gdf;
      const double grc = L.f * gw + s * v;
      const double gdv = s * r;
      // drc = dr_ij + v dt_c, dt_c = -(r . dr_ij)/rv
      gdt += over_axes(v * grc);
      const double gr = grc - div_rn(gdt, L.rv) * r;
      // dr_ij = dr_j - dr_i, dv_ij = dv_j - dv_i
      __syncwarp();
      if (lane < 4) {
        a[0] = g + flip(gr, !odd);
        a[2] = gv + flip(gdv, !odd);
        if (!y) ta[me] = L.t;
      }
      __syncwarp();
    }
  }
}

__global__ void __launch_bounds__(32) k_adjoint(const edmd_log_entry* __restrict__ log, int64_t M,
                                                const Disk* __restrict__ d, double* A, double* ta) {
  __shared__ Coll tile[32];
  adjoint_warp(log, M, d, A, ta, threadIdx.x, tile);
}

// every disk's adjoint brought back to t0 (transpose of the first free flight)
__global__ void k_adjoint_finish(int N, double* __restrict__ A, const double* __restrict__ ta, double t0) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  A[4 * i + 2] += A[4 * i + 0] * (ta[i] - t0);
  A[4 * i + 3] += A[4 * i + 1] * (ta[i] - t0);
}

__global__ void k_fill(double* p, int64_t n, double v) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// ---------------------------------------------------------------- batched kernels
// Every system of a context at once: system s owns the disks doff[s] ..
// doff[s] + N_s - 1 of the concatenated arrays and rows 4 doff[s] .. of T.

// system index of each disk
__global__ void k_disk_sys(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff, int nsys,
                           int32_t* __restrict__ dsys) {
  for (int s = blockIdx.y; s < nsys; s += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < sys[s].B.N; i += gridDim.x * blockDim.x)
      dsys[doff[s] + i] = s;
}

// every disk's clock set to its system's current time
__global__ void k_fill_sys_time(const SysDev* __restrict__ sys, const int32_t* __restrict__ dsys, int64_t TN,
                                double* __restrict__ tl) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < TN) tl[g] = sys[dsys[g]].st->t;
}

// one warp per system: the tangent map over its collisions logged from entry
// `from` to the chunk's end, nend[s]
__global__ void __launch_bounds__(32) k_tangent_apply_b(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff,
                                                        double* T, double* tl, int K, int64_t from,
                                                        const uint64_t* __restrict__ nend) {
  __shared__ Coll tile[32];
  const SysDev& S = sys[blockIdx.x];
  int64_t end = (int64_t)nend[blockIdx.x];
  if (end > S.log_cap) end = S.log_cap;
  const int64_t o = doff[blockIdx.x];
  tangent_apply_warp((const edmd_log_entry*)S.log + from, end - from, S.d, T + (size_t)4 * o * K, tl + o, K, threadIdx.x,
                     tile);
}

constexpr int GRAM_WARPS = 17;                  // warps of the 528 pairs of 32 columns
constexpr int GRAM_LOADS = 8;                   // elements of 32 rows a thread fetches: at least 4 K threads a block

// The Gram matrix of each system at its time tqs[s], one pair (k <= l) of
// columns per lane, the K (K + 1) / 2 pairs spread over the warps of gridDim.y
// blocks (deterministic: every pair sums its rows in index order).  FP64 issue
// bounds it: a warp per column left half its lanes idle and issued 32 columns'
// instructions for 16 (128 systems of 448 disks, 16 vectors: 665 us).
__global__ void __launch_bounds__(GRAM_WARPS * 32)
k_gram_b(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff, const double* __restrict__ T,
         const double* __restrict__ tl, int K, const double* __restrict__ tqs, double* __restrict__ G) {
  __shared__ double rows[32][33];
  const SysDev& S = sys[blockIdx.x];
  const int N = S.B.N;
  const double tq = tqs[blockIdx.x];            // the system's time at the end of the chunk
  const int64_t o = doff[blockIdx.x];
  const double* Ts = T + (size_t)4 * o * K;
  const double* tls = tl + o;
  const int p = blockIdx.y * blockDim.x + threadIdx.x, pairs = K * (K + 1) / 2;
  // pair p: l from the triangular root, k = p - l (l + 1) / 2
  int l = 0;
  while (l < K && (l + 1) * (l + 2) / 2 <= p) l++;
  const int k = p - l * (l + 1) / 2;
  const bool on = p < pairs;
  double acc = 0;
  // the next 32 rows are on their way while this thread's pair is summed: up
  // to GRAM_LOADS elements a thread, as (value, velocity row, time) still to be
  // flown to tq
  double x[GRAM_LOADS], v[GRAM_LOADS], t[GRAM_LOADS];
  auto fetch = [&](int e0) {
#pragma unroll
    for (int u = 0; u < GRAM_LOADS; u++) {
      const int q = threadIdx.x + u * blockDim.x, e = e0 + q / K, c = q % K;
      x[u] = v[u] = 0;
      t[u] = tq;
      if (q < 32 * K && e < 4 * N) {
        x[u] = Ts[(size_t)e * K + c];
        if ((e & 3) < 2) { v[u] = Ts[(size_t)(e + 2) * K + c]; t[u] = tls[e >> 2]; }
      }
    }
  };
  fetch(0);
  for (int e0 = 0; e0 < 4 * N; e0 += 32) {
#pragma unroll
    for (int u = 0; u < GRAM_LOADS; u++) {
      const int q = threadIdx.x + u * blockDim.x, r = q / K;
      if (q < 32 * K) rows[r][q % K] = (r & 3) < 2 ? x[u] + v[u] * (tq - t[u]) : x[u];
    }
    __syncthreads();
    fetch(e0 + 32);
    if (on)
#pragma unroll 8
      for (int r = 0; r < 32; r++) acc += rows[r][k] * rows[r][l];
    __syncthreads();
  }
  if (on) {
    G[(size_t)blockIdx.x * K * K + k * K + l] = acc;
    G[(size_t)blockIdx.x * K * K + l * K + k] = acc;
  }
}

// one warp per system
__global__ void __launch_bounds__(32) k_chol_b(const double* __restrict__ G, int nsys, int K,
                                               double* __restrict__ Rinv, double* __restrict__ logdiag,
                                               int accumulate, int* __restrict__ fail) {
  __shared__ double M[32][33], Q[32][33];
  const int s = blockIdx.x;
  if (s >= nsys) return;
  chol_warp(G + (size_t)s * K * K, K, Rinv + (size_t)s * K * K, logdiag + (size_t)s * K, accumulate, fail + s,
            M, Q, threadIdx.x);
}

template <int KM>
__global__ void __launch_bounds__(RINV_THREADS) k_apply_rinv_b(const SysDev* __restrict__ sys,
                                                               const int64_t* __restrict__ doff, double* T, double* tl,
                                                               int K, const double* __restrict__ tqs,
                                                               const double* __restrict__ Rinv) {
  const int s = blockIdx.y, N = sys[s].B.N;
  if ((int)blockIdx.x * RINV_THREADS >= 4 * N) return;
  const int64_t o = doff[s];
  apply_rinv_rows<KM>(T + (size_t)4 * o * K, tl + o, N, blockIdx.x * RINV_THREADS + threadIdx.x, K, tqs[s],
                      Rinv + (size_t)s * K * K);
}

// one warp per system: the transposed map backwards over its log
__global__ void __launch_bounds__(32) k_adjoint_b(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff,
                                                  double* A, double* ta) {
  __shared__ Coll tile[32];
  const SysDev& S = sys[blockIdx.x];
  int64_t M = (int64_t)S.st->nlog;
  if (M > S.log_cap) M = S.log_cap;
  adjoint_warp((const edmd_log_entry*)S.log, M, S.d, A + 4 * (size_t)doff[blockIdx.x], ta + doff[blockIdx.x], threadIdx.x,
               tile);
}

// every disk's position flown (virtually) to its system's current time
__global__ void k_positions_now_b(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff,
                                  const int32_t* __restrict__ dsys, int64_t TN, double* __restrict__ x,
                                  double* __restrict__ y) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= TN) return;
  const int s = dsys[g];
  const Disk p = sys[s].d[g - doff[s]];
  const double t = sys[s].st->t;
  x[g] = p.x + p.vx * (t - p.tl);
  y[g] = p.y + p.vy * (t - p.tl);
}

// one block per system: MSD = (1/N) sum |u_i - <u>|^2 of the minimum-image
// displacements u from (x0, y0) to (x1, y1), its gradient with respect to
// the final positions in A (velocity parts zero) and the direct term
// 2 (u_i - <u>) / N in (dux, duy); sums over disks by a fixed tree
__global__ void k_msd_b(const SysDev* __restrict__ sys, const int64_t* __restrict__ doff,
                        const double* __restrict__ x0, const double* __restrict__ y0,
                        const double* __restrict__ x1, const double* __restrict__ y1, double* __restrict__ A,
                        double* __restrict__ ta, double* __restrict__ dux, double* __restrict__ duy,
                        double* __restrict__ msd) {
  __shared__ double sx[256], sy[256];
  const SysDev& S = sys[blockIdx.x];
  const int N = S.B.N;
  const double Lx = S.B.Lx, Ly = S.B.Ly, T = S.st->t;
  const int64_t o = doff[blockIdx.x];
  auto disp = [&](int i, double* ux, double* uy) {
    double dx = x1[o + i] - x0[o + i], dy = y1[o + i] - y0[o + i];
    dx -= Lx * nearbyint(dx / Lx);
    dy -= Ly * nearbyint(dy / Ly);
    *ux = dx; *uy = dy;
  };
  double ax = 0, ay = 0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    double ux, uy;
    disp(i, &ux, &uy);
    ax += ux; ay += uy;
  }
  sx[threadIdx.x] = ax; sy[threadIdx.x] = ay;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) { sx[threadIdx.x] += sx[threadIdx.x + w]; sy[threadIdx.x] += sy[threadIdx.x + w]; }
    __syncthreads();
  }
  const double mx = sx[0] / N, my = sy[0] / N;
  __syncthreads();
  double acc = 0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    double ux, uy;
    disp(i, &ux, &uy);
    const double a = ux - mx, b = uy - my;
    acc += a * a + b * b;
    double* Ai = A + 4 * (o + i);
    Ai[0] = 2.0 * a / N; Ai[1] = 2.0 * b / N; Ai[2] = 0; Ai[3] = 0;
    dux[o + i] = 2.0 * a / N; duy[o + i] = 2.0 * b / N;
    ta[o + i] = T;
  }
  sx[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sx[threadIdx.x] += sx[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) msd[blockIdx.x] = sx[0] / N;
}

// every disk's adjoint brought back to its system's initial time t0[s]
__global__ void k_adjoint_finish_b(const int32_t* __restrict__ dsys, int64_t TN, double* __restrict__ A,
                                   const double* __restrict__ ta, const double* __restrict__ t0) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= TN) return;
  const double t = t0[dsys[g]];
  A[4 * g + 2] += A[4 * g + 0] * (ta[g] - t);
  A[4 * g + 3] += A[4 * g + 1] * (ta[g] - t);
}

__global__ void k_sys_times(const SysDev* __restrict__ sys, int nsys, double* __restrict__ t,
                            uint64_t* __restrict__ nend) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  t[s] = sys[s].st->t;
  if (nend) nend[s] = sys[s].st->nlog;
}

// a chunk logged from entry `from` on moves to the front of each log, where
// edmd_get_log reads it
__global__ void k_log_front(const SysDev* __restrict__ sys, int64_t from) {
  const SysDev& S = sys[blockIdx.x];
  edmd_log_entry* log = (edmd_log_entry*)S.log;
  const int64_t end = (int64_t)S.st->nlog < S.log_cap ? (int64_t)S.st->nlog : S.log_cap;
  for (int64_t e = from + threadIdx.x; e < end; e += blockDim.x) log[e - from] = log[e];
  __syncthreads();
  if (threadIdx.x == 0) S.st->nlog -= (uint64_t)from;
}

// every system's log written from entry n (or its saved length) on
__global__ void k_set_log(const SysDev* __restrict__ sys, int nsys, uint64_t n, const uint64_t* __restrict__ saved) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < nsys) sys[s].st->nlog = saved ? saved[s] : n;
}

// positions of one system flown (virtually) to time t, without touching the state
__global__ void k_positions_at(const Disk* __restrict__ d, int N, double t, double* __restrict__ x,
                               double* __restrict__ y) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  Disk p = d[i];
  x[i] = p.x + p.vx * (t - p.tl);
  y[i] = p.y + p.vy * (t - p.tl);
}

}  // namespace

// ==================================================================== log + checkpoints

static int upload_sysdev(edmd_ctx* ctx) {
  CK(cudaMemcpyAsync(ctx->ds, ctx->hs.data(), ctx->nsys * sizeof(SysDev), cudaMemcpyHostToDevice,
                     ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return EDMD_OK;
}

extern "C" int edmd_set_log_capacity(edmd_ctx* ctx, int64_t cap) {
  if (!ctx || cap < 0) return EDMD_ERR_ARG;
  if (cap > INT64_MAX / (int64_t)sizeof(edmd_log_entry) / ctx->nsys)   // its bytes are no number
    return set_err(ctx, EDMD_ERR_CUDA, "collision log: out of memory");
  if (cap > ctx->log_cap) {
    if (ctx->logbuf) cudaFree(ctx->logbuf);
    ctx->logbuf = nullptr;
    ctx->log_cap = 0;
    for (SysDev& S : ctx->hs) { S.log = nullptr; S.log_cap = 0; }
    CK(dalloc(&ctx->logbuf, (size_t)ctx->nsys * cap));
    ctx->log_cap = cap;
  }
  for (int s = 0; s < ctx->nsys; s++) {
    ctx->hs[s].log = ctx->logbuf + (size_t)s * ctx->log_cap;
    ctx->hs[s].log_cap = ctx->log_cap;
  }
  return upload_sysdev(ctx);
}

extern "C" int edmd_clear_log(edmd_ctx* ctx) {
  if (!ctx) return EDMD_ERR_ARG;
  k_set_log<<<(ctx->nsys + 127) / 128, 128, 0, ctx->stream>>>(ctx->ds, ctx->nsys, 0, nullptr);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(ctx->stream));
  return EDMD_OK;
}

extern "C" int edmd_get_log(edmd_ctx* ctx, int32_t s, edmd_log_entry* out, int64_t cap, int64_t* n) {
  if (!ctx || s < 0 || s >= ctx->nsys || !n) return EDMD_ERR_ARG;
  uint64_t nl = 0;
  CK(sync_copy(ctx, &nl, &ctx->st[s].nlog, 8, cudaMemcpyDeviceToHost));
  *n = (int64_t)nl;
  int64_t k = (int64_t)nl < cap ? (int64_t)nl : cap;
  if (k > ctx->log_cap) k = ctx->log_cap;
  if (out && k > 0)
    CK(sync_copy(ctx, out, ctx->hs[s].log, k * sizeof(edmd_log_entry), cudaMemcpyDeviceToHost));
  return (int64_t)nl > ctx->log_cap ? EDMD_ERR_CAPACITY : EDMD_OK;
}

// the arrays that make up the engine state of every system in the context
static void state_parts(edmd_ctx* ctx, std::vector<std::pair<void*, size_t>>& parts) {
  const size_t TN = ctx->total_N;
  size_t TE = 0, TT = 0;
  for (const SysDev& S : ctx->hs) {
    TE += 2 * (size_t)S.B.N + NSPECIAL;
    for (int h = 0; h < S.nlev; h++) TT += S.lev_cnt[h];
  }
  parts = {{ctx->d, TN * sizeof(Disk)}, {ctx->vr, TN * 8}, {ctx->cx, TN * 4}, {ctx->cy, TN * 4},
           {ctx->prv, TN * 4}, {ctx->crossX, TN * 4}, {ctx->crossY, TN * 4},
           {ctx->head, (size_t)ctx->total_C * 4}, {ctx->ev, TE * sizeof(Ev)}, {ctx->on, TE * 4},
           {ctx->op, TE * 4}, {ctx->tree, TT * sizeof(Node)}, {ctx->st, ctx->nsys * sizeof(SysState)}};
  if (ctx->cal) parts.push_back({ctx->cal, TN * CAL_SUB * CAL_LINE * 2});
  if (ctx->mask) parts.push_back({ctx->mask, TN * 2});
}

int ckpt_save(edmd_ctx* ctx, int32_t slot) {
  std::vector<std::pair<void*, size_t>> parts;
  state_parts(ctx, parts);
  size_t total = 0;
  for (auto& p : parts) total += align_up(p.second, 256);
  if ((int)ctx->ckpt.size() <= slot) ctx->ckpt.resize(slot + 1, nullptr);
  if ((int)ctx->ckpt_dirty.size() <= slot) ctx->ckpt_dirty.resize(slot + 1, 0);
  ctx->ckpt_dirty[slot] = ctx->round_dirty ? 1 : 0;
  if (!ctx->ckpt[slot]) CK(cudaMalloc(&ctx->ckpt[slot], total));
  char* dst = (char*)ctx->ckpt[slot];
  for (auto& p : parts) {
    CK(cudaMemcpyAsync(dst, p.first, p.second, cudaMemcpyDeviceToDevice, ctx->stream));
    dst += align_up(p.second, 256);
  }
  CK(cudaStreamSynchronize(ctx->stream));
  return EDMD_OK;
}

int ckpt_restore(edmd_ctx* ctx, int32_t slot) {
  if (slot >= (int)ctx->ckpt.size() || !ctx->ckpt[slot]) return EDMD_ERR_ARG;
  std::vector<std::pair<void*, size_t>> parts;
  state_parts(ctx, parts);
  const char* src = (const char*)ctx->ckpt[slot];
  for (auto& p : parts) {
    CK(cudaMemcpyAsync(p.first, src, p.second, cudaMemcpyDeviceToDevice, ctx->stream));
    src += align_up(p.second, 256);
  }
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->round_dirty = ctx->ckpt_dirty[slot] != 0;
  return EDMD_OK;
}

extern "C" int edmd_checkpoint_save(edmd_ctx* ctx, int32_t slot) {
  if (!ctx || slot < 0 || slot > CKPT_PUBLIC_MAX) return EDMD_ERR_ARG;
  return ckpt_save(ctx, slot);
}

extern "C" int edmd_checkpoint_restore(edmd_ctx* ctx, int32_t slot) {
  if (!ctx || slot < 0 || slot > CKPT_PUBLIC_MAX) return EDMD_ERR_ARG;
  return ckpt_restore(ctx, slot);
}

// ==================================================================== tangent driver

static int current_time(edmd_ctx* ctx, int s, double* t) {
  CK(sync_copy(ctx, t, &ctx->st[s].t, 8, cudaMemcpyDeviceToHost));
  return EDMD_OK;
}

// one advance of every system, logging collision geometry from entry `from` on,
// at most `room` entries a system; *longest: the longest log, or that of system
// s >= 0
static int advance_logged(edmd_ctx* ctx, int64_t ncoll, int64_t from, int64_t room, int s, int64_t* longest) {
  k_set_log<<<(ctx->nsys + 127) / 128, 128, 0, ctx->stream>>>(ctx->ds, ctx->nsys, (uint64_t)from, nullptr);
  CK(cudaGetLastError());
  int rc = edmd_advance(ctx, ncoll, INFINITY, EDMD_F_LOG | EDMD_F_COUNT_NORMAL, (int64_t)1 << 60, nullptr);
  if (rc) return rc;
  std::vector<uint64_t> nl(ctx->nsys);
  CK(sync_copy2d(ctx, nl.data(), 8, &ctx->st[0].nlog, sizeof(SysState), 8, ctx->nsys, cudaMemcpyDeviceToHost));
  int64_t most = 0;
  for (uint64_t v : nl) {
    const int64_t n = (int64_t)v - from;
    if (n > room) return set_err(ctx, EDMD_ERR_CAPACITY, "collision log overflow");
    most = n > most ? n : most;
  }
  if (longest) *longest = s >= 0 ? (int64_t)nl[s] - from : most;
  return EDMD_OK;
}

// The gradient drivers log the collisions of the whole call (one forward run)
// where that takes no more memory than the checkpoints and the segment's log of
// a run in segments of ckpt_every, or at most LOG_FREE_BYTES, and never more
// than LOG_ALL_BYTES; else they run in segments (twice as long).  The log stays
// with the context, as the checkpoints do.
constexpr int64_t LOG_ALL_BYTES = (int64_t)2 << 30, LOG_FREE_BYTES = (int64_t)64 << 20;
static bool log_whole(edmd_ctx* ctx, int64_t n_coll, int64_t ckpt_every) {
  std::vector<std::pair<void*, size_t>> parts;
  state_parts(ctx, parts);
  double state = 0;
  for (auto& p : parts) state += (double)align_up(p.second, 256);
  const double entry = (double)sizeof(edmd_log_entry) * ctx->nsys, all = entry * (n_coll + 16.0);
  const double segments = entry * (ckpt_every + 16.0) + state * (double)((n_coll - 1) / ckpt_every + 2);
  return all <= (double)LOG_ALL_BYTES && all <= std::max((double)LOG_FREE_BYTES, segments);
}

// log lengths put back at the end of a call
struct LogLengths {
  edmd_ctx* ctx;
  uint64_t* saved = nullptr;
  explicit LogLengths(edmd_ctx* c) : ctx(c) {}
  cudaError_t save() {
    cudaError_t e = dalloc(&saved, ctx->nsys);
    return e != cudaSuccess ? e : cudaMemcpy2DAsync(saved, 8, &ctx->st[0].nlog, sizeof(SysState), 8, ctx->nsys,
                                                    cudaMemcpyDeviceToDevice, ctx->stream);
  }
  ~LogLengths() {
    if (!saved) return;
    k_set_log<<<(ctx->nsys + 127) / 128, 128, 0, ctx->stream>>>(ctx->ds, ctx->nsys, 0, saved);
    cudaStreamSynchronize(ctx->stream);
    cudaFree(saved);
  }
};

// What a tangent driver's chunks alternate between: two halves of the logs and
// the chunk's end times and log ends.  The tangent map and the QR of a chunk
// run on a second stream beside the next chunk's forward run; the forward run
// after that waits until the map has read the half it is going to write (one
// half: see chunk_logs).
struct Chunks {
  double* tq[2] = {nullptr, nullptr};
  uint64_t* nend[2] = {nullptr, nullptr};
  cudaEvent_t ran[2] = {nullptr, nullptr}, mapped[2] = {nullptr, nullptr};
  ~Chunks() {
    for (int k = 0; k < 2; k++) {
      if (tq[k]) cudaFree(tq[k]);
      if (nend[k]) cudaFree(nend[k]);
      if (ran[k]) cudaEventDestroy(ran[k]);
      if (mapped[k]) cudaEventDestroy(mapped[k]);
    }
  }
  cudaError_t make(int nsys) {
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 2 && e == cudaSuccess; k++) {
      e = dalloc(&tq[k], nsys);
      if (e == cudaSuccess) e = dalloc(&nend[k], nsys);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ran[k], cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&mapped[k], cudaEventDisableTiming);
    }
    return e;
  }
};

// Logs of two halves for a run of several chunks; of one where there is no room
// for two: a chunk's forward run then waits for the map of the one before.
static int chunk_logs(edmd_ctx* ctx, int64_t half, bool several, bool* two) {
  *two = several && half <= INT64_MAX / 2 && edmd_set_log_capacity(ctx, 2 * half) == EDMD_OK;
  if (*two) return EDMD_OK;
  cudaGetLastError();
  return edmd_set_log_capacity(ctx, half);
}

// The last chunk's collisions at the front of the logs when a run ends, also by
// an error (declared before what waits for the second stream).
struct LastChunk {
  edmd_ctx* ctx;
  int64_t from = 0;
  ~LastChunk() {
    if (from) k_log_front<<<ctx->nsys, 128, 0, ctx->stream>>>(ctx->ds, from);
  }
};

constexpr int GRAM_BLOCKS = 1024;

// CholQR2 of one system's tangent block at the time *tqp, on stream st
static int cholqr(edmd_ctx* ctx, double* T, double* tl, int N, int K, const double* tqp, double* G, double* Gp,
                  double* Rinv, double* logdiag, int* fail, bool accumulate, cudaStream_t st) {
  for (int pass = 0; pass < 2; pass++) {    // CholQR2: the second pass restores orthogonality
    int blocks = (4 * N + 31) / 32;
    if (blocks > GRAM_BLOCKS) blocks = GRAM_BLOCKS;
    k_gram<<<blocks, 1024, 0, st>>>(T, tl, N, K, tqp, Gp);
    k_gram_sum<<<1, 1024, 0, st>>>(Gp, blocks, K, G);
    k_chol<<<1, 32, 0, st>>>(G, K, Rinv, logdiag, accumulate ? 1 : 0, fail);
    const int rb = (4 * N + RINV_THREADS - 1) / RINV_THREADS;
    if (K <= 16) k_apply_rinv<16><<<rb, RINV_THREADS, 0, st>>>(T, tl, N, K, tqp, Rinv);
    else k_apply_rinv<32><<<rb, RINV_THREADS, 0, st>>>(T, tl, N, K, tqp, Rinv);
    CK(cudaGetLastError());
  }
  return EDMD_OK;
}

extern "C" int edmd_tangent_run(edmd_ctx* ctx, int32_t s, int32_t K, int64_t n_coll, int64_t qr_every,
                                uint64_t seed, double* tangent_io, double* lyap_out) {
  if (!ctx || s < 0 || s >= ctx->nsys || K < 1 || K > 32 || n_coll < 0 || qr_every < 0)
    return EDMD_ERR_ARG;
  if (ctx->engine != EDMD_ENGINE_WARP) return set_err(ctx, EDMD_ERR_ARG, "tangents need the warp engine");
  const int N = ctx->hs[s].B.N;
  const int64_t most = n_coll > 0 ? n_coll : 1;
  const int64_t chunk = qr_every > 0 && qr_every < most ? qr_every : most;
  const int64_t half = chunk + 16;
  double *T = nullptr, *tl = nullptr, *G = nullptr, *Gp = nullptr, *Rinv = nullptr, *logdiag = nullptr;
  int* fail = nullptr;
  CK(dalloc(&T, (size_t)4 * N * K));
  CK(dalloc(&tl, N));
  CK(dalloc(&G, K * K));
  CK(dalloc(&Gp, (size_t)GRAM_BLOCKS * K * K));
  CK(dalloc(&Rinv, K * K));
  CK(dalloc(&logdiag, K));
  CK(dalloc(&fail, 1));
  struct Free { void* p[7]; ~Free() { for (void* q : p) if (q) cudaFree(q); } } guard{{T, tl, G, Gp, Rinv, logdiag, fail}};
  Chunks ch;
  CK(ch.make(1));
  bool two = false;
  int rc = chunk_logs(ctx, half, n_coll > chunk, &two);
  if (rc) return rc;
  if (!ctx->stream2) CK(cudaStreamCreateWithFlags(&ctx->stream2, cudaStreamNonBlocking));
  cudaStream_t st2 = ctx->stream2;
  LastChunk last{ctx};
  struct Idle { edmd_ctx* c; ~Idle() { cudaStreamSynchronize(c->stream2); } } idle{ctx};   // before the frees
  CK(call_begin(ctx));
  double t0;
  if ((rc = current_time(ctx, s, &t0))) return rc;
  // initial vectors: the caller's ([K][N][4]) or seeded random orthonormal ones
  std::vector<double> h((size_t)4 * N * K);
  if (tangent_io) {
    for (int k = 0; k < K; k++)
      for (int e = 0; e < 4 * N; e++) h[(size_t)e * K + k] = tangent_io[(size_t)k * 4 * N + e];
  } else {
    std::mt19937_64 g(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    for (auto& v : h) v = nd(g);
  }
  CK(cudaMemcpyAsync(T, h.data(), h.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  k_fill<<<(N + 255) / 256, 256, 0, ctx->stream>>>(tl, N, t0);
  CK(cudaMemsetAsync(logdiag, 0, K * sizeof(double), ctx->stream));
  CK(cudaMemsetAsync(fail, 0, 4, ctx->stream));
  k_sys_times<<<1, 32, 0, ctx->stream>>>(ctx->ds + s, 1, ch.tq[0], nullptr);
  if (!tangent_io &&
      (rc = cholqr(ctx, T, tl, N, K, ch.tq[0], G, Gp, Rinv, logdiag, fail, false, ctx->stream)))
    return rc;
  // the tangent vectors are the second stream's from here on
  CK(cudaEventRecord(ch.ran[0], ctx->stream));
  CK(cudaStreamWaitEvent(st2, ch.ran[0], 0));
  int64_t done = 0;
  for (int c = 0; done < n_coll; c ^= 1) {
    int64_t want = n_coll - done < chunk ? n_coll - done : chunk;
    int64_t nl = 0;
    const int64_t from = two && c ? half : 0;
    if (done > (two ? chunk : 0)) CK(cudaStreamWaitEvent(ctx->stream, ch.mapped[two ? c : c ^ 1], 0));
    last.from = from;
    if ((rc = advance_logged(ctx, want, from, half, s, &nl))) return rc;
    k_sys_times<<<1, 32, 0, ctx->stream>>>(ctx->ds + s, 1, ch.tq[c], nullptr);
    CK(cudaEventRecord(ch.ran[c], ctx->stream));
    CK(cudaStreamWaitEvent(st2, ch.ran[c], 0));
    k_tangent_apply<<<1, 32, 0, st2>>>((const edmd_log_entry*)ctx->hs[s].log + from, nl, ctx->hs[s].d, T, tl, K);
    CK(cudaGetLastError());
    if (qr_every > 0 && (rc = cholqr(ctx, T, tl, N, K, ch.tq[c], G, Gp, Rinv, logdiag, fail, true, st2))) return rc;
    CK(cudaEventRecord(ch.mapped[c], st2));
    done += want;
    if (nl < want) break;     // the run ended early (tmax or t_stop)
  }
  CK(cudaEventRecord(ch.ran[0], st2));
  CK(cudaStreamWaitEvent(ctx->stream, ch.ran[0], 0));
  {
    int hf = 0;
    CK(sync_copy(ctx, &hf, fail, 4, cudaMemcpyDeviceToHost));
    if (hf) return set_err(ctx, EDMD_ERR_ARG, "tangent vectors became linearly dependent");
  }
  double t = t0;
  if ((rc = current_time(ctx, s, &t))) return rc;
  if (lyap_out) {
    std::vector<double> ld(K);
    CK(sync_copy(ctx, ld.data(), logdiag, K * 8, cudaMemcpyDeviceToHost));
    for (int k = 0; k < K; k++) lyap_out[k] = (t > t0) ? ld[k] / (t - t0) : 0.0;
  }
  if (tangent_io) {
    // tangents at the final time (virtual flight of every row)
    CK(sync_copy(ctx, h.data(), T, h.size() * 8, cudaMemcpyDeviceToHost));
    std::vector<double> htl(N);
    CK(sync_copy(ctx, htl.data(), tl, N * 8, cudaMemcpyDeviceToHost));
    for (int k = 0; k < K; k++)
      for (int i = 0; i < N; i++)
        for (int c = 0; c < 4; c++) {
          double v = h[(size_t)(4 * i + c) * K + k];
          if (c < 2) v += h[(size_t)(4 * i + c + 2) * K + k] * (t - htl[i]);
          tangent_io[(size_t)k * 4 * N + 4 * i + c] = v;
        }
  }
  CK(call_end(ctx));
  return EDMD_OK;
}

// ==================================================================== adjoint driver

extern "C" int edmd_msd_gradient(edmd_ctx* ctx, int32_t s, int64_t n_coll, int64_t ckpt_every,
                                 double t_obs, double* msd_out, double* g_vx, double* g_vy,
                                 double* g_x, double* g_y) {
  if (!ctx || s < 0 || s >= ctx->nsys || n_coll < 1 || ckpt_every < 1) return EDMD_ERR_ARG;
  if (ctx->engine != EDMD_ENGINE_WARP) return set_err(ctx, EDMD_ERR_ARG, "adjoints need the warp engine");
  ckpt_every = std::min(ckpt_every, n_coll);
  const int N = ctx->hs[s].B.N;
  const double Lx = ctx->hs[s].B.Lx, Ly = ctx->hs[s].B.Ly;
  // one logged forward run, or checkpointed segments run twice
  bool whole = log_whole(ctx, n_coll, ckpt_every);
  int rc = whole ? edmd_set_log_capacity(ctx, n_coll + 16) : EDMD_OK;
  if (rc) { whole = false; cudaGetLastError(); }         // no room for it
  if (!whole) rc = edmd_set_log_capacity(ctx, ckpt_every + 16);
  if (rc) return rc;
  LogLengths lengths(ctx);
  CK(lengths.save());
  int64_t nlog_all = 0;
  double *A = nullptr, *ta = nullptr, *px = nullptr, *py = nullptr;
  CK(dalloc(&A, 4 * (size_t)N));
  CK(dalloc(&ta, N));
  CK(dalloc(&px, N));
  CK(dalloc(&py, N));
  struct Free { void* p[4]; ~Free() { for (void* q : p) if (q) cudaFree(q); } } guard{{A, ta, px, py}};
  CK(call_begin(ctx));
  double t0, T;
  if ((rc = current_time(ctx, s, &t0))) return rc;
  std::vector<double> x0(N), y0(N), x1(N), y1(N);
  k_positions_at<<<(N + 127) / 128, 128, 0, ctx->stream>>>(ctx->hs[s].d, N, t0, px, py);
  CK(cudaMemcpyAsync(x0.data(), px, N * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaMemcpyAsync(y0.data(), py, N * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  // forward sweep: exact engine checkpoints at every segment boundary
  const int64_t nseg = whole ? 0 : (n_coll + ckpt_every - 1) / ckpt_every;
  std::vector<int64_t> seglen(nseg);
  if (whole && (rc = advance_logged(ctx, n_coll, 0, n_coll + 16, s, &nlog_all))) return rc;
  for (int64_t g = 0; g < nseg; g++) {
    if ((rc = edmd_checkpoint_save(ctx, (int32_t)g))) return rc;
    seglen[g] = (g == nseg - 1) ? n_coll - g * ckpt_every : ckpt_every;
    rc = edmd_advance(ctx, seglen[g], INFINITY, EDMD_F_COUNT_NORMAL, (int64_t)1 << 60, nullptr);
    if (rc) return rc;
  }
  if (!whole && (rc = edmd_checkpoint_save(ctx, (int32_t)nseg))) return rc;
  if ((rc = current_time(ctx, s, &T))) return rc;
  if (t_obs >= 0) {
    if (t_obs < T) return set_err(ctx, EDMD_ERR_ARG, "t_obs precedes the last processed event");
    T = t_obs;
  }
  k_positions_at<<<(N + 127) / 128, 128, 0, ctx->stream>>>(ctx->hs[s].d, N, T, px, py);
  CK(cudaMemcpyAsync(x1.data(), px, N * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaMemcpyAsync(y1.data(), py, N * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  // MSD = (1/N) sum |u_i - mean(u)|^2, u = minimum-image displacement
  std::vector<double> ux(N), uy(N);
  double mx = 0, my = 0;
  for (int i = 0; i < N; i++) {
    double dx = x1[i] - x0[i], dy = y1[i] - y0[i];
    dx -= Lx * std::nearbyint(dx / Lx);
    dy -= Ly * std::nearbyint(dy / Ly);
    ux[i] = dx; uy[i] = dy; mx += dx; my += dy;
  }
  mx /= N; my /= N;
  double msd = 0;
  std::vector<double> hA(4 * (size_t)N, 0.0);
  for (int i = 0; i < N; i++) {
    double a = ux[i] - mx, b = uy[i] - my;
    msd += a * a + b * b;
    hA[4 * i + 0] = 2.0 * a / N;
    hA[4 * i + 1] = 2.0 * b / N;
  }
  msd /= N;
  CK(cudaMemcpyAsync(A, hA.data(), hA.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  k_fill<<<(N + 255) / 256, 256, 0, ctx->stream>>>(ta, N, T);
  // reverse sweep over the log; else recompute each segment from its checkpoint, then its adjoint
  const edmd_log_entry* const log = (const edmd_log_entry*)ctx->hs[s].log;
  if (whole) k_adjoint<<<1, 32, 0, ctx->stream>>>(log, nlog_all, ctx->hs[s].d, A, ta);
  for (int64_t g = nseg - 1; g >= 0; g--) {
    if ((rc = edmd_checkpoint_restore(ctx, (int32_t)g))) return rc;
    int64_t nl = 0;
    if ((rc = advance_logged(ctx, seglen[g], 0, ckpt_every + 16, s, &nl))) return rc;
    k_adjoint<<<1, 32, 0, ctx->stream>>>(log, nl, ctx->hs[s].d, A, ta);
  }
  CK(cudaGetLastError());
  k_adjoint_finish<<<(N + 127) / 128, 128, 0, ctx->stream>>>(N, A, ta, t0);
  CK(cudaMemcpyAsync(hA.data(), A, hA.size() * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  // leave the engine at the end of the run
  if (!whole && (rc = edmd_checkpoint_restore(ctx, (int32_t)nseg))) return rc;
  // u = r(t) - r(0) also depends on the initial positions directly
  for (int i = 0; i < N; i++) {
    if (g_x) g_x[i] = hA[4 * i + 0] - 2.0 * (ux[i] - mx) / N;
    if (g_y) g_y[i] = hA[4 * i + 1] - 2.0 * (uy[i] - my) / N;
    if (g_vx) g_vx[i] = hA[4 * i + 2];
    if (g_vy) g_vy[i] = hA[4 * i + 3];
  }
  if (msd_out) *msd_out = msd;
  CK(call_end(ctx));
  return EDMD_OK;
}

// ==================================================================== batched drivers

namespace {

// device arrays every batched driver needs: each system's first disk and each
// disk's system; freed with the scope
struct BatchIndex {
  int64_t* doff = nullptr;
  int32_t* dsys = nullptr;
  ~BatchIndex() {
    if (doff) cudaFree(doff);
    if (dsys) cudaFree(dsys);
  }
};

int batch_index(edmd_ctx* ctx, BatchIndex& bi) {
  CK(dalloc(&bi.doff, ctx->nsys));
  CK(dalloc(&bi.dsys, ctx->total_N));
  CK(cudaMemcpyAsync(bi.doff, ctx->disk_off.data(), ctx->nsys * sizeof(int64_t), cudaMemcpyHostToDevice,
                     ctx->stream));
  dim3 g((unsigned)((ctx->maxN + 255) / 256), (unsigned)(ctx->nsys < 65535 ? ctx->nsys : 65535));
  k_disk_sys<<<g, 256, 0, ctx->stream>>>(ctx->ds, bi.doff, ctx->nsys, bi.dsys);
  CK(cudaGetLastError());
  return EDMD_OK;
}

// CholQR2 of every system's tangent block at the times tqs, on stream st
int cholqr_b(edmd_ctx* ctx, const BatchIndex& bi, double* T, double* tl, int K, double* G, double* Rinv,
             double* logdiag, int* fail, bool accumulate, const double* tqs, cudaStream_t st) {
  // all pairs of a system in one block, or (fewer systems than SMs) spread over blocks
  int dev = 0, nsm = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int pair_warps = (K * (K + 1) / 2 + 31) / 32, split = std::max(1, std::min(pair_warps, nsm / ctx->nsys));
  const int warps = std::max((pair_warps + split - 1) / split, (4 * K + 31) / 32);
  for (int pass = 0; pass < 2; pass++) {    // CholQR2: the second pass restores orthogonality
    k_gram_b<<<dim3(ctx->nsys, (pair_warps + warps - 1) / warps), 32 * warps, 0, st>>>(ctx->ds, bi.doff, T, tl, K, tqs, G);
    k_chol_b<<<ctx->nsys, 32, 0, st>>>(G, ctx->nsys, K, Rinv, logdiag, accumulate ? 1 : 0, fail);
    const dim3 rb((4 * ctx->maxN + RINV_THREADS - 1) / RINV_THREADS, ctx->nsys);
    if (K <= 16) k_apply_rinv_b<16><<<rb, RINV_THREADS, 0, st>>>(ctx->ds, bi.doff, T, tl, K, tqs, Rinv);
    else k_apply_rinv_b<32><<<rb, RINV_THREADS, 0, st>>>(ctx->ds, bi.doff, T, tl, K, tqs, Rinv);
    CK(cudaGetLastError());
  }
  return EDMD_OK;
}

int check_fail(edmd_ctx* ctx, const int* fail) {
  std::vector<int> h(ctx->nsys);
  CK(sync_copy(ctx, h.data(), fail, ctx->nsys * sizeof(int), cudaMemcpyDeviceToHost));
  for (int s = 0; s < ctx->nsys; s++)
    if (h[s]) return set_err(ctx, EDMD_ERR_ARG, "tangent vectors of system " + std::to_string(s) +
                                                    " became linearly dependent");
  return EDMD_OK;
}

int sys_times(edmd_ctx* ctx, double* host) {
  CK(sync_copy2d(ctx, host, 8, &ctx->st[0].t, sizeof(SysState), 8, ctx->nsys, cudaMemcpyDeviceToHost));
  return EDMD_OK;
}

}  // namespace

extern "C" int edmd_tangent_run_batch(edmd_ctx* ctx, int32_t K, int64_t n_coll, int64_t qr_every, uint64_t seed,
                                      double* lyap_out) {
  if (!ctx || K < 1 || K > 32 || n_coll < 0 || qr_every < 0) return EDMD_ERR_ARG;
  if (ctx->engine != EDMD_ENGINE_WARP) return set_err(ctx, EDMD_ERR_ARG, "tangents need the warp engine");
  const int64_t TN = ctx->total_N;
  const int nsys = ctx->nsys;
  const int64_t most = n_coll > 0 ? n_coll : 1;
  const int64_t chunk = qr_every > 0 && qr_every < most ? qr_every : most;
  const int64_t half = chunk + 16;
  int rc = EDMD_OK;
  BatchIndex bi;
  if ((rc = batch_index(ctx, bi))) return rc;
  double *T = nullptr, *tl = nullptr, *G = nullptr, *Rinv = nullptr, *logdiag = nullptr;
  int* fail = nullptr;
  CK(dalloc(&T, (size_t)4 * TN * K));
  CK(dalloc(&tl, TN));
  CK(dalloc(&G, (size_t)nsys * K * K));
  CK(dalloc(&Rinv, (size_t)nsys * K * K));
  CK(dalloc(&logdiag, (size_t)nsys * K));
  CK(dalloc(&fail, nsys));
  struct Free { void* p[6]; ~Free() { for (void* q : p) if (q) cudaFree(q); } } guard{{T, tl, G, Rinv, logdiag, fail}};
  Chunks ch;
  CK(ch.make(nsys));
  bool two = false;
  if ((rc = chunk_logs(ctx, half, n_coll > chunk, &two))) return rc;
  if (!ctx->stream2) CK(cudaStreamCreateWithFlags(&ctx->stream2, cudaStreamNonBlocking));
  cudaStream_t st2 = ctx->stream2;
  LastChunk last{ctx};
  struct Idle { edmd_ctx* c; ~Idle() { cudaStreamSynchronize(c->stream2); } } idle{ctx};   // before the frees
  const unsigned gs = (unsigned)((nsys + 127) / 128);
  // system s starts from the vectors edmd_tangent_run draws from seed + s
  // (drawn on the host before the timed part of the call)
  // systems are drawn on host threads, each from its own generator (128 systems
  // of 448 disks, 16 vectors: 40 ms on one thread)
  const size_t nh = (size_t)4 * TN * K;
  std::unique_ptr<double[]> h(new double[nh]);
  {
    std::atomic<int> next{0};
    run_threads(std::min(nsys, host_threads((int64_t)nh, 1 << 14)), [&](int) {
      for (int s = next++; s < nsys; s = next++) {
        std::mt19937_64 g(seed + (uint64_t)s);
        std::normal_distribution<double> nd(0.0, 1.0);
        double* hs = h.get() + (size_t)4 * ctx->disk_off[s] * K;
        for (size_t e = 0; e < (size_t)4 * ctx->hs[s].B.N * K; e++) hs[e] = nd(g);
      }
    });
  }
  CK(call_begin(ctx));
  std::vector<double> t0(nsys), t1(nsys);
  if ((rc = sys_times(ctx, t0.data()))) return rc;
  CK(host_copies(ctx, {{h.get(), T, (int64_t)nh * 8}}, true));
  k_fill_sys_time<<<(unsigned)((TN + 255) / 256), 256, 0, ctx->stream>>>(ctx->ds, bi.dsys, TN, tl);
  CK(cudaMemsetAsync(logdiag, 0, (size_t)nsys * K * sizeof(double), ctx->stream));
  CK(cudaMemsetAsync(fail, 0, nsys * sizeof(int), ctx->stream));
  k_sys_times<<<gs, 128, 0, ctx->stream>>>(ctx->ds, nsys, ch.tq[0], nullptr);
  if ((rc = cholqr_b(ctx, bi, T, tl, K, G, Rinv, logdiag, fail, false, ch.tq[0], ctx->stream))) return rc;
  // the tangent vectors are the second stream's from here on
  CK(cudaEventRecord(ch.ran[0], ctx->stream));
  CK(cudaStreamWaitEvent(st2, ch.ran[0], 0));
  int64_t done = 0;
  for (int c = 0; done < n_coll; c ^= 1) {
    const int64_t want = n_coll - done < chunk ? n_coll - done : chunk;
    const int64_t from = two && c ? half : 0;
    if (done > (two ? chunk : 0)) CK(cudaStreamWaitEvent(ctx->stream, ch.mapped[two ? c : c ^ 1], 0));
    last.from = from;
    if ((rc = advance_logged(ctx, want, from, half, -1, nullptr))) return rc;
    k_sys_times<<<gs, 128, 0, ctx->stream>>>(ctx->ds, nsys, ch.tq[c], ch.nend[c]);   // the chunk's end
    CK(cudaEventRecord(ch.ran[c], ctx->stream));
    CK(cudaStreamWaitEvent(st2, ch.ran[c], 0));
    k_tangent_apply_b<<<nsys, 32, 0, st2>>>(ctx->ds, bi.doff, T, tl, K, from, ch.nend[c]);
    CK(cudaGetLastError());
    if (qr_every > 0 && (rc = cholqr_b(ctx, bi, T, tl, K, G, Rinv, logdiag, fail, true, ch.tq[c], st2))) return rc;
    CK(cudaEventRecord(ch.mapped[c], st2));
    done += want;
  }
  CK(cudaEventRecord(ch.ran[0], st2));
  CK(cudaStreamWaitEvent(ctx->stream, ch.ran[0], 0));
  if ((rc = check_fail(ctx, fail))) return rc;
  if (lyap_out) {
    std::vector<double> ld((size_t)nsys * K);
    CK(sync_copy(ctx, ld.data(), logdiag, ld.size() * 8, cudaMemcpyDeviceToHost));
    if ((rc = sys_times(ctx, t1.data()))) return rc;
    for (int s = 0; s < nsys; s++)
      for (int k = 0; k < K; k++)
        lyap_out[(size_t)s * K + k] = (t1[s] > t0[s]) ? ld[(size_t)s * K + k] / (t1[s] - t0[s]) : 0.0;
  }
  CK(call_end(ctx));
  return EDMD_OK;
}

extern "C" int edmd_msd_gradient_batch(edmd_ctx* ctx, int64_t n_coll, int64_t ckpt_every, double* msd_out,
                                       double* g_vx, double* g_vy, double* g_x, double* g_y) {
  if (!ctx || n_coll < 1 || ckpt_every < 1) return EDMD_ERR_ARG;
  if (ctx->engine != EDMD_ENGINE_WARP) return set_err(ctx, EDMD_ERR_ARG, "adjoints need the warp engine");
  ckpt_every = std::min(ckpt_every, n_coll);
  const int64_t TN = ctx->total_N;
  const int nsys = ctx->nsys;
  // one logged forward run, or checkpointed segments run twice
  bool whole = log_whole(ctx, n_coll, ckpt_every);
  int rc = whole ? edmd_set_log_capacity(ctx, n_coll + 16) : EDMD_OK;
  if (rc) { whole = false; cudaGetLastError(); }         // no room for it
  if (!whole) rc = edmd_set_log_capacity(ctx, ckpt_every + 16);
  if (rc) return rc;
  LogLengths lengths(ctx);
  CK(lengths.save());
  BatchIndex bi;
  if ((rc = batch_index(ctx, bi))) return rc;
  double *A = nullptr, *ta = nullptr, *x0 = nullptr, *y0 = nullptr, *x1 = nullptr, *y1 = nullptr;
  double *dux = nullptr, *duy = nullptr, *t0 = nullptr, *msd = nullptr;
  CK(dalloc(&A, 4 * (size_t)TN));
  CK(dalloc(&ta, TN)); CK(dalloc(&x0, TN)); CK(dalloc(&y0, TN)); CK(dalloc(&x1, TN)); CK(dalloc(&y1, TN));
  CK(dalloc(&dux, TN)); CK(dalloc(&duy, TN)); CK(dalloc(&t0, nsys)); CK(dalloc(&msd, nsys));
  struct Free { void* p[10]; ~Free() { for (void* q : p) if (q) cudaFree(q); } }
      guard{{A, ta, x0, y0, x1, y1, dux, duy, t0, msd}};
  CK(call_begin(ctx));
  const unsigned gT = (unsigned)((TN + 127) / 128);
  k_sys_times<<<(nsys + 127) / 128, 128, 0, ctx->stream>>>(ctx->ds, nsys, t0, nullptr);
  k_positions_now_b<<<gT, 128, 0, ctx->stream>>>(ctx->ds, bi.doff, bi.dsys, TN, x0, y0);
  CK(cudaGetLastError());
  // forward sweep: exact engine checkpoints at every segment boundary
  const int64_t nseg = whole ? 0 : (n_coll + ckpt_every - 1) / ckpt_every;
  std::vector<int64_t> seglen(nseg);
  if (whole && (rc = advance_logged(ctx, n_coll, 0, n_coll + 16, -1, nullptr))) return rc;
  for (int64_t g = 0; g < nseg; g++) {
    if ((rc = edmd_checkpoint_save(ctx, (int32_t)g))) return rc;
    seglen[g] = (g == nseg - 1) ? n_coll - g * ckpt_every : ckpt_every;
    rc = edmd_advance(ctx, seglen[g], INFINITY, EDMD_F_COUNT_NORMAL, (int64_t)1 << 60, nullptr);
    if (rc) return rc;
  }
  if (!whole && (rc = edmd_checkpoint_save(ctx, (int32_t)nseg))) return rc;
  k_positions_now_b<<<gT, 128, 0, ctx->stream>>>(ctx->ds, bi.doff, bi.dsys, TN, x1, y1);
  k_msd_b<<<nsys, 256, 0, ctx->stream>>>(ctx->ds, bi.doff, x0, y0, x1, y1, A, ta, dux, duy, msd);
  CK(cudaGetLastError());
  // reverse sweep over the logs; else recompute each segment from its checkpoint, then its adjoint
  if (whole) k_adjoint_b<<<nsys, 32, 0, ctx->stream>>>(ctx->ds, bi.doff, A, ta);
  for (int64_t g = nseg - 1; g >= 0; g--) {
    if ((rc = edmd_checkpoint_restore(ctx, (int32_t)g))) return rc;
    if ((rc = advance_logged(ctx, seglen[g], 0, ckpt_every + 16, -1, nullptr))) return rc;
    k_adjoint_b<<<nsys, 32, 0, ctx->stream>>>(ctx->ds, bi.doff, A, ta);
  }
  CK(cudaGetLastError());
  k_adjoint_finish_b<<<gT, 128, 0, ctx->stream>>>(bi.dsys, TN, A, ta, t0);
  CK(cudaGetLastError());
  // leave the engine at the end of the run
  if (!whole && (rc = edmd_checkpoint_restore(ctx, (int32_t)nseg))) return rc;
  std::vector<double> hA(4 * (size_t)TN), hx(TN), hy(TN);
  CK(sync_copy(ctx, hA.data(), A, hA.size() * 8, cudaMemcpyDeviceToHost));
  CK(sync_copy(ctx, hx.data(), dux, TN * 8, cudaMemcpyDeviceToHost));
  CK(sync_copy(ctx, hy.data(), duy, TN * 8, cudaMemcpyDeviceToHost));
  if (msd_out) CK(sync_copy(ctx, msd_out, msd, nsys * 8, cudaMemcpyDeviceToHost));
  // u = r(t) - r(0) also depends on the initial positions directly
  for (int64_t g = 0; g < TN; g++) {
    if (g_x) g_x[g] = hA[4 * g + 0] - hx[g];
    if (g_y) g_y[g] = hA[4 * g + 1] - hy[g];
    if (g_vx) g_vx[g] = hA[4 * g + 2];
    if (g_vy) g_vy[g] = hA[4 * g + 3];
  }
  CK(call_end(ctx));
  return EDMD_OK;
}
