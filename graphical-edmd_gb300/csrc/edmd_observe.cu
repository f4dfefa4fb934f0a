// edmd_observe.cu -- observables computed on the device from the engine state.
//
// Pair correlation g(r) of calculate_pcf (src/pcf.c:16-75): every unordered
// pair closer than max_r (minimum image, PBC src/EDMD.c:5896) adds 2 to bin
// (int)(r / dr); the histogram is then divided by 2 pi r dr rho N at the bin
// centres r = (i + 0.5) dr.  The device counts pairs exactly (integers) over
// the cell lists, so the result equals the reference's O(N^2) loop bit for
// bit; positions are the stored ones, as the reference reads them.
#include <cmath>
#include "edmd_ctx.h"

namespace {

// Every pair once, one thread per disk: the disks of the cells after its own
// (rows above, and to the right in its row) within reach, and its own cell's of
// larger index.  Bound by FP64 issue, so a pair costs the two differences and
// the squared distance only: its bin, (int)(sqrt(d2) / dr), is a monotone
// function of d2 whose steps `step` the host has found exactly (step[b]: the
// least d2 of bin b), so an FP32 estimate and two integer compares give it.
// (Square root, division and tests on half-idle lanes in FP64: 0.92 ms for 10^5
// disks, max_r = 10; so 0.21.)
__global__ void __launch_bounds__(128) k_pcf_half(const SysDev* __restrict__ sys, int s, float inv_dr, int nb, int kx,
                                                  int ky, const double* __restrict__ step, double d2max,
                                                  unsigned long long* __restrict__ hist) {
  extern __shared__ unsigned int cnt[];
  for (int b = threadIdx.x; b < nb; b += blockDim.x) cnt[b] = 0;
  __syncthreads();
  const SysDev& S = sys[s];
  const Box& B = S.B;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B.N) {
    const double px = S.d[i].x, py = S.d[i].y;
    const int X = S.cx[i], Y = S.cy[i];
    for (int oy = 0; oy <= ky; oy++) {
      int cy = Y + oy;
      if (cy >= B.Nyc) cy -= B.Nyc;
      const int32_t* row = S.head + (int64_t)cy * B.Nxc;
      for (int ox = oy ? -kx : 0; ox <= kx; ox++) {
        int cx = X + ox;
        if (cx < 0) cx += B.Nxc;
        if (cx >= B.Nxc) cx -= B.Nxc;
        int j = row[cx];
        int guard = 0;
        while (j != NIL && guard++ < B.N) {
          const Disk* Q = S.d + j;
          double dx = Q->x - px, dy = Q->y - py;
          const int nx = Q->nxt;
          if (oy || ox || j > i) {
            pbc_i(B, dx, dy);
            const double d2 = dx * dx + dy * dy;
            if (__double_as_longlong(d2) < __double_as_longlong(d2max)) {        // both non-negative
              const long long u = __double_as_longlong(d2);
              const int e = (int)(u >> 52) - 1023;
              const float f = e < -126 ? 0.0f : __int_as_float(((e + 127) << 23) | (int)((u >> 29) & 0x7fffff));
              int b = (int)(sqrtf(f) * inv_dr);
              b = b < nb ? b : nb - 1;
              if (u < __double_as_longlong(step[b])) b--;
              else if (u >= __double_as_longlong(step[b + 1])) b++;
              atomicAdd(&cnt[b], 1u);
            }
          }
          j = nx;
        }
      }
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    if (cnt[b]) atomicAdd(&hist[b], (unsigned long long)cnt[b]);
}

// the least d2 >= 0 at which the monotone `above` holds, from a guess nearby
template <class F>
double first_above(double d2, F above) {
  while (d2 > 0 && above(d2)) d2 = std::nextafter(d2, 0.0);
  while (!above(d2)) d2 = std::nextafter(d2, INFINITY);
  return d2;
}

// one thread per disk i: pairs (i, j > i) in the cells within reach, for
// boxes that the reach wraps around
__global__ void k_pcf(const SysDev* __restrict__ sys, int s, double dr, double max_r, int nb,
                      int kx, int ky, unsigned long long* __restrict__ hist) {
  extern __shared__ unsigned long long sh[];
  for (int b = threadIdx.x; b < nb; b += blockDim.x) sh[b] = 0;
  __syncthreads();
  const SysDev& S = sys[s];
  const Box& B = S.B;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B.N) {
    const Disk P = S.d[i];
    const int X = S.cx[i], Y = S.cy[i];
    // offsets covering the whole grid visit every column / row once
    const int x0 = kx * 2 + 1 >= B.Nxc ? 0 : X - kx, nx = kx * 2 + 1 >= B.Nxc ? B.Nxc : 2 * kx + 1;
    const int y0 = ky * 2 + 1 >= B.Nyc ? 0 : Y - ky, ny = ky * 2 + 1 >= B.Nyc ? B.Nyc : 2 * ky + 1;
    for (int oy = 0; oy < ny; oy++) {
      int cy = (y0 + oy) % B.Nyc;
      if (cy < 0) cy += B.Nyc;
      for (int ox = 0; ox < nx; ox++) {
        int cx = (x0 + ox) % B.Nxc;
        if (cx < 0) cx += B.Nxc;
        int j = S.head[cy * B.Nxc + cx];
        int guard = 0;
        while (j != NIL && guard++ < B.N) {
          const Disk Q = S.d[j];
          if (j > i) {
            double dx = Q.x - P.x, dy = Q.y - P.y;
            pbc(B, dx, dy);
            const double r = sqrt(dx * dx + dy * dy);
            if (r < max_r) {
              const int bin = (int)(r / dr);
              if (bin < nb) atomicAdd(&sh[bin], 1ull);
            }
          }
          j = Q.nxt;
        }
      }
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    if (sh[b]) atomicAdd(&hist[b], sh[b]);
}

}  // namespace

extern "C" int edmd_get_pcf(edmd_ctx* ctx, int32_t s, double dr, double max_r, double* g_out,
                            int32_t cap, int32_t* nbins_out) {
  if (!ctx || s < 0 || s >= ctx->nsys || !(dr > 0) || !(max_r > 0) || !g_out || cap < 1)
    return EDMD_ERR_ARG;
  const SysDev& S = ctx->hs[s];
  const Box& B = S.B;
  if (max_r > (B.Lx < B.Ly ? B.Lx : B.Ly) / 2)
    return set_err(ctx, EDMD_ERR_ARG, "max_r above half the box: the minimum image is ambiguous");
  const int nb = (int)(max_r / dr);        // num_bins of calculate_pcf
  if (nb < 1 || nb > 65536) return set_err(ctx, EDMD_ERR_ARG, "bad number of bins");
  if (nb > cap) return set_err(ctx, EDMD_ERR_CAPACITY, "g(r) output too small");
  // a disk's stored position lies in its cell, so partners within max_r are
  // at most ceil(max_r / cell) + 1 cells away
  const int kx = (int)ceil(max_r / B.cxs) + 1, ky = (int)ceil(max_r / B.cys) + 1;
  if (ctx->pcf_bins < nb) {                // histogram and bin steps, kept for the next call
    if (ctx->pcf) cudaFree(ctx->pcf);
    ctx->pcf = nullptr;
    ctx->pcf_bins = 0;
    CK(cudaMalloc(&ctx->pcf, (2 * (size_t)nb + 1) * 8));
    ctx->pcf_bins = nb;
  }
  unsigned long long* hist = (unsigned long long*)ctx->pcf;
  CK(cudaMemsetAsync(hist, 0, nb * sizeof(unsigned long long), ctx->stream));
  // cells are distinct up to the reach, a block's counts fit 32 bits, and bins
  // are wide enough for the FP32 estimate (d2 below 2^-126, which it takes for
  // zero, lies in bin 0) and for first_above (b dr b dr is a normal number)
  std::vector<double> step;                // to the device: kept until the copy back
  if (2 * kx + 1 <= B.Nxc && 2 * ky + 1 <= B.Nyc && B.N < (1 << 25) && dr >= 1e-12) {
    step.resize(nb + 1);
    step[0] = 0;
    for (int b = 1; b <= nb; b++)
      step[b] = first_above(b * dr * (b * dr), [&](double d2) { return (int)(std::sqrt(d2) / dr) >= b; });
    const double far = first_above(max_r * max_r, [&](double d2) { return !(std::sqrt(d2) < max_r); });
    double* dstep = (double*)ctx->pcf + nb;
    CK(cudaMemcpyAsync(dstep, step.data(), (nb + 1) * 8, cudaMemcpyHostToDevice, ctx->stream));
    k_pcf_half<<<(B.N + 127) / 128, 128, nb * sizeof(unsigned int), ctx->stream>>>(
        ctx->ds, s, (float)(1.0 / dr), nb, kx, ky, dstep, far < step[nb] ? far : step[nb], hist);
  } else {
    k_pcf<<<(B.N + 127) / 128, 128, nb * sizeof(unsigned long long), ctx->stream>>>(ctx->ds, s, dr, max_r, nb,
                                                                                     kx, ky, hist);
  }
  CK(cudaGetLastError());
  std::vector<unsigned long long> h(nb);
  CK(sync_copy(ctx, h.data(), hist, nb * 8, cudaMemcpyDeviceToHost));
  // normalisation of calculate_pcf, same operations in the same order
  const double volume = B.Lx * B.Ly;
  const double density = B.N / volume;
  for (int i = 0; i < nb; i++) {
    const double r = (i + 0.5) * dr;
    const double shell_volume = 2 * M_PI * r * dr;
    const double norm = shell_volume * density * B.N;
    const double g = 2.0 * (double)h[i];
    g_out[i] = norm > 0 ? g / norm : 0.0;
  }
  if (nbins_out) *nbins_out = nb;
  return EDMD_OK;
}
