// afid_stats.cu — on-device statistics and outputs: the wall-normal profiles of
// CalcMeanProfiles.F90, the spectra of spectra.F90 and the movie planes of MakeMovie*Cut.F90.
//
// The fifteen y-z averages written to means.h5 (Tbar, vybar, vzbar, vxT, vyT, vzT, Trms, vxrms,
// vyrms, vzrms, vxvy, vxvz, vyvz, chiT, epsilon) are reduced in two passes: every block walks
// through neighbouring x-columns with one thread per wall-normal row k and keeps the fifteen
// running sums in registers, writes them as one partial row per block, and a second kernel adds the
// partials in a fixed order (deterministic, no atomics).  The host applies the reference's
// normalisation (CalcMeanProfiles.F90:88-102, 203-207).
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "afid_internal.h"

namespace afid {

constexpr int kNumProfiles = 15;

// Sums over columns of the fifteen integrands of CalcMeanProfiles.F90:48-72 (means and second
// moments), :104-128 (chiT) and :164-199 (epsilon).  A block walks along y through `len` columns of
// one z index, one thread per row k (blockDim.x >= nxm), and carries what the next column uses
// again: of the 38 values an integrand set reads, 22 are loaded per column.  With the columns strided
// over the blocks every value was loaded, and one launch bound of 1024 threads held the fifteen sums
// and their operands to 64 registers: 252 us at 256 x 192 x 192 cells, now 181.
// partial[(b*15 + q)*nxm + k].
template <int MAXT>
__global__ void __launch_bounds__(MAXT)
    k_mean_partial(Geom g0, Tables t, const double *__restrict__ vx, const double *__restrict__ vy,
                   const double *__restrict__ vz, const double *__restrict__ temp, int i0, int len, int nseg,
                   double *__restrict__ partial) {
  const int nxm = g0.nxm, k = threadIdx.x;
  if (k >= nxm) return;
  const int i = i0 + blockIdx.x / nseg, js = blockIdx.x % nseg * len, je = min(js + len, g0.nym);
  Geom g = g0;
  bind_instance(g, i);
  double acc[kNumProfiles];
#pragma unroll
  for (int q = 0; q < kNumProfiles; ++q) acc[q] = 0.0;
  const int kp = k + 1, km = max(k - 1, 0), kpc = min(k + 1, nxm - 1);
  const bool lo = (k == 0), hi = (k == nxm - 1);
  const double udx3m = __ldg(t.udx3m + k);
  const double tdx = 0.5 * g.dx / __ldg(t.g3rm + k);                                                     // :113-126
  const double tdx2 = 0.125 * (g.dx / __ldg(t.g3rm + k)) * (g.dx / __ldg(t.g3rm + k));  // :182-197
  const double dz = g.dz, dy = g.dy;
  const int ip = zinc(g, i), im = zdec(g, i);
  // at (j - 1, i) and (j - 1, i + 1), and at column j: rows k, k + 1, k - 1 of the centre, row k of i +- 1
  const int jm = wrap_dec(js, g.nym);
  size_t c = col_off(g, js, i), cip = col_off(g, js, ip), cim = col_off(g, js, im);
  double txm = vx[col_off(g, jm, i) + k], txm1 = vx[col_off(g, jm, i) + kp];
  double tm = temp[col_off(g, jm, i) + k], zm = vz[col_off(g, jm, i) + k], zmip = vz[col_off(g, jm, ip) + k];
  double xc = vx[c + k], xc1 = vx[c + kp], yc = vy[c + k], ycp = vy[c + kpc], ycm = vy[c + km];
  double yip = vy[cip + k], yim = vy[cim + k], zc = vz[c + k], zip = vz[cip + k], tc = temp[c + k];
  for (int j = js; j < je; ++j) {
    const int jp = wrap_inc(j, g.nym);
    const size_t cjp = col_off(g, jp, i), cjpip = col_off(g, jp, ip), cjpim = col_off(g, jp, im);
    const double xn = vx[cjp + k], xn1 = vx[cjp + kp], yn = vy[cjp + k], ynp = vy[cjp + kpc], ynm = vy[cjp + km];
    const double ynip = vy[cjpip + k], ynim = vy[cjpim + k], zn = vz[cjp + k], znip = vz[cjpip + k];
    const double tn = temp[cjp + k];
    const double tip = temp[cip + k], tim = temp[cim + k], tcp = temp[c + kpc], tcm = temp[c + km];
    const double xip = vx[cip + k], xip1 = vx[cip + kp], xim = vx[cim + k], xim1 = vx[cim + kp];
    const double zcp = vz[c + kpc], zcm = vz[c + km], zipp = vz[cip + kpc], zipm = vz[cip + km];
    const double vxm = 0.5 * (xc + xc1), vym = 0.5 * (yc + yn), vzm = 0.5 * (zc + zip);
    acc[0] += tc;
    acc[1] += vym;
    acc[2] += vzm;
    acc[3] += vxm * tc;
    acc[4] += vym * tc;
    acc[5] += vzm * tc;
    acc[6] += tc * tc;
    acc[7] += 0.5 * (xc * xc + xc1 * xc1);
    acc[8] += 0.5 * (yc * yc + yn * yn);
    acc[9] += 0.5 * (zc * zc + zip * zip);
    acc[10] += 0.25 * (xc + xc1) * (yc + yn);
    acc[11] += 0.25 * (xc + xc1) * (zc + zip);
    acc[12] += 0.25 * (yc + yn) * (zc + zip);
    // chiT: horizontal gradients, then the wall-normal one with the plate values at the walls
    const double tz = (tip - tim) * 0.5 * dz, ty = (tn - tm) * 0.5 * dy;
    double tx = tcp - tcm;  // the wall rows repeat their own value
    if (lo || hi) {
      const size_t pl = (size_t)j + (size_t)g.nym * i;
      tx += lo ? 2.0 * g.tfixs * (tc - __ldg(t.tempbp + pl)) : 0.0;
      tx += hi ? 2.0 * g.tfixn * (__ldg(t.temptp + pl) - tc) : 0.0;
    }
    acc[13] += tz * tz + ty * ty + (tx * tdx) * (tx * tdx);
    // epsilon: the seven interior terms, then the wall-normal derivatives of vz and vy
    const double e1 = (zip - zc) * dz;
    const double a2 = ynip - ynim, b2 = yip - yim;
    const double a3 = xip1 - xim1, b3 = xip - xim;
    const double a4 = znip - zmip, b4 = zn - zm;
    const double e5 = (yn - yc) * dy;
    const double a6 = xn1 - txm1, b6 = xn - txm;
    const double e7 = (xc1 - xc) * udx3m;
    double eps = e1 * e1 + 0.125 * dz * dz * (a2 * a2 + b2 * b2) + 0.125 * dz * dz * (a3 * a3 + b3 * b3) +
                 0.125 * dy * dy * (a4 * a4 + b4 * b4) + e5 * e5 + 0.125 * dy * dy * (a6 * a6 + b6 * b6) + e7 * e7;
    // d/dx of vz at (j, i+1), (j, i) and vy at (j+1, i), (j, i)
    double zxi = zipp - zipm, zxc = zcp - zcm, yxj = ynp - ynm, yxc = ycp - ycm;
    if (lo) {
      zxi += g.inslws * 2.0 * (zip - 0.0);
      zxc += g.inslws * 2.0 * (zc - 0.0);
      yxj += g.inslws * 2.0 * (yn - g.xminusu);
      yxc += g.inslws * 2.0 * (yc - g.xminusu);
    }
    if (hi) {
      zxi += g.inslwn * 2.0 * (0.0 - zip);
      zxc += g.inslwn * 2.0 * (0.0 - zc);
      yxj += g.inslwn * 2.0 * (g.xplusu - yn);
      yxc += g.inslwn * 2.0 * (g.xplusu - yc);
    }
    eps += tdx2 * (zxi * zxi + zxc * zxc) + tdx2 * (yxj * yxj + yxc * yxc);
    acc[14] += eps;
    txm = xc;
    txm1 = xc1;
    tm = tc;
    zm = zc;
    zmip = zip;
    xc = xn;
    xc1 = xn1;
    yc = yn;
    ycp = ynp;
    ycm = ynm;
    yip = ynip;
    yim = ynim;
    zc = zn;
    zip = znip;
    tc = tn;
    c = cjp;
    cip = cjpip;
    cim = cjpim;
  }
#pragma unroll
  for (int q = 0; q < kNumProfiles; ++q) partial[((size_t)blockIdx.x * kNumProfiles + q) * nxm + k] = acc[q];
}

// The partials summed in a fixed order: 32 warps each every 32nd block's, then the 32 sums.  (One thread
// per profile row over all blocks took 29 us at 592 blocks, eight warps 38 us at 1152.)
constexpr int kReduceWarps = 32;
__global__ void __launch_bounds__(32 * kReduceWarps)
    k_mean_reduce(const double *__restrict__ partial, int nblocks, int nxm, double *__restrict__ out) {
  __shared__ double part[kReduceWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = kNumProfiles * nxm;
  const int e = blockIdx.x * 32 + lane;  // e = q*nxm + k
  double s = 0.0;
  if (e < n) {
#pragma unroll 4
    for (int b = warp; b < nblocks; b += kReduceWarps) s += partial[(size_t)b * n + e];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < n) {
#pragma unroll
    for (int w = 1; w < kReduceWarps; ++w) s += part[w][lane];
    out[e] = s;
  }
}

}  // namespace afid

using namespace afid;

namespace afid {

// Profiles of the columns [col0, col0 + ncols) into host out[15 * nxm], normalised by ny_nz
// (the number of y-z points averaged over) with the instance's ren / pect.
int ctx_mean_profiles(afid_ctx_t *ctx, int col0, int ncols, double ny_nz, double ren, double pect, double *out) {
  const Geom &g = ctx->L.g;
  const int nxm = g.nxm;
  // segments of whole z indices' columns: about four blocks of 256 rows an SM, at least four columns
  const int nz = ncols / g.nym, threads = (nxm + 31) / 32 * 32;
  const int want = 148 * std::max(1, 1024 / threads);
  const int parts = std::max(1, std::min(want / nz, (g.nym + 3) / 4));
  const int len = (g.nym + parts - 1) / parts, nseg = (g.nym + len - 1) / len, nb = nseg * nz;
  const size_t need = (size_t)nb * kNumProfiles * nxm + (size_t)kNumProfiles * nxm;
  if (ctx->stats_elems < need) {
    if (ctx->stats_buf) cudaFree(ctx->stats_buf);
    ctx->stats_buf = nullptr;
    ctx->stats_elems = 0;
    if (cudaMalloc(&ctx->stats_buf, need * sizeof(double)) != cudaSuccess) return AFID_E_ALLOC;
    ctx->stats_elems = need;
  }
  double *partial = ctx->stats_buf, *sums = ctx->stats_buf + (size_t)nb * kNumProfiles * nxm;
  auto kern = threads <= 256 ? k_mean_partial<256> : threads <= 512 ? k_mean_partial<512> : k_mean_partial<1024>;
  kern<<<nb, threads, 0, ctx->stream>>>(g, ctx->L.t, ctx->vx, ctx->vy, ctx->vz, ctx->temp, col0 / g.nym, len, nseg,
                                        partial);
  k_mean_reduce<<<(kNumProfiles * nxm + 31) / 32, 32 * kReduceWarps, 0, ctx->stream>>>(partial, nb, nxm, sums);
  ctx->launches += 2;
  cudaError_t e = cudaGetLastError();
  std::vector<double> h((size_t)kNumProfiles * nxm);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h.data(), sums, h.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return ctx_fail(ctx, e);
  // CalcMeanProfiles.F90:88-102 (x inym x inzm), square roots of the rms rows, :203-207
  const double inv = 1.0 / ny_nz;
  for (int q = 0; q < kNumProfiles; ++q)
    for (int k = 0; k < nxm; ++k) {
      double v = h[(size_t)q * nxm + k] * inv;
      if (q >= 6 && q <= 9) v = std::sqrt(v);
      if (q == 13) v /= pect;
      if (q == 14) v /= ren;
      out[(size_t)q * nxm + k] = v;
    }
  return AFID_OK;
}

}  // namespace afid

extern "C" int afid_gpu_mean_profiles(afid_ctx_t *ctx, double *out) {
  if (!ctx || !out || ctx->L.g.batch) return AFID_E_INVALID;
  cudaSetDevice(ctx->dev);
  const Geom &g = ctx->L.g;
  return ctx_mean_profiles(ctx, 0, g.nym * g.nzm, (double)g.nym * (double)g.nzm, g.ren, g.pect, out);
}

// ------------------------------------------------------------------------------------------
// Spectra (spectra.F90): the y r2c + z c2c Fourier coefficients of vx, vy, vz and temp at
// k = 1..nxm, normalised by 1/(nym*nzm) (CalcFourierCoef, :70-96), accumulated as dt*|F|^2
// (AddRealSpectrum, :101-114) and divided by the averaging interval when read (WriteSpectra).
// The transforms are the Poisson solver's forward kernels with the field as their input.
// ------------------------------------------------------------------------------------------
namespace afid {

template <typename C>
__global__ void k_spec_acc(const C *__restrict__ spec, int nxm, int nyh, int nzm, int ldxc, double dt,
                           double *__restrict__ acc) {
  const size_t n = (size_t)nxm * nyh * nzm;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(e % nxm);
    const size_t m = e / nxm;  // ky + nyh*kz
    const C v = spec[m * ldxc + k];
    const double re = (double)v.x, im = (double)v.y;
    acc[e] += dt * (re * re + im * im);
  }
}

}  // namespace afid

extern "C" {

int afid_gpu_spectra_reset(afid_ctx_t *ctx) {
  if (!ctx || ctx->L.g.batch) return AFID_E_INVALID;
  cudaSetDevice(ctx->dev);
  const Geom &g = ctx->L.g;
  const size_t n = (size_t)4 * g.nxm * g.nyh * g.nzm;
  if (!ctx->spec_acc) {
    if (cudaMalloc(&ctx->spec_acc, n * sizeof(double)) != cudaSuccess) {
      ctx->spec_acc = nullptr;
      return AFID_E_ALLOC;
    }
  }
  ctx->spec_tav = 0.0;
  cudaError_t e = cudaMemsetAsync(ctx->spec_acc, 0, n * sizeof(double), ctx->stream);
  return e == cudaSuccess ? AFID_OK : ctx_fail(ctx, e);
}

int afid_gpu_spectra_update(afid_ctx_t *ctx, double dt) {
  if (!ctx || ctx->L.g.batch || !(dt > 0.0)) return AFID_E_INVALID;
  if (!ctx->spec_acc) {
    const int s = afid_gpu_spectra_reset(ctx);
    if (s != AFID_OK) return s;
  }
  cudaSetDevice(ctx->dev);
  const Geom &g = ctx->L.g;
  const size_t n = (size_t)g.nxm * g.nyh * g.nzm;
  SubstepBuffers b = ctx_buffers(ctx);
  const double *fields[4] = {ctx->vx, ctx->vy, ctx->vz, ctx->temp};
  for (int f = 0; f < 4; ++f) {
    b.fft_field = fields[f];
    cudaError_t e = launch_stage(ctx->L, b, 0, Stage::DivFftY);
    if (e == cudaSuccess && g.nzm > 1) e = launch_stage(ctx->L, b, 0, Stage::FftZFwd);
    if (e != cudaSuccess) return ctx_fail(ctx, e);
    double *acc = ctx->spec_acc + (size_t)f * n;
    const int nb = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    if (ctx->L.mixed)
      k_spec_acc<<<nb, 256, 0, ctx->stream>>>((const float2 *)ctx->spec, g.nxm, g.nyh, g.nzm, g.ldxc, dt, acc);
    else
      k_spec_acc<<<nb, 256, 0, ctx->stream>>>((const double2 *)ctx->spec, g.nxm, g.nyh, g.nzm, g.ldxc, dt, acc);
    e = cudaGetLastError();
    if (e != cudaSuccess) return ctx_fail(ctx, e);
    ctx->launches += (g.nzm > 1) ? 3 : 2;
  }
  ctx->spec_tav += dt;
  return AFID_OK;
}

int afid_gpu_spectra_read(afid_ctx_t *ctx, int which, double *out, double *tav) {
  if (!ctx || !out || which < 0 || which > 3 || !ctx->spec_acc || !(ctx->spec_tav > 0.0)) return AFID_E_INVALID;
  cudaSetDevice(ctx->dev);
  const Geom &g = ctx->L.g;
  const size_t n = (size_t)g.nxm * g.nyh * g.nzm;
  cudaError_t e = cudaMemcpyAsync(out, ctx->spec_acc + (size_t)which * n, n * sizeof(double), cudaMemcpyDeviceToHost,
                                  ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return ctx_fail(ctx, e);
  const double inv = 1.0 / ctx->spec_tav;  // WriteSpectra: divide by the averaging interval
  for (size_t q = 0; q < n; ++q) out[q] *= inv;
  if (tav) *tav = ctx->spec_tav;
  return AFID_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------
// Planes of a field (MakeMovie{X,Y,Z}Cut.F90): a wall-parallel plane at k gathered by a kernel,
// the others as strided 2-D copies.
// ------------------------------------------------------------------------------------------
namespace afid {

__global__ void k_xcut(const double *__restrict__ f, int ldx, int nym, int nzm, int k, double *__restrict__ out) {
  const size_t n = (size_t)nym * nzm;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    out[e] = f[k + (size_t)ldx * e];
}

}  // namespace afid

extern "C" int afid_gpu_slice(afid_ctx_t *ctx, int which, int axis, int index, double *out) {
  if (!ctx || !out || which < 0 || which > 4 || ctx->L.g.batch) return AFID_E_INVALID;
  cudaSetDevice(ctx->dev);
  const Geom &g = ctx->L.g;
  const double *f = (which == 0) ? ctx->vx : (which == 1) ? ctx->vy : (which == 2) ? ctx->vz
                  : (which == 3) ? ctx->temp : ctx->pr;
  const size_t dp = (size_t)g.ldx * sizeof(double), w = (size_t)g.nx * sizeof(double);
  cudaError_t e = cudaSuccess;
  if (axis == 0) {  // x = const: out[i][j], nzm x nym
    if (index < 0 || index >= g.nx) return AFID_E_INVALID;
    const size_t n = (size_t)g.nym * g.nzm;
    if (ctx->stats_elems < n) {
      if (ctx->stats_buf) cudaFree(ctx->stats_buf);
      ctx->stats_buf = nullptr;
      ctx->stats_elems = 0;
      if (cudaMalloc(&ctx->stats_buf, n * sizeof(double)) != cudaSuccess) return AFID_E_ALLOC;
      ctx->stats_elems = n;
    }
    k_xcut<<<(int)std::min<size_t>((n + 255) / 256, 148 * 8), 256, 0, ctx->stream>>>(f, g.ldx, g.nym, g.nzm, index,
                                                                                      ctx->stats_buf);
    ctx->launches += 1;
    e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(out, ctx->stats_buf, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
  } else if (axis == 1) {  // y = const: out[i][k], nzm x nx
    if (index < 0 || index >= g.nym) return AFID_E_INVALID;
    e = cudaMemcpy2DAsync(out, w, f + (size_t)g.ldx * index, dp * g.nym, w, g.nzm, cudaMemcpyDeviceToHost, ctx->stream);
  } else if (axis == 2) {  // z = const: out[j][k], nym x nx
    if (index < 0 || index >= g.nzm) return AFID_E_INVALID;
    e = cudaMemcpy2DAsync(out, w, f + (size_t)g.ldx * g.nym * index, dp, w, g.nym, cudaMemcpyDeviceToHost, ctx->stream);
  } else {
    return AFID_E_INVALID;
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? AFID_OK : ctx_fail(ctx, e);
}

// ---- plane means (h5tools/means.F90 ymean / zmean / ymeanr / zmeanr) ----------------------
// Mean over y (axis 1: out[i][k], planes x rows of nxc) or over z (axis 2: out[j][k]) of a
// field stored x-fastest with stride ld, ny rows per z-plane, nz planes.  The sum runs in the
// reference's order (the averaged index ascending) and is divided once at the end.
__global__ void k_plane_mean(const double *__restrict__ f, int ld, int ny, int nz, int nxc, int axis,
                             double *__restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;  // i (y-mean) or j (z-mean)
  if (k >= nxc) return;
  double acc = 0.0;
  if (axis == 1) {
    const double *p = f + (size_t)ld * ny * r + k;
    for (int j = 0; j < ny; ++j) acc += p[(size_t)ld * j];
    out[(size_t)r * nxc + k] = acc / (double)ny;
  } else {
    const double *p = f + (size_t)ld * r + k;
    for (int i = 0; i < nz; ++i) acc += p[(size_t)ld * ny * i];
    out[(size_t)r * nxc + k] = acc / (double)nz;
  }
}

namespace {
int plane_mean(afid_ctx_t *ctx, const double *f, int ld, int ny, int nz, int nxc, int axis, double *out) {
  const size_t n = (size_t)(axis == 1 ? nz : ny) * nxc;
  if (ctx->stats_elems < n) {
    if (ctx->stats_buf) cudaFree(ctx->stats_buf);
    ctx->stats_buf = nullptr;
    ctx->stats_elems = 0;
    if (cudaMalloc(&ctx->stats_buf, n * sizeof(double)) != cudaSuccess) return AFID_E_ALLOC;
    ctx->stats_elems = n;
  }
  const dim3 grid((unsigned)((nxc + 127) / 128), (unsigned)(axis == 1 ? nz : ny));
  k_plane_mean<<<grid, 128, 0, ctx->stream>>>(f, ld, ny, nz, nxc, axis, ctx->stats_buf);
  ctx->launches += 1;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, ctx->stats_buf, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? AFID_OK : ctx_fail(ctx, e);
}
}  // namespace

extern "C" int afid_gpu_mean_plane(afid_ctx_t *ctx, int which, int axis, double *out) {
  if (!ctx || !out || which < 0 || which > 3 || (axis != 1 && axis != 2) || ctx->L.g.batch) return AFID_E_INVALID;
  cudaSetDevice(ctx->dev);
  const Geom &g = ctx->L.g;
  const double *f = (which == 0) ? ctx->vx : (which == 1) ? ctx->vy : (which == 2) ? ctx->vz : ctx->temp;
  return plane_mean(ctx, f, g.ldx, g.nym, g.nzm, g.nx, axis, out);
}

extern "C" int afid_gpu_sal_mean_plane(afid_ctx_t *ctx, int axis, double *out) {
  if (!ctx || !out || !ctx->sal || (axis != 1 && axis != 2)) return AFID_E_INVALID;
  cudaSetDevice(ctx->dev);
  const SalGeom &sg = ctx->sal->sg;
  return plane_mean(ctx, ctx->sal->sal, sg.ldr, sg.nymr, sg.nzmr, sg.nxmr, axis, out);
}
