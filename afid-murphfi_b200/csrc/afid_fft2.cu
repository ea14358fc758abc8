// afid_fft2.cu — the y and z transforms of lengths that are not 32 x {1,2,3,4,6,8,12,16,24,32}, as
// two or three register transforms: N = R1 M, M = R2 or R2 R3.
//
// With n = n1 M + m and k = k1 + R1 k',
//   X[k] = sum_m w_M^(m k') [ w_N^(m k1) sum_{n1} w_R1^(n1 k1) x[n1 M + m] ],
// and the sum over m again so for three factors.  A thread takes the R1 points of its row from
// global memory (z) or the staged tile (y), transforms them in registers and puts them, twiddled, into
// shared memory; after a barrier a thread takes R2 of those, and so on; the last transform's results go
// straight to global memory (the y r2c passes them through shared memory once more to split the
// packed pair).  The kernels these replace (k_div_fft_y, k_fft_z, k_ifft_y: a shared-memory pass and a
// barrier per radix-2..5 factor with runtime radices and divisions) stay for lengths without such
// factors.
//   240 x 200 (y x z) x 180 FP64, us a launch: z 86 -> 30 (0.72 of the copy bandwidth), y forward with
//   the divergence 124 -> 102, y inverse 84 -> 37; 320 x 300 x 225 mixed: 110 -> 42, 202 -> 177 (8% less
//   again with coherent loads), 136 -> 64;
//   three transforms, 450 x 432 x 96 mixed: z 128 -> 50, y inverse 133 -> 74; 480 x 100 x 96 FP64: 52 -> 37.
// Lengths 32 x {..} keep the warp transform, which is as fast or faster there (384 FP64 z 116 us against
// 203 by two transforms; 128 FP64 y forward 5.8 against 8.0).
// Rows of 128 bytes move per x tile (8 complex doubles, 16 complex floats, 8 packed pairs of
// velocities).  The lengths of the transforms are launch arguments and the transform of each
// length is reached by a switch; RMAX, the largest one a kernel holds, sets its registers.
#include <algorithm>

#include "afid_device.cuh"
#include "afid_internal.h"

namespace afid {

namespace {

template <typename TS>
struct Pair2;
template <>
struct Pair2<double> {
  using type = double2;
};
template <>
struct Pair2<float> {
  using type = float2;
};

using Split = FftSplit;

// Threads a block is compiled for: a thread per row of the widest of two transforms, 256 for three
// (the threads loop over the rows).  Blocks an SM that the registers are cut for: 512 threads in FP64
// (128 registers), 1024 in FP32, so that one block's loads run beside another's transforms.
__host__ __device__ constexpr int block_threads(int W, int RMAX, bool THREE) {
  return THREE ? 256 : (W * RMAX + 31) / 32 * 32;
}
template <typename TS>
__host__ __device__ constexpr int blocks_per_sm(int W, int RMAX, bool THREE) {
  const int n = (sizeof(TS) == 8 ? 512 : 1024) / block_threads(W, RMAX, THREE);
  return RMAX > 20 ? 1 : n < 1 ? 1 : n;
}

// DFT of the first R registers of x in natural order, R <= RMAX; ts = N / R.
template <int R, int RMAX, bool INV, typename T>
__device__ __forceinline__ void dft_r(typename Cplx<T>::type (&x)[RMAX], const typename Cplx<T>::type *__restrict__ tw,
                                      int ts) {
  if constexpr (R <= RMAX) {
    typename Cplx<T>::type a[R];
#pragma unroll
    for (int q = 0; q < R; ++q) a[q] = x[q];
    reg_fft_rec<INV, T, R, 0, 1>(a, tw, ts);
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = a[q];
  }
}
template <int RMAX, bool INV, typename T>
__device__ __forceinline__ void dft_any(int R, typename Cplx<T>::type (&x)[RMAX],
                                        const typename Cplx<T>::type *__restrict__ tw, int ts) {
  switch (R) {
    case 2: dft_r<2, RMAX, INV, T>(x, tw, ts); break;
    case 3: dft_r<3, RMAX, INV, T>(x, tw, ts); break;
    case 4: dft_r<4, RMAX, INV, T>(x, tw, ts); break;
    case 5: dft_r<5, RMAX, INV, T>(x, tw, ts); break;
    case 6: dft_r<6, RMAX, INV, T>(x, tw, ts); break;
    case 8: dft_r<8, RMAX, INV, T>(x, tw, ts); break;
    case 9: dft_r<9, RMAX, INV, T>(x, tw, ts); break;
    case 10: dft_r<10, RMAX, INV, T>(x, tw, ts); break;
    case 12: dft_r<12, RMAX, INV, T>(x, tw, ts); break;
    case 15: dft_r<15, RMAX, INV, T>(x, tw, ts); break;
    case 16: dft_r<16, RMAX, INV, T>(x, tw, ts); break;
    case 18: dft_r<18, RMAX, INV, T>(x, tw, ts); break;
    case 20: dft_r<20, RMAX, INV, T>(x, tw, ts); break;
    case 25: dft_r<25, RMAX, INV, T>(x, tw, ts); break;
  }
}

// Element (k1, m) of column c of the tile sits at ((k1 M + m) W + c).  The first transform's results
// of row m, twiddled by w_N^(m k1):
template <int RMAX, bool INV, typename T>
__device__ __forceinline__ void put_first(typename Cplx<T>::type *s, typename Cplx<T>::type (&x)[RMAX],
                                          const Split &f, int W, int m, int c,
                                          const typename Cplx<T>::type *__restrict__ tw) {
  dft_any<RMAX, INV, T>(f.r1, x, tw, f.m);
#pragma unroll
  for (int k1 = 0; k1 < RMAX; ++k1)
    if (k1 < f.r1) s[(k1 * f.m + m) * W + c] = k1 == 0 ? x[0] : cmul(x[k1], twiddle<INV, T>(tw, m * k1));
}
// The middle of three transforms, in place: rows (k1, n3) over n2, twiddled by w_M^(n3 k2).
template <int RMAX, bool INV, typename T>
__device__ __forceinline__ void middle(typename Cplx<T>::type *s, const Split &f, int W, int c,
                                       const typename Cplx<T>::type *__restrict__ tw) {
  for (int row = threadIdx.x / W; row < f.r1 * f.r3; row += blockDim.x / W) {
    const int k1 = row / f.r3, n3 = row - k1 * f.r3;
    typename Cplx<T>::type x[RMAX], *p = s + (k1 * f.m + n3) * W + c;
#pragma unroll
    for (int n2 = 0; n2 < RMAX; ++n2)
      if (n2 < f.r2) x[n2] = p[n2 * f.r3 * W];
    dft_any<RMAX, INV, T>(f.r2, x, tw, f.r1 * f.r3);
#pragma unroll
    for (int k2 = 0; k2 < RMAX; ++k2)
      if (k2 < f.r2) p[k2 * f.r3 * W] = k2 == 0 ? x[0] : cmul(x[k2], twiddle<INV, T>(tw, f.r1 * n3 * k2));
  }
}
// The last transform: row (k1, k2) over n3 (two transforms: row k1 over n2); its results are the
// elements k = first + step t of the whole, t = 0 .. count - 1.
struct Last {
  int rows, count, step;
};
__device__ __forceinline__ Last last_of(const Split &f) {
  return f.r3 > 1 ? Last{f.r1 * f.r2, f.r3, f.r1 * f.r2} : Last{f.r1, f.r2, f.r1};
}
template <int RMAX, bool INV, typename T>
__device__ __forceinline__ int last(const typename Cplx<T>::type *s, typename Cplx<T>::type (&x)[RMAX],
                                    const Split &f, const Last &l, int W, int row, int c,
                                    const typename Cplx<T>::type *__restrict__ tw) {
  const int k1 = f.r3 > 1 ? row / f.r2 : row, k2 = f.r3 > 1 ? row - k1 * f.r2 : 0;
  const typename Cplx<T>::type *p = s + (k1 * f.m + k2 * f.r3) * W + c;
#pragma unroll
  for (int t = 0; t < RMAX; ++t)
    if (t < l.count) x[t] = p[t * W];
  dft_any<RMAX, INV, T>(l.count, x, tw, l.rows);
  return k1 + f.r1 * k2;
}

// z c2c in place.  Block: W x points (8 FP64, 16 FP32) at one ky.
template <int RMAX, bool THREE, bool INV, typename TS>
__global__ void __launch_bounds__(block_threads(128 / (2 * (int)sizeof(TS)), RMAX, THREE),
                                  blocks_per_sm<TS>(128 / (2 * (int)sizeof(TS)), RMAX, THREE))
    k_fft2_z(Geom g, typename Cplx<TS>::type *spec, Split f,
             const typename Cplx<TS>::type *__restrict__ tw) {
  chain_begin();
  using C = typename Cplx<TS>::type;
  constexpr int W = 128 / (int)sizeof(C);
  extern __shared__ __align__(16) unsigned char smem_f2[];
  C *s = reinterpret_cast<C *>(smem_f2);
  const int c = threadIdx.x % W, k = blockIdx.x * W + c;
  const bool in = k < g.nxm;
  const size_t zs = (size_t)g.nyh * g.ldxc;
  C *base = spec + (size_t)blockIdx.y * g.ldxc + k;
  for (int m = threadIdx.x / W; m < f.m; m += blockDim.x / W) {
    C x[RMAX];
#pragma unroll
    for (int n1 = 0; n1 < RMAX; ++n1)
      if (n1 < f.r1) {
        x[n1].x = 0;
        x[n1].y = 0;
        if (in) x[n1] = base[(size_t)(n1 * f.m + m) * zs];
      }
    put_first<RMAX, INV, TS>(s, x, f, W, m, c, tw);
    if constexpr (!THREE) break;  // a thread per row
  }
  __syncthreads();
  if constexpr (THREE) {
    middle<RMAX, INV, TS>(s, f, W, c, tw);
    __syncthreads();
  }
  const Last l = last_of(f);
  for (int row = threadIdx.x / W; row < l.rows; row += blockDim.x / W) {
    C x[RMAX];
    const int k0 = last<RMAX, INV, TS>(s, x, f, l, W, row, c, tw);
#pragma unroll
    for (int t = 0; t < RMAX; ++t)
      if (t < l.count && in) base[(size_t)(k0 + l.step * t) * zs] = x[t];
    if constexpr (!THREE) break;
  }
}

// Divergence (pressure.F90:147-158), forward y r2c and 1/(nym nzm) as k_div_fft_y.  Block: 16 x
// points (8 packed pairs) at one z index.
template <int RMAX, typename TS>
__global__ void __launch_bounds__(block_threads(8, RMAX, false), blocks_per_sm<TS>(8, RMAX, false))
    k_fft2_div(Geom g0, Tables t, const StepCoef *sc_all, int ns, const double *vx,
               const double *vy, const double *vz, typename Cplx<TS>::type *spec, Split f,
               const typename Cplx<TS>::type *__restrict__ tw, const double *field) {
  chain_begin();
  using C = typename Cplx<TS>::type;
  constexpr int W = 8;
  extern __shared__ __align__(16) unsigned char smem_f2[];
  C *s = reinterpret_cast<C *>(smem_f2);
  const int k0 = blockIdx.x * 16, i = blockIdx.y;
  Geom g = g0;
  if (!inst_active(g, i)) return;
  bind_instance(g, i);
  const int q = threadIdx.x % W, row0 = threadIdx.x / W, dj = blockDim.x / W;
  const int kk = k0 + 2 * q, N = g.nym, nxm = g.nxm;
  {
    // the packed rows first: taken straight into the transform's registers, six values a row, they
    // left 384 threads an SM and took as long as the kernel before
    const StepCoef sc = sc_all[sc_slot(g, i, ns)];
    const double usdtal = 1.0 / (sc.dt * sc.al);
    const size_t c0 = col_off(g, 0, i) + kk, ci = col_off(g, 0, zinc(g, i)) + kk;
    const double2 ux = kk < nxm ? __ldg(reinterpret_cast<const double2 *>(t.udx3m + kk)) : make_double2(0.0, 0.0);
    auto put = [&](int j, double a, double b) {
      C z;
      z.x = (TS)a;
      z.y = (TS)b;
      s[j * W + q] = z;
    };
    if (kk >= nxm) {
      for (int j = row0; j < N; j += dj) put(j, 0.0, 0.0);
    } else if (field) {  // spectra: the field itself
      for (int j = row0; j < N; j += dj) {
        const double2 v = *reinterpret_cast<const double2 *>(field + c0 + (size_t)j * g.ldx);
        put(j, v.x, (kk + 1 < nxm) ? v.y : 0.0);
      }
    } else {
      const bool two = kk + 1 < nxm;
      const int d2 = two ? 2 : 1;  // an existing value where the pair's second point does not
#pragma unroll 4
      for (int j = row0; j < N; j += dj) {
        const size_t o = (size_t)j * g.ldx, op = (size_t)wrap_inc(j, N) * g.ldx;
        const double2 zi = *reinterpret_cast<const double2 *>(vz + ci + o);
        const double2 zc = *reinterpret_cast<const double2 *>(vz + c0 + o);
        const double2 yj = *reinterpret_cast<const double2 *>(vy + c0 + op);
        const double2 yc = *reinterpret_cast<const double2 *>(vy + c0 + o);
        const double2 xc = *reinterpret_cast<const double2 *>(vx + c0 + o);
        const double x2 = vx[c0 + o + d2];
        const double dv1 = ((zi.y - zc.y) * g.dz + (yj.y - yc.y) * g.dy + (x2 - xc.y) * ux.y) * usdtal;
        put(j, ((zi.x - zc.x) * g.dz + (yj.x - yc.x) * g.dy + (xc.y - xc.x) * ux.x) * usdtal, two ? dv1 : 0.0);
      }
    }
  }
  __syncthreads();
  C x[RMAX];
  if (row0 < f.m) {
    // rows n1 M + m in, elements (k1, m) out: the same places, so only this thread's
#pragma unroll
    for (int n1 = 0; n1 < RMAX; ++n1)
      if (n1 < f.r1) x[n1] = s[(n1 * f.m + row0) * W + q];
    put_first<RMAX, false, TS>(s, x, f, W, row0, q, tw);
  }
  __syncthreads();
  const Last l = last_of(f);
  if (row0 < l.rows) last<RMAX, false, TS>(s, x, f, l, W, row0, q, tw);
  __syncthreads();
  if (row0 < l.rows) {  // in natural order, for the split of the pairs
#pragma unroll
    for (int t2 = 0; t2 < RMAX; ++t2)
      if (t2 < l.count) s[(row0 + l.step * t2) * W + q] = x[t2];
  }
  __syncthreads();
  const TS norm = (TS)(1.0 / (nz_norm(g) * (double)N)), half = (TS)0.5;
  for (int e = threadIdx.x; e < g.nyh * 16; e += blockDim.x) {
    const int ex = e & 15, ky = e >> 4, kx = k0 + ex;
    if (kx >= nxm) continue;
    const C zk = s[ky * W + (ex >> 1)], zn = s[(ky == 0 ? 0 : N - ky) * W + (ex >> 1)];
    C X;
    if ((ex & 1) == 0) {
      X.x = (zk.x + zn.x) * half;
      X.y = (zk.y - zn.y) * half;
    } else {
      X.x = (zk.y + zn.y) * half;
      X.y = (zn.x - zk.x) * half;
    }
    X.x *= norm;
    X.y *= norm;
    spec[(size_t)(ky + (size_t)g.nyh * i) * g.ldxc + kx] = X;
  }
}

// Backward y c2r as k_ifft_y.  Block: 16 x points (8 packed pairs) at one z index.  Rows above N/2 are the
// conjugates of rows N - j.  With two transforms the half spectrum is staged with asynchronous
// copies, all in flight at once; with three a row is read straight from global memory, twice (its place
// in shared memory would have to be kept until every row's first transform is done).
template <int RMAX, bool THREE, typename TS>
__global__ void __launch_bounds__(block_threads(8, RMAX, THREE), blocks_per_sm<TS>(8, RMAX, THREE))
    k_fft2_ify(Geom g, const typename Cplx<TS>::type *spec, TS *phi, Split f,
               const typename Cplx<TS>::type *__restrict__ tw) {
  chain_begin();
  using C = typename Cplx<TS>::type;
  using V = typename Pair2<TS>::type;
  constexpr int W = 8;
  extern __shared__ __align__(16) unsigned char smem_f2[];
  C *s = reinterpret_cast<C *>(smem_f2);  // [N/2 + 1][16] staged (two transforms), then [N][W]
  const int i = blockIdx.y;
  if (!inst_active(g, i)) return;
  const int k0 = blockIdx.x * 16, N = g.nym, nvalid = min(16, g.nxm - k0);
  const C *src = spec + (size_t)g.nyh * i * g.ldxc + k0;
  if constexpr (!THREE) {
    for (int e = threadIdx.x; e < g.nyh * 16; e += blockDim.x) {
      const int c = e & 15, jj = e >> 4;
      const bool ok = c < nvalid;
      cp_async_zfill<(int)sizeof(C)>(&s[e], ok ? (const void *)(src + (size_t)jj * g.ldxc + c) : (const void *)src,
                                     ok);
    }
    cp_async_wait_all();
    __syncthreads();
  }
  const int p = threadIdx.x % W, row0 = threadIdx.x / W, dj = blockDim.x / W, k = k0 + 2 * p;
  const bool in0 = k < g.nxm, in1 = k + 1 < g.nxm;
  // row j of the packed sequence Z = X + iY of the pair
  auto packed = [&](int j) {
    const bool cj = 2 * j > N;
    const int jj = cj ? N - j : j;
    C X, Y, Z;
    if constexpr (THREE) {
      X.x = X.y = Y.x = Y.y = 0;
      if (in0) X = src[(size_t)jj * g.ldxc + 2 * p];
      if (in1) Y = src[(size_t)jj * g.ldxc + 2 * p + 1];
    } else {
      X = s[jj * 16 + 2 * p];
      Y = s[jj * 16 + 2 * p + 1];
    }
    if (cj) {
      X.y = -X.y;
      Y.y = -Y.y;
    }
    if (jj == 0 || 2 * jj == N) {
      X.y = 0;
      Y.y = 0;
    }
    Z.x = X.x - Y.y;
    Z.y = X.y + Y.x;
    return Z;
  };
  if constexpr (THREE) {
    for (int m = row0; m < f.m; m += dj) {
      C x[RMAX];
#pragma unroll
      for (int n1 = 0; n1 < RMAX; ++n1)
        if (n1 < f.r1) x[n1] = packed(n1 * f.m + m);
      put_first<RMAX, true, TS>(s, x, f, W, m, p, tw);
    }
    __syncthreads();
    middle<RMAX, true, TS>(s, f, W, p, tw);
  } else {
    C x[RMAX];
    if (row0 < f.m) {
#pragma unroll
      for (int n1 = 0; n1 < RMAX; ++n1)
        if (n1 < f.r1) x[n1] = packed(n1 * f.m + row0);
    }
    __syncthreads();  // the staged rows have been read
    if (row0 < f.m) put_first<RMAX, true, TS>(s, x, f, W, row0, p, tw);
  }
  __syncthreads();
  const Last l = last_of(f);
  for (int row = row0; row < l.rows; row += dj) {
    C x[RMAX];
    const int kf = last<RMAX, true, TS>(s, x, f, l, W, row, p, tw);
    TS *dst = phi + col_off(g, 0, i) + k;
#pragma unroll
    for (int t = 0; t < RMAX; ++t)
      if (t < l.count) {
        TS *d = dst + (size_t)(kf + l.step * t) * g.ldx;
        if (in1) {
          V v;
          v.x = x[t].x;
          v.y = x[t].y;
          *reinterpret_cast<V *>(d) = v;
        } else if (in0) {
          d[0] = x[t].x;
        }
      }
    if constexpr (!THREE) break;
  }
}

// Dynamic shared memory: N rows of W columns; the inverse y transform by two stages N/2 + 1 rows of 16
// points in the same place.
size_t fft2_smem(const Split &f, int W, size_t elem, Stage st) {
  const size_t n = (size_t)f.r1 * f.m, tile = n * W;
  if (st == Stage::IfftY && f.r3 == 1) return std::max(tile, (n / 2 + 1) * 16) * elem;
  return tile * elem;
}

template <int RMAX, bool THREE, typename TS>
cudaError_t launch_r(const LaunchCtx &L, const SubstepBuffers &b, int ns, Stage st, const Split &f) {
  using C = typename Cplx<TS>::type;
  const Geom &g = L.g;
  C *spec = (C *)b.spec;
  const C *twy = (const C *)L.twy, *twz = (const C *)L.twz;
  const bool z = st == Stage::FftZFwd || st == Stage::FftZInv;
  const int W = z ? 128 / (int)sizeof(C) : 8;
  const int threads = block_threads(W, std::max(f.r1, f.r2), THREE);
  const size_t smem = fft2_smem(f, W, sizeof(C), st);
  auto fit = [&](auto kern) { return smem > 48 * 1024 ? allow_dynamic_smem(kern) : cudaSuccess; };
  cudaError_t e;
  if (z) {
    const dim3 grid((g.nxm + W - 1) / W, g.nyh);
    auto kern = st == Stage::FftZFwd ? k_fft2_z<RMAX, THREE, false, TS> : k_fft2_z<RMAX, THREE, true, TS>;
    if ((e = fit(kern)) != cudaSuccess) return e;
    launch_chained(L, kern, grid, threads, smem, g, spec, f, twz);
    return cudaGetLastError();
  }
  const dim3 grid((g.nxm + 15) / 16, g.nzm);
  if constexpr (!THREE) {
    if (st == Stage::DivFftY) {
      auto kern = k_fft2_div<RMAX, TS>;
      if ((e = fit(kern)) != cudaSuccess) return e;
      launch_chained(L, kern, grid, threads, smem, g, L.t, b.sc, ns, b.vx_o, b.vy_o, b.vz_o, spec, f, twy,
                     b.fft_field);
      return cudaGetLastError();
    }
  }
  auto kern = k_fft2_ify<RMAX, THREE, TS>;
  if ((e = fit(kern)) != cudaSuccess) return e;
  launch_chained(L, kern, grid, threads, smem, g, spec, (TS *)b.phi, f, twy);
  return cudaGetLastError();
}

}  // namespace

// The factors of N: two up to 20 with the smaller larger one (r1 <= r2: more threads load, fewer values
// each), else three up to 16, else 625 = 25 x 25; r1 = 0 without any.  Above 20 the two transforms'
// registers (180 to 255 in FP64) leave too few threads (1024 points by two transforms of 32, FP32: the
// inverse y transform 36 us against 32 by three); every other length with such a factor splits
// otherwise.  625 gains on the general kernels all the same: 64 x 625 x 64, z in FP64 33.1 -> 23.8
// us, the y forward transform in mixed 53.7 -> 35.2 (in FP64 59.8 -> 64.8).
FftSplit fft2_split(int N) {
  static const int kR[] = {1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 25};
  FftSplit f{0, 0, 0, 0};
  int best = 1 << 30;
  auto take = [&](int a, int b, int c, int most, int rank) {
    const int big = std::max(a, std::max(b, c));
    if (a * b * c != N || big > most || rank + big >= best) return;
    best = rank + big;
    f = FftSplit{a, b, c, b * c};
  };
  for (int a : kR)
    for (int b : kR) {
      if (a <= b) {
        take(a, b, 1, 20, 0);
        take(a, b, 1, 25, 2000);
      }
      for (int c : kR)
        if (a > 1 && b > 1 && c > 1 && a >= b && b >= c) take(a, b, c, 16, 1000);
    }
  return f;
}

template <typename TS>
bool launch_fft2(const LaunchCtx &L, const SubstepBuffers &b, int ns, Stage st, cudaError_t *err) {
  const bool z = st == Stage::FftZFwd || st == Stage::FftZInv;
  const Split f = z ? L.split_z : L.split_y;
  if (f.r1 == 0) return false;
  // The forward y transform by three is not built: against k_div_fft_y, which is bound by the same loads
  // of the velocities, it took 99 us and not 84 in FP64 (480 x 100 x 96); in mixed it would be the
  // faster one (450 x 432 x 96: 173 and not 197).
  if (st == Stage::DivFftY && f.r3 > 1) return false;
  if (fft2_smem(f, z ? 64 / (int)sizeof(TS) : 8, 2 * sizeof(TS), st) > kMaxDynSmem) return false;
  if (f.r3 > 1)
    *err = f.r1 <= 10 ? launch_r<10, true, TS>(L, b, ns, st, f) : launch_r<16, true, TS>(L, b, ns, st, f);
  else
    *err = f.r2 <= 10   ? launch_r<10, false, TS>(L, b, ns, st, f)
           : f.r2 <= 16 ? launch_r<16, false, TS>(L, b, ns, st, f)
           : f.r2 <= 20 ? launch_r<20, false, TS>(L, b, ns, st, f)
                        : launch_r<25, false, TS>(L, b, ns, st, f);
  return true;
}
template bool launch_fft2<double>(const LaunchCtx &, const SubstepBuffers &, int, Stage, cudaError_t *);
template bool launch_fft2<float>(const LaunchCtx &, const SubstepBuffers &, int, Stage, cudaError_t *);

}  // namespace afid
