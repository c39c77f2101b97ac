// One-point statistics, statsp (stotf.F90:51-291), with the x pre-pass rhsp
// does when dostat is set (rhsp.F90:70-92). Not on the substep path: the
// reference computes them every avcrt steps (bl_1.F90:92).
//
//   k_stats_x    tiles of neighbouring x-lines in shared memory:
//                u_x = interpx_new(u) shifted by one plane (rhsp.F90:71-79),
//                dudx = diffx(u_x), dwdx = diffx(w), dvdx = diffx(v)
//                (lip.f90:703-765, fd_ix and fd_dx), into the line scratch
//                s1, s2, s3, t1
//   k_stats_y    tiles of neighbouring y-columns of a group of planes:
//                buf1..buf5 = interpy_new of u_x, w, dwdx, dudx (fd_iy) and
//                p (fd_iyp) onto the wall positions, buf6..buf8 = diffy of
//                buf1, buf2, v (fd_dvdy) (stotf.F90:101-110,
//                lip.f90:666-699,767-809), into t2 and t3
//   k_stats_acc  one warp per row (i, j): the k = 0 terms, the sums over the
//                spanwise modes (cte = 1 for k = 0, 2 otherwise,
//                stotf.F90:118-217) reduced across the warp, and the triple
//                products over the physical points after three c2r
//                transforms (stotf.F90:264-285), added to the accumulators
//
// The groups of planes are sized so that the eight buffers fit in t2 and
// t3. Every compact solve is the reference's recurrence in chunks of K rows
// per thread (lines.cuh); the sums over k and over the physical points are reduced in a different
// order than the reference's serial loops (rounding-level differences).
#include <algorithm>

#include "devcommon.cuh"
#include "lines.cuh"
#include "otbl_internal.cuh"
#include "zline.cuh"

namespace otbl {

namespace {

#define C8(c, r, j) (c)[((size_t)(j)-1) * 8 + (r)-1]

__device__ __forceinline__ double rd(double x, int xr) { return xr ? (double)(float)x : x; }

// The window and weights of a compact operator's right-hand side: row r (of n)
// takes cnt weights of row wr of the table times the input rows o..o+cnt-1;
// its recurrence starts at row `first` (rows before it are the right-hand side
// itself).
struct Win {
  int o, cnt, wr;
};
// interpx_new (lip.f90:736-765)
struct OpIntX {
  static constexpr int first = 0;
  __device__ static Win win(int r, int n) {
    if (r == 0) return {0, 4, 0};
    return r <= n - 3 ? Win{r - 1, 4, 2} : Win{n - 4, 4, r};
  }
};
// diffx_inplace (lip.f90:703-731)
struct OpDifX {
  static constexpr int first = 0;
  __device__ static Win win(int r, int n) {
    if (r < 2) return {0, 5, r};
    return r <= n - 3 ? Win{r - 2, 5, 2} : Win{n - 5, 5, r};
  }
};
// interpy_new (lip.f90:767-809): TIPO 0 from ny+1 rows, zero at the wall, TIPO
// 1 from ny rows
template <int TIPO>
struct OpIntY {
  static constexpr int first = 1;
  __device__ static Win win(int r, int n) {
    if (r == 0) return {1, TIPO == 0 ? 0 : 4, 0};
    if (r == 1) return {1, 5, 1};
    return r <= n - 3 ? Win{r - 1, 4, r} : Win{n - 3, TIPO == 1 ? 3 : 4, r};
  }
};
// diffy_inplace (lip.f90:666-699)
struct OpDifY {
  static constexpr int first = 0;
  __device__ static Win win(int r, int n) {
    if (r < 2) return {0, 4, r};
    return r <= n - 3 ? Win{r - 2, 5, r} : Win{n - 4, 4, r};
  }
};

// One operator (table c8, 8 values per row: five weights, then l, 1/pivot,
// upper) on the lines of a tile in shared memory ([rows][L] pairs), chunk q of
// K rows of lane `lane` to y. Uses ex (2 x blockDim values) and px (2 x
// blockDim products). On return every thread has read the tile.
template <typename OP, int K>
__device__ __forceinline__ void stats_solve(const double *__restrict__ c8, const double2 *tile, int n, int C, int L,
                                            int q, int lane, int xr, double2 (&y)[K], double2 *ex, double *px) {
  const int t = threadIdx.x, NT = blockDim.x, s = q * K;
  double l[K], d[K], u[K], pl = 1.0, pu = 1.0;
#pragma unroll
  for (int b = 0; b < K; ++b) {
    const int r = s + b;
    y[b] = make_double2(0.0, 0.0);
    l[b] = d[b] = u[b] = 0.0;
    if (r < n) {
      const Win w = OP::win(r, n);
      const double *cw = c8 + (size_t)w.wr * 8, *cr = c8 + (size_t)r * 8;
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        if (m < w.cnt) {
          const double2 v = tile[(w.o + m) * L + lane];
          fma2(y[b], __ldg(cw + m), make_double2(rd(v.x, xr), rd(v.y, xr)));
        }
      }
      if (r < OP::first) {
        d[b] = 1.0;
      } else {
        d[b] = __ldg(cr + 6);
        if (r > OP::first) l[b] = -__ldg(cr + 5);
        if (r < n - 1) u[b] = __ldg(cr + 7);
      }
    }
    pl *= l[b];
  }
#pragma unroll
  for (int b = 0; b < K; ++b) pu *= -u[b] * d[b];
  ex[t] = forward_end<K, 1, double>(y, l);
  px[t] = pl;
  px[NT + t] = pu;
  __syncthreads();
  forward_from<K, 1, double>(y, l, chunk_carry<double>(ex + t - L, -L, px + t - L, -L, q));
  ex[NT + t] = backward_end<K, 1, double>(y, d, u);
  __syncthreads();
  backward_from<K, 1, double>(y, d, u, chunk_carry<double>(ex + NT + t + L, L, px + NT + t + L, L, C - 1 - q));
}

struct StatsOps {
  const double *fdvdy, *fdx, *fix, *fiy, *fiyp;
};

// the eight buffers of a group of G planes: buffer b at base[b] + (il*ny +
// j-1)*nz1 + kr
struct StatsBufs {
  double *b[8];
};

// blockIdx.y: 0 u (u_x, dudx), 1 w (dwdx), 2 v (dvdx); a CTA takes L pairs of
// neighbouring lines
template <int K>
__global__ void __launch_bounds__(256) k_stats_x(DCoef c, StatsOps op, const double *__restrict__ u,
                                                 const double *__restrict__ v, const double *__restrict__ w,
                                                 double *ux, double *dudx, double *dwdx, double *dvdx, int C, int L) {
  extern __shared__ __align__(16) unsigned char stsm[];
  const int nx = c.nx, ny = c.ny, xr = c.xround, f = blockIdx.y, t = threadIdx.x, NT = blockDim.x;
  const int npp = (c.nz1 >> 1) * (f == 2 ? ny : ny + 1), p0 = blockIdx.x * L;
  if (p0 >= npp) return;  // the whole CTA
  const int q = min(t / L, C - 1), lane = t % L, s = q * K;
  const bool on = t < C * L && p0 + lane < npp;
  double2 *tile = reinterpret_cast<double2 *>(stsm), *ex = tile + (size_t)nx * L;
  double *px = reinterpret_cast<double *>(ex + 2 * NT);
  const double2 *in = reinterpret_cast<const double2 *>(f == 0 ? u : (f == 1 ? w : v));
  for (int e = t; e < nx * L; e += NT) {
    const int r = e / L, m = p0 + (e - r * L);
    cp_async_v(tile + e, in + (size_t)r * npp + min(m, npp - 1), m < npp);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  double2 y[K];
  double *out = f == 0 ? dudx : (f == 1 ? dwdx : dvdx);
  if (f == 0) {
    stats_solve<OpIntX, K>(op.fix, tile, nx, C, L, q, lane, xr, y, ex, px);
    // shifted by one plane: out(i+1) = interp(i), out(1) = interp(1)
    if (t < C * L) {
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int r = s + b;
        if (r < nx - 1) tile[(r + 1) * L + lane] = y[b];
        if (r == 0) tile[lane] = y[b];
      }
    }
    __syncthreads();
    double2 *o = reinterpret_cast<double2 *>(ux);
    for (int e = t; e < nx * L; e += NT) {  // the chx2p transposes back to planes round to REAL4
      const int r = e / L, m = p0 + (e - r * L);
      const double2 x = tile[e];
      if (m < npp) o[(size_t)r * npp + m] = make_double2(rd(x.x, xr), rd(x.y, xr));
    }
    stats_solve<OpDifX, K>(op.fdx, tile, nx, C, L, q, lane, 0, y, ex, px);  // of the unrounded u_x
  } else {
    stats_solve<OpDifX, K>(op.fdx, tile, nx, C, L, q, lane, xr, y, ex, px);
  }
  if (!on) return;
  double2 *o = reinterpret_cast<double2 *>(out) + (size_t)s * npp + p0 + lane;
#pragma unroll
  for (int b = 0; b < K; ++b)
    if (s + b < nx) o[(size_t)b * npp] = make_double2(rd(y[b].x, xr), rd(y[b].y, xr));
}

// blockIdx.y: 0 u_x (buf1, buf6), 1 w (buf2, buf7), 2 dwdx (buf3), 3 dudx
// (buf4), 4 p (buf5), 5 v (buf8); a CTA takes L neighbouring modes of the G
// planes from i0 on
template <typename TP, int K>
__global__ void __launch_bounds__(256) k_stats_y(DCoef c, StatsOps op, const double *__restrict__ ux,
                                                 const double *__restrict__ w, const double *__restrict__ dwdx,
                                                 const double *__restrict__ dudx, const TP *__restrict__ p,
                                                 const double *__restrict__ v, StatsBufs bf, int i0, int G, int C,
                                                 int L) {
  extern __shared__ __align__(16) unsigned char stsm[];
  const int ny = c.ny, nk = c.nz1 >> 1, f = blockIdx.y, t = threadIdx.x, NT = blockDim.x;
  const int rows = f < 4 ? ny + 1 : ny, ncm = G * nk, m0 = blockIdx.x * L;
  const int q = min(t / L, C - 1), lane = t % L, s = q * K;
  double2 *tile = reinterpret_cast<double2 *>(stsm), *ex = tile + (size_t)(ny + 1) * L;
  double *px = reinterpret_cast<double *>(ex + 2 * NT);
  const double *in = f == 0 ? ux : (f == 1 ? w : (f == 2 ? dwdx : (f == 3 ? dudx : v)));
  for (int e = t; e < rows * L; e += NT) {
    const int r = e / L, m = min(m0 + (e - r * L), ncm - 1), il = m / nk, k = m - il * nk;
    const size_t at = ((size_t)(i0 - 1 + il) * rows + r) * nk + k;
    if (f == 4) {
      const V2<TP> x = __ldg(reinterpret_cast<const V2<TP> *>(p) + at);
      tile[e] = make_double2((double)x.x, (double)x.y);
    } else {
      tile[e] = __ldg(reinterpret_cast<const double2 *>(in) + at);
    }
  }
  __syncthreads();
  const int m = min(m0 + lane, ncm - 1), il = m / nk, k = m - il * nk;
  const bool on = t < C * L && m0 + lane < ncm;
  double2 y[K];
  auto store = [&](double *base) {
    double2 *o = reinterpret_cast<double2 *>(base) + ((size_t)il * ny + s) * nk + k;
#pragma unroll
    for (int b = 0; b < K; ++b)
      if (on && s + b < ny) o[(size_t)b * nk] = y[b];
  };
  if (f < 4) {
    stats_solve<OpIntY<0>, K>(op.fiy, tile, ny, C, L, q, lane, 0, y, ex, px);
    store(f == 0 ? bf.b[0] : (f == 1 ? bf.b[1] : (f == 2 ? bf.b[2] : bf.b[3])));
    if (f < 2) {
      if (t < C * L) {
#pragma unroll
        for (int b = 0; b < K; ++b)
          if (s + b < ny) tile[(s + b) * L + lane] = y[b];
      }
      __syncthreads();
      stats_solve<OpDifY, K>(op.fdvdy, tile, ny, C, L, q, lane, 0, y, ex, px);
      store(f == 0 ? bf.b[5] : bf.b[6]);
    }
  } else if (f == 4) {
    stats_solve<OpIntY<1>, K>(op.fiyp, tile, ny, C, L, q, lane, 0, y, ex, px);
    store(bf.b[4]);
  } else {
    stats_solve<OpDifY, K>(op.fdvdy, tile, ny, C, L, q, lane, 0, y, ex, px);
    store(bf.b[7]);
  }
}

// The same for columns of more than 256 chunks (rows above 8448), which no CTA
// holds: a thread per mode, serial sweeps, the forward one's values kept in
// the output.
template <typename OP, typename F>
__device__ __forceinline__ void stats_serial(const double *__restrict__ c8, F in, int n, double2 *out, int so) {
  double2 x = make_double2(0.0, 0.0);
  for (int r = 0; r < n; ++r) {
    const Win w = OP::win(r, n);
    double2 y = make_double2(0.0, 0.0);
    for (int m = 0; m < w.cnt; ++m) fma2(y, c8[(size_t)w.wr * 8 + m], in(w.o + m));
    if (r > OP::first) fma2(y, -c8[(size_t)r * 8 + 5], x);
    out[(size_t)r * so] = x = y;
  }
  for (int r = n - 1; r >= OP::first; --r) {
    double2 y = out[(size_t)r * so];
    const double *cr = c8 + (size_t)r * 8;
    if (r < n - 1) fma2(y, -cr[7], x);
    x = make_double2(y.x * cr[6], y.y * cr[6]);
    out[(size_t)r * so] = x;
  }
}

template <typename TP>
__global__ void __launch_bounds__(128) k_stats_y_tall(DCoef c, StatsOps op, const double *__restrict__ ux,
                                                      const double *__restrict__ w, const double *__restrict__ dwdx,
                                                      const double *__restrict__ dudx, const TP *__restrict__ p,
                                                      const double *__restrict__ v, StatsBufs bf, int i0, int G) {
  const int ny = c.ny, nk = c.nz1 >> 1, f = blockIdx.y, m = blockIdx.x * 128 + threadIdx.x;
  if (m >= G * nk) return;
  const int il = m / nk, k = m - il * nk, rows = f < 4 ? ny + 1 : ny;
  const double *src = f == 0 ? ux : (f == 1 ? w : (f == 2 ? dwdx : (f == 3 ? dudx : v)));
  const size_t at = (size_t)(i0 - 1 + il) * rows * nk + k;
  auto in = [&](int r) { return __ldg(reinterpret_cast<const double2 *>(src) + at + (size_t)r * nk); };
  auto inp = [&](int r) {
    const V2<TP> x = __ldg(reinterpret_cast<const V2<TP> *>(p) + at + (size_t)r * nk);
    return make_double2((double)x.x, (double)x.y);
  };
  auto buf = [&](int b) {
    double *base = b < 4 ? (b < 2 ? (b == 0 ? bf.b[0] : bf.b[1]) : (b == 2 ? bf.b[2] : bf.b[3]))
                         : (b < 6 ? (b == 4 ? bf.b[4] : bf.b[5]) : (b == 6 ? bf.b[6] : bf.b[7]));
    return reinterpret_cast<double2 *>(base) + (size_t)il * ny * nk + k;
  };
  if (f < 4) {
    double2 *o = buf(f);
    stats_serial<OpIntY<0>>(op.fiy, in, ny, o, nk);
    if (f < 2) stats_serial<OpDifY>(op.fdvdy, [&](int r) { return o[(size_t)r * nk]; }, ny, buf(5 + f), nk);
  } else if (f == 4) {
    stats_serial<OpIntY<1>>(op.fiyp, inp, ny, buf(4), nk);
  } else {
    stats_serial<OpDifY>(op.fdvdy, in, ny, buf(7), nk);
  }
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// the 27 sums over k, in the order of their OTBL_ST_* slots from OTBL_ST_US
enum { KS_US = 0, KS_VS, KS_WS, KS_UV, KS_UW, KS_VW, KS_PUP, KS_PVP, KS_PP, KS_PDUDX, KS_PDUDY, KS_PDVDX, KS_PDVDY,
       KS_PDWDZ, KS_VORTX, KS_VORTY, KS_VORTZ, KS_DISPU, KS_DISPV, KS_DISPW, KS_DISPUV, KS_N };

__global__ void __launch_bounds__(128) k_stats_acc(DCoef c, ZTab z, StatsBufs bf, const double *__restrict__ v,
                                                   const double *__restrict__ dvdx, double *acc, int i0, int G) {
  extern __shared__ __align__(16) unsigned char stsm[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int row = blockIdx.x * 4 + wid;
  const int nx = c.nx, ny = c.ny, nz1 = c.nz1, nz2 = c.nz2, M = z.M;
  if (row >= G * ny) return;
  const int il = row / ny, j = row - il * ny + 1, i = i0 + il;
  const size_t PV = (size_t)ny * nz1;
  const size_t rb = (size_t)il * PV + (size_t)(j - 1) * nz1, rv = (size_t)(i - 1) * PV + (size_t)(j - 1) * nz1;
  const double *b1 = bf.b[0] + rb, *b2 = bf.b[1] + rb, *b3 = bf.b[2] + rb, *b4 = bf.b[3] + rb;
  const double *b5 = bf.b[4] + rb, *b6 = bf.b[5] + rb, *b7 = bf.b[6] + rb, *b8 = bf.b[7] + rb;
  const double *vv = v + rv, *dv = dvdx + rv;
  double ks[KS_N];
#pragma unroll
  for (int q = 0; q < KS_N; ++q) ks[q] = 0.0;
  for (int k = lane; k <= nz2; k += 32) {
    const double cte = k == 0 ? 1.0 : 2.0, kz = c.kaz[k];
    const double u1r = b1[2 * k], u1i = b1[2 * k + 1], w2r = b2[2 * k], w2i = b2[2 * k + 1];
    const double vr = vv[2 * k], vi = vv[2 * k + 1], pr = b5[2 * k], pi = b5[2 * k + 1];
    const double x3r = b3[2 * k], x3i = b3[2 * k + 1], x4r = b4[2 * k], x4i = b4[2 * k + 1];
    const double x6r = b6[2 * k], x6i = b6[2 * k + 1], x7r = b7[2 * k], x7i = b7[2 * k + 1];
    const double x8r = b8[2 * k], x8i = b8[2 * k + 1], dvr = dv[2 * k], dvi = dv[2 * k + 1];
    // i kz times a mode: (-kz Im, kz Re)
    const double wzr = -w2i * kz, wzi = w2r * kz, uzr = -u1i * kz, uzi = u1r * kz;
    const double vzr = -vi * kz, vzi = vr * kz;
    ks[KS_US] += cte * (u1r * u1r + u1i * u1i);
    ks[KS_VS] += cte * (vr * vr + vi * vi);
    ks[KS_WS] += cte * (w2r * w2r + w2i * w2i);
    ks[KS_UV] += cte * (u1r * vr + u1i * vi);
    ks[KS_UW] += cte * (u1r * w2r + u1i * w2i);
    ks[KS_VW] += cte * (vr * w2r + vi * w2i);
    ks[KS_PUP] += cte * (pr * u1r + pi * u1i);
    ks[KS_PVP] += cte * (pr * vr + pi * vi);
    ks[KS_PP] += cte * (pr * pr + pi * pi);
    ks[KS_PDUDX] += cte * (pr * x4r + pi * x4i);
    ks[KS_PDUDY] += cte * (pr * x6r + pi * x6i);
    ks[KS_PDVDX] += cte * (pr * dvr + pi * dvi);
    ks[KS_PDVDY] += cte * (pr * x8r + pi * x8i);
    ks[KS_PDWDZ] += cte * (pr * wzr + pi * wzi);
    double ar = x7r - vzr, ai = x7i - vzi;  // o_x = dwdy - dvdz
    ks[KS_VORTX] += cte * (ar * ar + ai * ai);
    ar = uzr - x3r, ai = uzi - x3i;  // o_y = dudz - dwdx
    ks[KS_VORTY] += cte * (ar * ar + ai * ai);
    ar = dvr - x6r, ai = dvi - x6i;  // o_z = dvdx - dudy
    ks[KS_VORTZ] += cte * (ar * ar + ai * ai);
    ks[KS_DISPU] += cte * ((x4r * x4r + x4i * x4i) + (uzr * uzr + uzi * uzi) + (x6r * x6r + x6i * x6i));
    ks[KS_DISPV] += cte * ((dvr * dvr + dvi * dvi) + (vzr * vzr + vzi * vzi) + (x8r * x8r + x8i * x8i));
    ks[KS_DISPW] += cte * ((wzr * wzr + wzi * wzi) + (x3r * x3r + x3i * x3i) + (x7r * x7r + x7i * x7i));
    ks[KS_DISPUV] += cte * ((uzr * vzr + uzi * vzi) + (x4r * dvr + x4i * dvi) + (x6r * x8r + x6i * x8i));
  }
#pragma unroll
  for (int q = 0; q < KS_N; ++q) ks[q] = warp_sum(ks[q]);
  // triple products of u, w, v in physical space (three c2r transforms)
  double2 *bu = reinterpret_cast<double2 *>(stsm) + (size_t)wid * 3 * M, *bw = bu + M, *bv = bw + M;
  line_c2r(z, b1, bu, lane);
  line_c2r(z, b2, bw, lane);
  line_c2r(z, vv, bv, lane);
  double t3[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // u3, v3, u2v, v2u, w2v, w2u
  for (int t = lane; t < M; t += 32) {
    const double2 a = bu[t], b = bw[t], d = bv[t];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double uu = h ? a.y : a.x, ww = h ? b.y : b.x, vp = h ? d.y : d.x;
      t3[0] += (uu * uu) * uu;
      t3[1] += (vp * vp) * vp;
      t3[2] += vp * (uu * uu);
      t3[3] += uu * (vp * vp);
      t3[4] += vp * (ww * ww);
      t3[5] += uu * (ww * ww);
    }
  }
#pragma unroll
  for (int q = 0; q < 6; ++q) t3[q] = warp_sum(t3[q]);
  if (lane == 0) {
    const size_t NS = (size_t)nx * ny, at = (size_t)(i - 1) * ny + (j - 1);
    double *A = acc + at;
    // k = 0: means, gradient means, mean vorticity (stotf.F90:118-134)
    A[OTBL_ST_UA * NS] += b1[0];
    A[OTBL_ST_VA * NS] += vv[0];
    A[OTBL_ST_WA * NS] += b2[0];
    A[OTBL_ST_PM * NS] += b5[0];
    A[OTBL_ST_DUDX0 * NS] += b4[0];
    A[OTBL_ST_DVDX0 * NS] += dv[0];
    A[OTBL_ST_DWDX0 * NS] += b3[0];
    A[OTBL_ST_DUDY0 * NS] += b6[0];
    A[OTBL_ST_DVDY0 * NS] += b8[0];
    A[OTBL_ST_DWDY0 * NS] += b7[0];
    A[OTBL_ST_VORTXA * NS] += b7[0];
    A[OTBL_ST_VORTYA * NS] -= b3[0];
    A[OTBL_ST_VORTZA * NS] += dv[0] - b6[0];
#pragma unroll
    for (int q = 0; q < KS_N; ++q) A[(OTBL_ST_US + q) * NS] += ks[q];
#pragma unroll
    for (int q = 0; q < 6; ++q) A[(OTBL_ST_U3 + q) * NS] += t3[q];
  }
}

static_assert(OTBL_ST_US + KS_N == OTBL_ST_U3, "the k sums fill the slots from OTBL_ST_US to OTBL_ST_U3");
static_assert(OTBL_ST_U3 + 6 == OTBL_NSTATS, "six triple products");
static_assert(OTBL_ST_US + KS_PDUDX == OTBL_ST_PDUDX && OTBL_ST_US + KS_DISPUV == OTBL_ST_DISPUV &&
                  OTBL_ST_US + KS_VORTX == OTBL_ST_VORTX,
              "k-sum slots in the order of OTBL_ST_*");

}  // namespace

size_t stats_bytes(int nx, int ny) { return (size_t)OTBL_NSTATS * nx * ny * sizeof(double); }

cudaError_t launch_statsp(otbl_ctx *c) {
  const int nx = c->cfg.nx, ny = c->cfg.ny, nz = c->cfg.nz, nz1 = c->dc.nz1;
  cudaStream_t s = c->stream;
  if (!c->stats) {
    void *p = nullptr;
    const size_t b = stats_bytes(nx, ny);
    cudaError_t e = cudaMalloc(&p, b);
    if (e != cudaSuccess) return e;
    c->allocs.push_back(p);
    c->bytes += b;
    c->stats = static_cast<double *>(p);
    e = cudaMemsetAsync(c->stats, 0, b, s);
    if (e != cudaSuccess) return e;
    c->stats_samples = 0;
  }
  otbl_coef_offsets o;
  otbl_coef_layout(nx, ny, nz, &o);
  StatsOps op;
  op.fdvdy = c->coef_dev + o.off[OTBL_C_FD_DVDY];
  op.fdx = c->coef_dev + o.off[OTBL_C_FD_DX];
  op.fix = c->coef_dev + o.off[OTBL_C_FD_IX];
  op.fiy = c->coef_dev + o.off[OTBL_C_FD_IY];
  op.fiyp = c->coef_dev + o.off[OTBL_C_FD_IYP];
  const size_t PU = (size_t)(ny + 1) * nz1, PV = (size_t)ny * nz1;
  double *ux = c->w.s1, *dudx = c->w.s2, *dwdx = c->w.s3, *dvdx = c->w.t1;
  // a chunk of 9 (longer lines: 33) rows per thread, as many lanes as 256
  // threads and 96 KB of tile hold
  auto shape = [](int n, int &K, int &C, int &L, int &NT, size_t &smem) {
    K = n <= 9 * 128 ? 9 : 33;
    C = (n + K - 1) / K;
    L = std::max(1, std::min(std::min(256 / C, 16), 6144 / (n + 1)));
    NT = (C * L + 31) / 32 * 32;
    smem = (size_t)(n + 1) * L * 16 + (size_t)NT * (32 + 16);
    return K == 9;
  };
  int K, C, L, NT;
  size_t sm;
  auto go = [&](auto kern, dim3 g, auto... args) {
    allow_smem(kern, sm);
    kern<<<g, NT, sm, s>>>(c->dc, op, args..., C, L);
    c->launches += 1;
  };
  const bool sx = shape(nx, K, C, L, NT, sm);
  const dim3 gx((unsigned)((PU / 2 + L - 1) / L), 3);
  go(sx ? k_stats_x<9> : k_stats_x<33>, gx, (const double *)c->f[OTBL_F_U], (const double *)c->f[OTBL_F_V],
     (const double *)c->f[OTBL_F_W], ux, dudx, dwdx, dvdx);
  // groups of G planes: four buffers of G planes in each of t2 and t3
  const size_t lu = otbl_field_len(nx, ny, nz, 1);
  const int G = (int)std::max<size_t>(1, std::min<size_t>(nx, lu / (4 * PV)));
  ZTab z;
  z.tw = reinterpret_cast<const double2 *>(c->w.twz);
  z.tw2 = reinterpret_cast<const double2 *>(c->w.twz2);
  z.M = nz / 2;
  z.nz = nz;
  z.nz2 = c->dc.nz2;
  const size_t smem = (size_t)4 * 3 * z.M * sizeof(double2);
  allow_smem(k_stats_acc, smem);
  for (int i0 = 1; i0 <= nx; i0 += G) {
    const int g = std::min(G, nx - i0 + 1);
    StatsBufs bf;
    for (int b = 0; b < 8; ++b) bf.b[b] = (b < 4 ? c->w.t2 : c->w.t3) + (size_t)(b % 4) * G * PV;
    const bool sy = shape(ny, K, C, L, NT, sm);
    const dim3 gy((g * (nz1 / 2) + L - 1) / L, 6);
    const double *cx = ux, *cw = c->f[OTBL_F_W], *cdw = dwdx, *cdu = dudx, *cv = c->f[OTBL_F_V];
    const float *pf = reinterpret_cast<const float *>(c->f[OTBL_F_P]);
    const double *pd = c->f[OTBL_F_P];
    if (C > 256) {
      const dim3 gt((g * (nz1 / 2) + 127) / 128, 6);
      if (c->f32[OTBL_F_P])
        k_stats_y_tall<float><<<gt, 128, 0, s>>>(c->dc, op, cx, cw, cdw, cdu, pf, cv, bf, i0, g);
      else
        k_stats_y_tall<double><<<gt, 128, 0, s>>>(c->dc, op, cx, cw, cdw, cdu, pd, cv, bf, i0, g);
      c->launches += 1;
    } else if (c->f32[OTBL_F_P]) {
      go(sy ? k_stats_y<float, 9> : k_stats_y<float, 33>, gy, cx, cw, cdw, cdu, pf, cv, bf, i0, g);
    } else {
      go(sy ? k_stats_y<double, 9> : k_stats_y<double, 33>, gy, cx, cw, cdw, cdu, pd, cv, bf, i0, g);
    }
    k_stats_acc<<<(g * ny + 3) / 4, 128, smem, s>>>(c->dc, z, bf, c->f[OTBL_F_V], dvdx, c->stats, i0, g);
    c->launches += 1;
  }
  c->stats_samples += 1;
  return cudaGetLastError();
}

}  // namespace otbl
