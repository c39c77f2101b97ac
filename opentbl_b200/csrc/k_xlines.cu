// Streamwise (x) line operators of lip.f90 (interpxx, difvisxx). A line is a
// fixed (j, kr) of the plane layout; its nx values are read with the plane
// stride, so the reference's chp2x transpose is replaced by these strided
// loads (its REAL4 rounding is applied at the same points when
// OTBL_XPOSE_FP32 is set). The tridiagonal solves are the chunked ones of
// lines.cuh: a CTA holds L pairs of neighbouring lines, a thread K planes of
// one pair.
#include <algorithm>

#include "devcommon.cuh"
#include "lines.cuh"
#include "otbl_internal.cuh"

namespace otbl {

// T is the arithmetic and output type: double, or float on the mixed path
// (the FP64 state is read and rounded on load, the FP32 coefficients are
// used). interpx reads the state (double), difvisx the products (T) and the
// state; outputs T.
struct XArgs {
  const void *in[3];
  const double *in2[3];  // the second input of difvisxx (velocity)
  void *out[3];
  int np[3];             // lines of each field
  int tiles[3];          // CTA tiles of each field
  const void *tab;       // coefficient tables (T): u-type, then v-type
  int C, lgL;
  CflReset reset;        // interpxx
};

// coefficients of a table: interpxx w0, w1, l, d, u; difvisxx the same for
// the convective system, then f1, f2, f3, l, d, u of the viscous one; after
// the C chunks' values, the chunk products P, Q of each system
constexpr int xcoefs(bool dv) { return dv ? 11 : 5; }
// Tables of lines longer than 1152 planes (K > 9) stay in global memory:
// with the tiles they exceed the shared memory of an SM.
constexpr bool x_table_global(int K) { return K > 9; }
static size_t xtab_elems(int K, int C, bool dv) {  // rounded up to a 16-byte multiple in either type
  return ((size_t)C * (xcoefs(dv) * K + (dv ? 4 : 2)) + 3) / 4 * 4;
}

// A persistent CTA walks tiles of L pairs of lines (neighbouring CTAs on
// neighbouring tiles, so the CTAs at work read contiguous rows). Each input
// tile is copied to shared memory by cp.async while the tile before it is
// being solved; its buffer is free as soon as every thread holds its rows in
// registers. Five CTA barriers per difvisxx tile, three per interpxx tile.
template <typename T, int K, bool DV, bool XR>
__global__ void __launch_bounds__(K > 9 ? 256 : 512, 1) k_xline(DCoefT<T> c, XArgs a) {
  using V = V2<T>;
  using TG = typename std::conditional<DV, T, double>::type;
  using VG = V2<TG>;
  constexpr int NCF = xcoefs(DV), S = NCF * K;
  constexpr bool GT = x_table_global(K);
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = 1 << a.lgL, C = a.C, NT = blockDim.x, t = threadIdx.x, lane = t & (L - 1);
  const int nx = c.nx;
  const int telems = (C * (S + (DV ? 4 : 2)) + 3) & ~3;
  T *tabs = reinterpret_cast<T *>(smraw);
  VG *gb = reinterpret_cast<VG *>(tabs + (GT ? 0 : telems));              // [nx][L]
  double2 *ub = reinterpret_cast<double2 *>(gb + (size_t)((nx * L + 1) & ~1));  // [nx][L], difvisxx
  V *ex = DV ? reinterpret_cast<V *>(ub + (size_t)nx * L) : reinterpret_cast<V *>(gb + (size_t)((nx * L + 1) & ~1));
  const int q = min(t >> a.lgL, C - 1);       // spare threads repeat the last chunk
  const int s = q * K, left = nx - s;         // first plane, planes from there on
  const int bl = q == C - 1 ? left - 1 : -1;  // the last plane's place in the chunk
  const T *tab = tabs + q * S, *P = tabs + C * S;
  const V zero = cmake<V>(T(0), T(0));
  auto cv = [&](auto g) {
    if constexpr (XR) return cmake<V>((T)rnd(g.x, 1), (T)rnd(g.y, 1));
    return cmake<V>((T)g.x, (T)g.y);
  };
  const int n0 = a.tiles[0], n1 = n0 + a.tiles[1], ntile = n1 + a.tiles[2];
  auto field = [&](int tile) { return tile < n0 ? 0 : (tile < n1 ? 1 : 2); };
  auto first_pair = [&](int tile, int f) { return (tile - (f == 0 ? 0 : (f == 1 ? n0 : n1))) << a.lgL; };
  // copies a tile of a field (base in, npp pairs per plane) into buf
  auto stage = [&](auto *buf, const auto *in, int p0, int npp) {
    const bool ok = p0 + lane < npp;
    const auto *g = in + (size_t)(t >> a.lgL) * npp + (ok ? p0 + lane : 0);
    const size_t step = (size_t)(NT >> a.lgL) * npp;
    for (int e = t; e < nx * L; e += NT) {
      cp_async_v(buf + e, g, ok);
      g += step;
    }
    cp_async_commit();
  };
  auto stage_u = [&](int tile) {
    if constexpr (DV) {
      if (tile < ntile) {
        const int f = field(tile);
        stage(ub, reinterpret_cast<const double2 *>(pick3(a.in2, f)), first_pair(tile, f), pick3(a.np, f) >> 1);
      } else {
        cp_async_commit();
      }
    }
  };
  auto stage_g = [&](int tile) {
    if (tile < ntile) {
      const int f = field(tile);
      stage(gb, static_cast<const VG *>(pick3(a.in, f)), first_pair(tile, f), pick3(a.np, f) >> 1);
    } else {
      cp_async_commit();
    }
  };
  stage_u(blockIdx.x);
  stage_g(blockIdx.x);
  if (!DV && blockIdx.x == 0) a.reset(c.ny);
  const T rex = c.S[OTBL_S_REX], idx = c.S[OTBL_S_IDX], uinf = c.S[OTBL_S_UINF];
  int have = -1;  // the table in shared memory
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int f = field(tile), which = f == 0 ? 0 : 1, npp = pick3(a.np, f) >> 1;
    const int pm = first_pair(tile, f) + lane;
    if (which != have) {  // (every thread is past the barrier after its last use of the old table)
      const T *src = static_cast<const T *>(a.tab) + (size_t)which * telems;
      if constexpr (GT) {
        tab = src + q * S;
        P = src + C * S;
      } else {
        __syncthreads();
        for (int e = t; e < telems; e += NT) tabs[e] = src[e];
      }
      have = which;
    }
    V xu[DV ? K : 1];
    V uN = zero, uN1 = zero;
    if constexpr (DV) {
      cp_async_wait<1>();
      __syncthreads();
      const double2 *u = ub + (size_t)s * L + lane;
      const int ic = which == 0 ? 3 : 1;
      const T *vb = c.cofvbx;
      V um = q > 0 ? cv(u[-L]) : zero, u0 = cv(u[0]);
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const V up = b + 1 < left ? cv(u[(b + 1) * L]) : zero;
        V r = zero;
        fma2(r, tab[5 * K + b], up);
        fma2(r, tab[6 * K + b], u0);
        fma2(r, tab[7 * K + b], um);
        xu[b] = r;
        um = u0;
        u0 = up;
      }
      if (q == 0) {
#pragma unroll
        for (int m = 1; m <= 4; ++m) fma2(xu[0], M4(vb, ic, m), cv(u[(m - 1) * L]));
      }
      if (q == C - 1) {
        const double2 *ul = ub + (size_t)(nx - 1) * L + lane;
        uN = cv(ul[0]);
        uN1 = cv(ul[-L]);
        V r = zero;
        fma2(r, M4(vb, ic + 1, 1), uN);
        fma2(r, M4(vb, ic + 1, 2), uN1);
        fma2(r, M4(vb, ic + 1, 3), cv(ul[-2 * L]));
        fma2(r, M4(vb, ic + 1, 4), cv(ul[-3 * L]));
#pragma unroll
        for (int b = 0; b < K; ++b)
          xu[b] = select2(b == bl, r, xu[b]);
      }
      chunk_forward<K, 1, T>(xu, tab + 8 * K, P + 2 * C, ex, q, t, L);
      stage_u(tile + gridDim.x);  // every thread holds its planes
      cp_async_wait<1>();         // this tile's g, made visible by the next barrier
      chunk_backward<K, 1, T>(xu, tab + 9 * K, tab + 10 * K, P + 3 * C, ex + NT, q, C, t, L);
    } else {
      cp_async_wait<0>();
      __syncthreads();
    }
    V y[K];
    {
      // difvisxx: w0 g_{i-1} + w1 g_i; interpxx: w0 g_i + w1 g_{i+1}
      const VG *g = gb + (size_t)s * L + lane;
      V g0 = DV ? (q > 0 ? cv(g[-L]) : zero) : cv(g[0]);
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int o = DV ? b : b + 1;
        const V g1 = o < left ? cv(g[o * L]) : zero;
        V r = zero;
        fma2(r, tab[b], g0);
        fma2(r, tab[K + b], g1);
        y[b] = r;
        g0 = g1;
      }
      const VG *gl = gb + (size_t)(nx - 1) * L + lane;
      const int cf = DV ? (which == 0 ? 1 : 2) : (which == 0 ? 3 : 4), cl = DV ? cf + 2 : (which == 0 ? 2 : 1);
      if (q == 0) {
#pragma unroll
        for (int m = 1; m <= 4; ++m) fma2(y[0], DV ? M5(c.dcbx, cf, m) : M4(c.inbx, cf, m), cv(g[(m - 1) * L]));
      }
      if (q == C - 1) {
        V r = zero;
#pragma unroll
        for (int m = 1; m <= 4; ++m) fma2(r, DV ? M5(c.dcbx, cl, m) : M4(c.inbx, cl, m), cv(gl[(1 - m) * L]));
#pragma unroll
        for (int b = 0; b < K; ++b)
          y[b] = select2(b == bl, r, y[b]);
      }
    }
    chunk_forward<K, 1, T>(y, tab + 2 * K, P, ex, q, t, L);
    stage_g(tile + gridDim.x);
    chunk_backward<K, 1, T>(y, tab + 3 * K, tab + 4 * K, P + C, ex + NT, q, C, t, L);
    if (pm < npp && t < C * L) {
      V *out = static_cast<V *>(pick3(a.out, f)) + (size_t)s * npp + pm;
#pragma unroll
      for (int b = 0; b < K; ++b) {
        if (b < left) {
          V v = y[b];
          if constexpr (DV) {
            fma2(v, rex, xu[b]);
            if (b == bl) {  // outflow: lip.f90:105,132
              v.x = uinf * (uN.x - uN1.x) * idx;
              v.y = uinf * (uN.y - uN1.y) * idx;
            }
          }
          if constexpr (XR) v = cmake<V>((T)rnd(v.x, 1), (T)rnd(v.y, 1));
          *out = v;
          out += npp;
        }
      }
    }
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// launches and tables
// ---------------------------------------------------------------------------
// Planes per chunk: the shortest of 5, 9, 17, 33 whose chunks leave a CTA at
// least four pairs of lines (64-byte rows in FP64), so that short lines get
// short serial chains and long ones full sectors.
static int x_chunk(int nx) {
  if (nx <= 160) return 5;
  for (int K : {9, 17})
    if ((nx + K - 1) / K <= 128) return K;
  return 33;
}

size_t xline_table_bytes(int nx, bool mixed) {
  const int K = x_chunk(nx), C = (nx + K - 1) / K;
  return 2 * (xtab_elems(K, C, false) + xtab_elems(K, C, true)) * (mixed ? sizeof(float) : sizeof(double));
}

template <typename T>
static cudaError_t x_tables(otbl_ctx *c) {
  const int nx = c->cfg.nx, K = x_chunk(nx), C = (nx + K - 1) / K;
  otbl_coef_offsets o;
  otbl_coef_layout(nx, c->cfg.ny, c->cfg.nz, &o);
  std::vector<T> cf(c->coef_host.begin(), c->coef_host.end());
  auto A = [&](int id) { return cf.data() + o.off[id]; };
  std::vector<T> all;
  for (int dv = 0; dv < 2; ++dv)
    for (int wh = 0; wh < 2; ++wh) {
      const int S = xcoefs(dv) * K;
      std::vector<T> tab(xtab_elems(K, C, dv), T(0));
      T *P = tab.data() + (size_t)C * S;
      auto put = [&](int i, int r, T v) { tab[(size_t)(r / K) * S + i * K + r % K] = v; };
      const T *icon = dv ? A(wh ? OTBL_C_DCXV : OTBL_C_DCXU) : A(wh ? OTBL_C_INXV : OTBL_C_INXU);
      const T *econ = dv ? A(wh ? OTBL_C_COFCXV : OTBL_C_COFCXU) : A(wh ? OTBL_C_COFIVX : OTBL_C_COFIUX);
      for (int i = 1; i < nx - 1; ++i) {
        put(0, i, econ[2 * i]);
        put(1, i, econ[2 * i + 1]);
      }
      auto ldu = [&](int at) { return [&put, at](int i, int r, T v) { put(at + i, r, v); }; };
      chunk_factors<T>(ldu(2), K, nx, icon, 0, P, P + C);
      if (dv) {
        const T *ev = A(wh ? OTBL_C_COFVXV : OTBL_C_COFVXU);
        for (int i = 1; i < nx - 1; ++i)
          for (int k = 0; k < 3; ++k) put(5 + k, i, ev[3 * i + k]);
        chunk_factors<T>(ldu(8), K, nx, A(wh ? OTBL_C_VIXV : OTBL_C_VIXU), 0, P + 2 * C, P + 3 * C);
      }
      all.insert(all.end(), tab.begin(), tab.end());
    }
  const cudaError_t e =
      cudaMemcpyAsync(c->w.xtab, all.data(), all.size() * sizeof(T), cudaMemcpyHostToDevice, c->stream);
  return e == cudaSuccess ? cudaStreamSynchronize(c->stream) : e;
}

cudaError_t prepare_xlines(otbl_ctx *c) { return c->mixed ? x_tables<float>(c) : x_tables<double>(c); }

template <typename T, bool DV>
static cudaError_t xline_launch(otbl_ctx *c, const DCoefT<T> &dc, XArgs &a) {
  const int nx = c->cfg.nx, K = x_chunk(nx), C = (nx + K - 1) / K;
  // threads per CTA: 256 (512 for lines of more than 64 chunks), or a half or
  // a quarter of that when the autotuner found narrower CTAs faster (tune_bs
  // 128, 64, 32), and what shared memory holds
  const int most = std::max((C > 64 && K <= 9 ? 4 : 2) * c->tune_bs[DV ? 1 : 0], C);
  auto bytes = [&](int lg) {
    const size_t n = ((size_t)nx << lg) + 1, nt = ((C << lg) + 31) / 32 * 32;
    return (x_table_global(K) ? 0 : xtab_elems(K, C, DV) * sizeof(T)) + n * (DV ? 16 + sizeof(V2<T>) : 16) +
           2 * nt * sizeof(V2<T>) + 16;
  };
  const size_t room = 232448;
  int lg = 0;
  while ((C << (lg + 1)) <= most && lg < 4 && bytes(lg + 1) <= room) ++lg;
  const size_t smem = bytes(lg);
  if (smem > room) return cudaErrorInvalidConfiguration;
  a.C = C;
  a.lgL = lg;
  a.tab = static_cast<const T *>(c->w.xtab) + (DV ? 2 * xtab_elems(K, C, false) : 0);
  int ntile = 0;
  for (int f = 0; f < 3; ++f) {
    a.tiles[f] = (a.np[f] / 2 + (1 << lg) - 1) >> lg;
    ntile += a.tiles[f];
  }
  const int NT = ((C << lg) + 31) / 32 * 32;
  auto go = [&](auto kern) {
    allow_smem(kern, smem);
    const int regs = K > 9 ? 256 : 128;  // per thread, by the launch bounds
    const int per = std::max(1, std::min((int)(233472 / (smem + 1024)), 65536 / (regs * NT)));
    kern<<<std::min(ntile, per * sm_count()), NT, smem, c->stream>>>(dc, a);
  };
  auto byk = [&](auto xr) {
    constexpr bool XR = decltype(xr)::value;
    switch (K) {
      case 5: go(k_xline<T, 5, DV, XR>); break;
      case 9: go(k_xline<T, 9, DV, XR>); break;
      case 17: go(k_xline<T, 17, DV, XR>); break;
      default: go(k_xline<T, 33, DV, XR>);
    }
  };
  if constexpr (sizeof(T) == 8) {
    if (c->dc.xround)
      byk(std::true_type{});
    else
      byk(std::false_type{});
  } else {
    byk(std::false_type{});
  }
  return cudaGetLastError();
}

template <bool DV>
static cudaError_t xlines(otbl_ctx *c, const void *const (&in)[3], void *const (&out)[3], int reset) {
  const int nz1 = c->dc.nz1, ny = c->cfg.ny;
  const double *st[3] = {c->f[OTBL_F_U], c->f[OTBL_F_V], c->f[OTBL_F_W]};
  XArgs a;
  for (int f = 0; f < 3; ++f) {
    a.in[f] = in[f];
    a.in2[f] = st[f];
    a.out[f] = out[f];
    a.np[f] = nz1 * (f == 1 ? ny : ny + 1);
  }
  if (reset) a.reset = {c->st, c->w.vm_bits};
  prof_begin(c, DV ? PK_DIFVISX : PK_INTERPX);
  const cudaError_t e = stream_xlines(c, DV) ? launch_xlines_stream(c, DV, reset)
                        : c->mixed           ? xline_launch<float, DV>(c, c->dcf, a)
                                             : xline_launch<double, DV>(c, c->dc, a);
  prof_end(c);
  c->launches += 1;
  return e;
}

cudaError_t launch_interpx(otbl_ctx *c, int reset) {
  return xlines<false>(c, {c->f[OTBL_F_U], c->f[OTBL_F_V], c->f[OTBL_F_W]}, {c->w.ux, c->w.vx, c->w.wx}, reset);
}

cudaError_t launch_difvisx(otbl_ctx *c) {
  return xlines<true>(c, {c->w.uu, c->w.uv, c->w.uw}, {c->w.cu, c->w.cv, c->w.cw}, 0);
}

}  // namespace otbl
