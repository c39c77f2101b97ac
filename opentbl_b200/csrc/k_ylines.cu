// Wall-normal (y) line operators of the substep on the plane layout, as the
// chunked solves of lines.cuh: a thread holds K rows of one spanwise mode
// (its real and imaginary column), the chunks of L neighbouring modes make a
// CTA, so every row access is a segment of L x 16 (8) bytes.
//   k_interpy    interpyy (lip.f90:359-440) of u, w and v in Fourier space
//   k_tail       the tail of rhsp (rhsp.F90:291-484)
//   k_pois_lu    pivots of the (x-mode, kz) y-systems of pois (once)
//   k_pois_solve their solution every substep (pois.f90:106-117, soltriy)
#include <cudaTypedefs.h>

#include <algorithm>
#include <type_traits>

#include "devcommon.cuh"
#include "lines.cuh"
#include "otbl_internal.cuh"

namespace otbl {

// two neighbouring columns' values at p, not kept in L1
__device__ __forceinline__ double2 ld_stream(const double2 *p) {
  double2 v;
  asm volatile("ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_stream(const float2 *p) {
  float2 v;
  asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
template <typename V>
__device__ __forceinline__ V ld_row(const V *p, bool ok) {
  return ok ? ld_stream(p) : cmake<V>(0, 0);
}

// Rows per chunk: 7 rows keep the tail's three solves in 168 registers on the
// mixed path (24 bytes spilled) and 255 in FP64 (48 bytes); boxes taller than
// 447 rows take longer chunks, above 3840 rows (256 chunks of 15) the serial
// kernels *_tall.
static int y_chunk(int ny) { return ny < 7 * 64 ? 7 : 15; }
constexpr bool y_table_global(int K) { return K > 7; }
// The tail's tables: coefficient i of row s + b of chunk q at tab[q S + i K +
// b], S = ncf K, the chunk products after the C chunks, rounded up to 16 bytes.
// Its persistent CTAs copy them to shared memory once (read through L1 they
// were evicted: 257x193x256, two thirds of their sectors from L2, a warp
// waited 12-18 cycles per instruction); boxes taller than 447 rows read them
// from global memory.
static size_t ytab_elems(int K, int C, int ncf, int nprod) { return ((size_t)C * (ncf * K + nprod) + 2 + 3) / 4 * 4; }
// lanes of a CTA of C chunks: what NT threads hold, at most 32, at least 1
static int y_lanes(int C, int NT) { return std::max(1, std::min(32, NT / C)); }
static int y_threads(int C, int L) { return (C * L + 31) / 32 * 32; }

// a thread's place: chunk q of mode mc (of ncm, in storage order), rows s..
struct YPlace {
  int L, C, t, NT, q, s, mc;
  bool active;
  __device__ YPlace(int L_, int C_, int K)
      : L(L_), C(C_), t(threadIdx.x), NT(blockDim.x), q(min(t / L_, C_ - 1)), s(q * K) {}
  __device__ void tile(int n, int ncm) {
    const int m = n * L + t % L;
    active = m < ncm && t < C * L;  // the others repeat a valid place and store nothing
    mc = min(m, ncm - 1);
  }
};

// interpyy, which 0: u, w (in rows ny+1), which 1: v (in rows ny); out rows
// 1..ny. blockIdx.y = field (u, w, v). T: arithmetic and output type (float
// on the mixed path, with the FP32 coefficient copy); the state is FP64. Its
// table is small enough to be read through L1 (coefficient i of row s + b of
// chunk q at [(i K + b) QS + q], one line per row): staged in shared memory by
// persistent CTAs, with the next tile's rows fetched ahead, it took 37.4
// against 33.3 us at 257x97x128 and 193 against 161 at 513x129x256.
struct InterpyArgs {
  const double *in[3];
  void *out[3];
  const void *tab[2];  // wA, wB, l, d, u, then P, Q, per which
  int which[3];
  int C, L;
};
constexpr int kYInterp = 5;

// a table read through L1
template <typename T>
struct LdgTab {
  const T *p;
  __device__ T operator[](int i) const { return __ldg(p + i); }
  __device__ T operator*() const { return __ldg(p); }
  __device__ LdgTab operator+(int i) const { return {p + i}; }
  __device__ LdgTab &operator+=(int i) {
    p += i;
    return *this;
  }
};

template <typename T, int K, int QS>
__global__ void __launch_bounds__(256, K > 7 ? 1 : 2) k_interpy(DCoefT<T> c, InterpyArgs a) {
  using V = V2<T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int f = blockIdx.y, ny = c.ny, nk = c.nz1 >> 1;
  YPlace w(a.L, a.C, K);
  w.tile(blockIdx.x, c.nx * nk);
  const int which = pick3(a.which, f), jin = which == 0 ? ny + 1 : ny, left = ny - w.s;
  const int i = w.mc / nk, k = w.mc - i * nk;
  const double2 *in = reinterpret_cast<const double2 *>(pick3(a.in, f)) + (size_t)i * jin * nk + k;
  const LdgTab<T> all{static_cast<const T *>(which == 0 ? a.tab[0] : a.tab[1])};
  const LdgTab<T> P = all + kYInterp * K * QS, tab = all + w.q;
  // u, w: e1 g(r) + e2 g(r+1), wall row 0; v: e1 g(r-1) + e2 g(r)
  const int off = which == 0 ? 0 : -1;
  double2 g[K + 1];
  const double2 *p = in + (ptrdiff_t)(w.s + off) * nk;
#pragma unroll
  for (int b = 0; b <= K; ++b) {
    const int r = w.s + off + b;
    g[b] = ld_row(p, r >= 0 && r < jin);
    p += nk;
  }
  V y[K], g0 = cmake<V>((T)g[0].x, (T)g[0].y);
#pragma unroll
  for (int b = 0; b < K; ++b) {
    const V g1 = cmake<V>((T)g[b + 1].x, (T)g[b + 1].y);
    V r = cmake<V>(T(0), T(0));
    fma2(r, tab[b * QS], g0);
    fma2(r, tab[(K + b) * QS], g1);
    y[b] = r;
    g0 = g1;
  }
  if (w.q == 0 && which == 1) {
#pragma unroll
    for (int m = 1; m <= 4; ++m) fma2(y[0], M4(c.inby, 3, m), cmake<V>((T)g[m].x, (T)g[m].y));
  }
  if (w.q == a.C - 1) {
    V r = cmake<V>(T(0), T(0));
#pragma unroll
    for (int m = 1; m <= 4; ++m) {
      const double2 v = ld_stream(in + (size_t)(jin - m) * nk);
      fma2(r, M4(c.inby, (which == 0 ? 1 : 4), m), cmake<V>((T)v.x, (T)v.y));
    }
#pragma unroll
    for (int b = 0; b < K; ++b) y[b] = select2(b == left - 1, r, y[b]);
  }
  V *ex = reinterpret_cast<V *>(smraw);
  chunk_forward<K, QS, T>(y, tab + 2 * K * QS, P, ex, w.q, w.t, w.L);
  chunk_backward<K, QS, T>(y, tab + 3 * K * QS, tab + 4 * K * QS, P + QS, ex + w.NT, w.q, a.C, w.t, w.L);
  if (!w.active) return;
  V *o = static_cast<V *>(pick3(a.out, f)) + ((size_t)i * ny + w.s) * nk + k;
#pragma unroll
  for (int b = 0; b < K; ++b) {
    if (b < left) *o = y[b];
    o += nk;
  }
}

// ---------------------------------------------------------------------------
// tail of rhsp (rhsp.F90:291-484) for planes 2..nx, one velocity component
// per blockIdx.y, in one pass: each thread reads its K rows of the product,
// the velocity, the difvisxx output, the kz product, the pressure and the RHS
// history once, solves differzy (of the product) and vistyy (of the old
// velocity), assembles the RHS (convective, viscous, pressure gradient),
// applies boun, forms the RK3 combination and the new RHS history, and solves
// implzy for the new velocity. W: element type of the intermediate fields, the
// pressure and the RHS history and of differzy's and vistyy's arithmetic
// (float on the mixed path); everything else is FP64.
// Bound: the fields' bytes in flight. The fields that the row-wise part needs
// are fetched by cp.async to the thread's own slots in shared memory, the
// next tile's as soon as this tile's are used, so they arrive during the
// solves; product and velocity are loaded to registers. FP64: two CTAs of 128
// threads per SM at 255 registers (at 128 and 168 registers the three solves
// spilled or the velocity had to be read twice: 257x97x128 219 and 209 us
// against 156), FP32: three at 168.
// ---------------------------------------------------------------------------
template <typename W>
struct TailArgs {
  double *u, *v, *w;                 // state: old on entry, new on exit
  const W *p;
  W *rhsupa, *rhsvpa, *rhswpa;       // old on entry, new on exit
  const W *cu, *cv, *cw;             // difvisxx outputs
  const W *uv, *uw, *vw, *vv, *ww;
  const W *tw[2];                    // differzy wA, wB, l, d, u; vistyy f1, f2, f3, l, d, u; P, Q of each
  const double *td[2];               // vyi (3), l, d, u of implzy, idyy; P, Q; A_2, C_{jee-1}
  const DState *st;
  int comp[3];
  int C[2], L[2], nw[2], nd[2];      // chunks, lanes, elements of the tables
};
constexpr int kTailW = 11, kTailD = 7;

// copies a coefficient table to shared memory (visible after a CTA barrier)
template <typename T>
__device__ __forceinline__ const T *stage_table(T *dst, const T *src, int n) {
  for (int e = threadIdx.x; e < n; e += blockDim.x) dst[e] = __ldg(src + e);
  return dst;
}

template <int COMP, typename W, int K>
__device__ __forceinline__ void tail_body(const DCoef &c, const DCoefT<W> &cw, const TailArgs<W> &a,
                                          unsigned char *smraw) {
  using VW = V2<W>;
  constexpr int WH = COMP == 1 ? 1 : 0;
  const int nx = c.nx, ny = c.ny, nk = c.nz1 >> 1, C = a.C[WH];
  const int ncm = (nx - 1) * nk;
  YPlace w(a.L[WH], C, K);
  const int q = w.q, s = w.s, t = w.t, L = w.L, NT = w.NT;
  const int jee = COMP == 1 ? ny : ny + 1, krows = COMP == 0 ? ny + 1 : ny, left = jee - s;
  double2 *ex = reinterpret_cast<double2 *>(smraw);
  VW *st = reinterpret_cast<VW *>(ex + 4 * NT) + t;
  const double *td = a.td[WH];
  const W *tw = a.tw[WH];
  if constexpr (!y_table_global(K)) {
    double *sd = reinterpret_cast<double *>(st - t + 5 * K * NT);
    td = stage_table(sd, td, a.nd[WH]);
    tw = stage_table(reinterpret_cast<W *>(sd + a.nd[WH]), tw, a.nw[WH]);
  }
  constexpr bool SLOTS = !y_table_global(K);  // else the rows are read when they are needed
  const double *PD = td + C * kTailD * K;
  const W *PW = tw + C * kTailW * K;
  td += q * kTailD * K;
  tw += q * kTailW * K;
  // the fields that the row-wise part needs, to the thread's slots: cx, kp,
  // p, history, p of the next plane
  auto stage = [&](int tile) {
    w.tile(tile, ncm);
    const int i = w.mc / nk + 2, k = w.mc - (i - 2) * nk;
    const bool last = i == nx;
    const size_t PU = (size_t)(ny + 1) * nk, PV = (size_t)ny * nk, o0 = (size_t)s * nk + k;
    const size_t pl = (size_t)(i - 1) * (COMP == 1 ? PV : PU) + o0, plv = (size_t)(i - 1) * PV + o0;
    const VW *kp = reinterpret_cast<const VW *>(COMP == 0 ? a.uw : (COMP == 1 ? a.vw : a.ww)) + (COMP == 0 ? pl : plv);
    const VW *cx = reinterpret_cast<const VW *>(COMP == 0 ? a.cu : (COMP == 1 ? a.cv : a.cw)) + pl;
    const VW *hp = reinterpret_cast<const VW *>(COMP == 0 ? a.rhsupa : (COMP == 1 ? a.rhsvpa : a.rhswpa)) + pl;
    const VW *pc = reinterpret_cast<const VW *>(a.p) + plv;
#pragma unroll
    for (int b = 0; b < K; ++b) {
      const int r = s + b;
      const size_t o = (size_t)b * nk;
      cp_async_v(st + b * NT, cx + o, r < jee);
      cp_async_v(st + (K + b) * NT, kp + o, !last && r < krows);
      cp_async_v(st + (2 * K + b) * NT, pc + o, r < ny);
      cp_async_v(st + (3 * K + b) * NT, hp + o, r < jee);
      if (COMP == 0) cp_async_v(st + (4 * K + b) * NT, pc + PV + o, !last && r < ny);
    }
    cp_async_commit();
  };
  if (SLOTS && blockIdx.x * L < ncm) stage(blockIdx.x);
  for (int tile = blockIdx.x; tile * L < ncm; tile += gridDim.x) {
    w.tile(tile, ncm);
    const int i = w.mc / nk + 2, k = w.mc - (i - 2) * nk;
    const bool last = i == nx;
    const size_t PU = (size_t)(ny + 1) * nk, PV = (size_t)ny * nk;
    const size_t pl = (size_t)(i - 1) * (COMP == 1 ? PV : PU) + k, plv = (size_t)(i - 1) * PV + k;
    const VW *prod = reinterpret_cast<const VW *>(COMP == 0 ? a.uv : (COMP == 1 ? a.vv : a.vw)) + plv;
    VW *hp = reinterpret_cast<VW *>(COMP == 0 ? a.rhsupa : (COMP == 1 ? a.rhsvpa : a.rhswpa)) + pl;
    const VW *pc = reinterpret_cast<const VW *>(a.p) + plv;
    double2 *vel = reinterpret_cast<double2 *>(COMP == 0 ? a.u : (COMP == 1 ? a.v : a.w)) + pl;
    constexpr int PO = WH == 0 ? -1 : 0;  // product rows s + PO ..
    VW g[K + 1];
    double2 u[K + 2];  // velocity rows s-1 .. s+K
#pragma unroll
    for (int b = 0; b <= K; ++b) {
      const int r = s + PO + b;
      g[b] = ld_row(prod + (ptrdiff_t)r * nk, !last && r >= 0 && r < ny);
    }
#pragma unroll
    for (int b = 0; b < K + 2; ++b) {
      const int r = s - 1 + b;
      u[b] = ld_row(vel + (ptrdiff_t)r * nk, r >= 0 && r < jee);
    }
    VW pk = cmake<VW>(W(0), W(0));  // v: the pressure row after the chunk
    if (COMP == 1) pk = ld_row(pc + (size_t)(s + K) * nk, s + K < ny);
    const double kz = c.kaz[k], kv = c.kvis[k];
    const double var1 = a.st->var1, var3 = a.st->var3, var4 = a.st->var4;
    const double v2 = last ? 0.0 : a.st->var2;
    const double idxx = c.S[OTBL_S_IDXX];
    auto cvw = [](auto x) { return cmake<VW>((W)x.x, (W)x.y); };
    // velocity after the pressure gradient (rhsp.F90:291-339)
    auto star = [&](double2 o, double idyy, VW p0, VW p1) {
      if (COMP == 0) {
        if (!last) {
          o.x = o.x - var1 * idxx * ((double)p1.x - (double)p0.x);
          o.y = o.y - var1 * idxx * ((double)p1.y - (double)p0.y);
        }
      } else if (COMP == 1) {
        o.x = o.x - var1 * idyy * ((double)p1.x - (double)p0.x);
        o.y = o.y - var1 * idyy * ((double)p1.y - (double)p0.y);
      } else {
        const double av = var1 * kz;
        o.x = o.x + av * (double)p0.y;
        o.y = o.y - av * (double)p0.x;
      }
      return o;
    };
    // ---- right-hand sides of differzy and vistyy (table weights are 0 on the
    // boundary rows, whose closures are added)
    __syncthreads();  // the tables are there, the exchange buffers are free
    VW yd[K], yv[K];
    const int chv = WH == 0 ? 3 : 1, ic = WH == 0 ? 3 : 1;
#pragma unroll
    for (int b = 0; b < K; ++b) {
      VW r = cmake<VW>(W(0), W(0));
      fma2(r, tw[b], g[b]);
      fma2(r, tw[K + b], g[b + 1]);
      yd[b] = r;
      r = cmake<VW>(W(0), W(0));
      fma2(r, tw[5 * K + b], cvw(u[b + 2]));
      fma2(r, tw[6 * K + b], cvw(u[b + 1]));
      fma2(r, tw[7 * K + b], cvw(u[b]));
      yv[b] = r;
    }
    if (q == 0) {
#pragma unroll
      for (int m = 1; m <= 4; ++m) {
        fma2(yd[0], M4(cw.dcby, chv, m), g[m - 1 - PO]);
        fma2(yv[0], M4(cw.cofvby, ic, m), cvw(u[m]));
      }
    }
    double2 ubt = make_double2(0.0, 0.0);  // boun's top row (boun.f90:33-55)
    if (left <= K + 1) {                   // the last chunk, or the one before a last chunk of one row
      VW bN = cmake<VW>(W(0), W(0)), top = bN;
      const double *cc = c.ccon;
#pragma unroll
      for (int m = 1; m <= 4; ++m) {
        const double2 o = ld_row(vel + (size_t)(jee - m) * nk, true);
        fma2(bN, M4(cw.cofvby, ic + 1, m), cvw(o));
        fma2(top, M4(cw.dcby, chv + 1, m), ld_row(prod + (size_t)(ny - m) * nk, !last));
        if (COMP != 1 && m > 1) {
          const int r = jee - m;
          const VW p0 = ld_row(pc + (size_t)r * nk, true);
          const VW p1 = ld_row(pc + PV + (size_t)r * nk, COMP == 0 && !last);
          const double2 v = star(o, 0.0, p0, p1);
          ubt.x += M2(cc, 1, m) * v.x;
          ubt.y += M2(cc, 1, m) * v.y;
        }
      }
      if (COMP == 1) {
        ubt.x = k == 0 ? c.vmagic[i - 1] : 0.0;
      } else {
        const double r = -1.0 / M2(cc, 1, 1);
        ubt.x *= r;
        ubt.y *= r;
      }
#pragma unroll
      for (int b = 0; b < K; ++b) {
        yd[b] = select2(b == left - 1, top, yd[b]);
        yv[b] = select2(b == left - 1, bN, yv[b]);
      }
    }
    // ---- both solves
    {
      VW *e0 = reinterpret_cast<VW *>(ex), *e1 = reinterpret_cast<VW *>(ex + NT);
      const W *ld = tw + 2 * K, *lv = tw + 8 * K;
      e0[t] = forward_end<K, 1, W>(yd, ld);
      e1[t] = forward_end<K, 1, W>(yv, lv);
      __syncthreads();
      forward_from<K, 1, W>(yd, ld, chunk_carry<W>(e0 + t - L, -L, PW + q - 1, -1, q));
      forward_from<K, 1, W>(yv, lv, chunk_carry<W>(e1 + t - L, -L, PW + 2 * C + q - 1, -1, q));
      e0 = reinterpret_cast<VW *>(ex + 2 * NT);
      e1 = reinterpret_cast<VW *>(ex + 3 * NT);
      e0[t] = backward_end<K, 1, W>(yd, ld + K, ld + 2 * K);
      e1[t] = backward_end<K, 1, W>(yv, lv + K, lv + 2 * K);
      __syncthreads();
      backward_from<K, 1, W>(yd, ld + K, ld + 2 * K,
                             chunk_carry<W>(e0 + t + L, L, PW + C + q + 1, 1, C - 1 - q));
      backward_from<K, 1, W>(yv, lv + K, lv + 2 * K,
                             chunk_carry<W>(e1 + t + L, L, PW + 3 * C + q + 1, 1, C - 1 - q));
    }
    cp_async_wait<0>();  // the thread's own slots
    // ---- RHS assembly (rhsp.F90:164-169, 181-204, 351-418, 423-445), RK3
    // combination and the new RHS history (rhsp.F90:448-475)
    double2 res[K];
    double2 R1 = make_double2(0.0, 0.0), R2 = R1, R3 = R1, S1 = R1, S2 = R1, S3 = R1;
#pragma unroll
    for (int b = 0; b < K; ++b) {
      {
        const int r = s + b, j = r + 1;
        VW cxv, kpv, p0, hv, p2;
        if constexpr (SLOTS) {
          cxv = st[b * NT], kpv = st[(K + b) * NT], p0 = st[(2 * K + b) * NT], hv = st[(3 * K + b) * NT];
          p2 = COMP == 0 ? st[(4 * K + b) * NT] : (b < K - 1 ? st[(2 * K + (b < K - 1 ? b + 1 : b)) * NT] : pk);
        } else {
          const VW *kp = reinterpret_cast<const VW *>(COMP == 0 ? a.uw : (COMP == 1 ? a.vw : a.ww));
          const VW *cx = reinterpret_cast<const VW *>(COMP == 0 ? a.cu : (COMP == 1 ? a.cv : a.cw));
          const size_t o = (size_t)r * nk;
          cxv = ld_row(cx + pl + o, r < jee);
          kpv = ld_row(kp + (COMP == 0 ? pl : plv) + o, !last && r < krows);
          p0 = ld_row(pc + o, r < ny);
          hv = ld_row(hp + o, r < jee);
          p2 = COMP == 0 ? ld_row(pc + PV + o, !last && r < ny) : ld_row(pc + o + nk, r + 1 < ny);
        }
        const double2 u0 = u[b + 1];
        double2 R = make_double2((double)cxv.x, (double)cxv.y);
        const double2 kzt = make_double2(-kz * (double)kpv.y, kz * (double)kpv.x);
        if (!last) {
          const double2 d1 = make_double2((double)yd[b].x, (double)yd[b].y);
          if (COMP == 0) {
            R.x = (d1.x + kzt.x) + R.x;
            R.y = (d1.y + kzt.y) + R.y;
            if (j >= 2 && j <= ny) {
              R.x = R.x - u0.x * kv;
              R.y = R.y - u0.y * kv;
            }
          } else if (COMP == 1) {
            R.x = ((R.x - u0.x * kv) + kzt.x) + d1.x;
            R.y = ((R.y - u0.y * kv) + kzt.y) + d1.y;
          } else {
            if (j >= 2 && j <= ny) {
              R.x = R.x - u0.x * kv;
              R.y = R.y - u0.y * kv;
            }
            R.x = (R.x + d1.x) + kzt.x;
            R.y = (R.y + d1.y) + kzt.y;
          }
        }
        if (r == jee - 1 || (COMP == 1 && r == 0)) R = make_double2(0.0, 0.0);
        double2 sv = star(u0, COMP == 1 ? td[6 * K + b] : 0.0, p0, p2);
        if (COMP != 1 && b >= 1 && b <= 3) {
          (b == 1 ? R1 : (b == 2 ? R2 : R3)) = R;
          (b == 1 ? S1 : (b == 2 ? S2 : S3)) = sv;
        }
        if (r == jee - 1) sv = ubt;
        if (COMP == 1 && r == 0) sv = make_double2(0.0, 0.0);
        const double2 xv = make_double2((double)yv[b].x, (double)yv[b].y);
        res[b].x = sv.x - (var3 * R.x + v2 * xv.x + var4 * (double)hv.x);
        res[b].y = sv.y - (var3 * R.y + v2 * xv.y + var4 * (double)hv.y);
        if (w.active && r < jee && (COMP == 1 || r > 0)) hp[(size_t)r * nk] = cmake<VW>((W)R.x, (W)R.y);
        if (COMP != 1 && b == 0 && r == 0) res[0] = make_double2((double)hv.x, (double)hv.y);  // finished below
      }
    }
    const bool active = w.active;
    if (SLOTS && (tile + gridDim.x) * L < ncm) stage(tile + gridDim.x);  // the slots are free
    double2 ub1 = make_double2(0.0, 0.0);  // boun's wall row
    if (COMP != 1 && q == 0) {
      const double *ib = c.inby;
      const double f = -1.0 / M4(ib, 2, 1);
      ub1.x = f * (M4(ib, 2, 2) * S1.x + M4(ib, 2, 3) * S2.x + M4(ib, 2, 4) * S3.x);
      ub1.y = f * (M4(ib, 2, 2) * S1.y + M4(ib, 2, 3) * S2.y + M4(ib, 2, 4) * S3.y);
      const double2 R = make_double2(f * (M4(ib, 2, 2) * R1.x + M4(ib, 2, 3) * R2.x + M4(ib, 2, 4) * R3.x),
                                     f * (M4(ib, 2, 2) * R1.y + M4(ib, 2, 3) * R2.y + M4(ib, 2, 4) * R3.y));
      res[0].x = ub1.x - (var3 * R.x + v2 * (double)yv[0].x + var4 * res[0].x);
      res[0].y = ub1.y - (var3 * R.y + v2 * (double)yv[0].y + var4 * res[0].y);
      if (active) hp[0] = cmake<VW>((W)R.x, (W)R.y);
    }
    // ---- implzy (lip.f90:528-597): right-hand side from rows r-1..r+1 of the
    // combination, then the solve; the boundary rows carry ub1, ubt
    ex[t] = res[0];
    ex[NT + t] = res[K - 1];
    __syncthreads();
    {
      double2 rm = q > 0 ? ex[NT + t - L] : make_double2(0.0, 0.0);
      const double2 rn = q < C - 1 ? ex[t + L] : make_double2(0.0, 0.0);
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int r = s + b;
        const double2 rp = b < K - 1 ? res[b < K - 1 ? b + 1 : b] : rn, r0 = res[b];
        double2 v = make_double2(0.0, 0.0);
        fma2(v, td[b], rm);
        fma2(v, td[K + b], r0);
        fma2(v, td[2 * K + b], rp);
        if (r == 0) v = ub1;
        if (r == 1) fma2(v, -PD[2 * C], ub1);
        if (r == jee - 2) fma2(v, -PD[2 * C + 1], ubt);
        if (r == jee - 1) v = ubt;
        res[b] = v;
        rm = r0;
      }
    }
    chunk_forward<K, 1, double>(res, td + 3 * K, PD, ex + 2 * NT, q, t, L);
    chunk_backward<K, 1, double>(res, td + 4 * K, td + 5 * K, PD + C, ex, q, C, t, L);
    if (active) {
#pragma unroll
      for (int b = 0; b < K; ++b)
        if (b < left) vel[(size_t)(s + b) * nk] = res[b];
    }
  }
}

template <typename W, int K>
__global__ void __launch_bounds__(K > 7 ? 256 : 128, K > 7 ? 1 : (sizeof(W) == 8 ? 2 : 3))
    k_tail(DCoef c, DCoefT<W> cw, TailArgs<W> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int comp = pick3(a.comp, blockIdx.y);
  if (comp == 0)
    tail_body<0, W, K>(c, cw, a, smraw);
  else if (comp == 1)
    tail_body<1, W, K>(c, cw, a, smraw);
  else
    tail_body<2, W, K>(c, cw, a, smraw);
}

// ---------------------------------------------------------------------------
// pois.f90:106-117 + soltriy: tridiagonal in y per (x-mode, kz). The LU of
// each (i, k) system depends only on the grid, so its pivots are computed
// once (k_pois_lu) and every substep runs the pre-factored solve.
// ---------------------------------------------------------------------------
// dinv[(i-1)][j-1][k] = 1/pivot_j of the system (i, k), planes i = 2..nx
__global__ void k_pois_lu(DCoef c, double *dinv) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > c.nz2) return;
  const int i = blockIdx.y + 2, ny = c.ny, ny1 = ny - 1, nm = c.nz2 + 1;
  const double *ayp = c.ayp;
  const bool sing = (i == 2 && k == 0);
  auto a2 = [&](int j) {
    if (sing && j == ny1) return 2.0 * A3(ayp, 2, ny1);
    return A3(ayp, 2, j) - c.kaz2[k] - c.kmod[i - 2];
  };
  double *dv = dinv + (size_t)(i - 1) * ny * nm + k;
  double a2p = a2(1);
  for (int j = 2; j <= ny1; ++j) {
    const double d = 1.0 / a2p;
    dv[(size_t)(j - 2) * nm] = d;
    const double l = -A3(ayp, 1, j) * d;
    a2p = a2(j) + l * A3(ayp, 3, j - 1);
  }
  dv[(size_t)(ny1 - 1) * nm] = 1.0 / a2p;
}

// The solve in place on phi rows 0..ny-2 of planes 2..nx: y_r = rhs_r + l_r
// y_{r-1}, l_r = -ayp(1,r+1) dinv(r-1); then x_r = (y_r - ayp(3,r+1)
// x_{r+1}) dinv(r). The singular (i = 2, k = 0) system has its last row
// zeroed first (pois.f90:111-114). The launch takes the modes k0 <= k < k0 +
// nkm of every plane, in T (FP64, or FP32 for the higher spanwise modes of
// the mixed path, with FP32 coefficients and pivots); phi holds T. The chunk
// products differ per mode and are exchanged with the values; the smooth
// modes' products do not decay and take every chunk.
template <typename T, int K>
__global__ void __launch_bounds__(256, 2) k_pois_solve(DCoefT<T> c, T *phi, const T *__restrict__ dinv, int k0,
                                                       int nkm, int C, int L) {
  using V = V2<T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ny = c.ny, ny1 = ny - 1, nk = c.nz1 >> 1;
  YPlace w(L, C, K);
  w.tile(blockIdx.x, (c.nx - 1) * nkm);
  const int i = w.mc / nkm + 2, k = k0 + w.mc - (i - 2) * nkm, s = w.s, t = w.t, q = w.q;
  V *x = reinterpret_cast<V *>(phi) + ((size_t)(i - 1) * ny + s) * nk + k;
  const T *dv = dinv + ((size_t)(i - 1) * ny + s) * nk + k;
  const T *ayp = c.ayp + 3 * s;
  const bool sing = i == 2 && k == 0;
  V y[K];
  T l[K], d[K];
  T dp = q > 0 ? __ldg(dv - nk) : T(0);
#pragma unroll
  for (int b = 0; b < K; ++b) {
    const int r = s + b;
    y[b] = ld_row(x + (size_t)b * nk, r < ny1 && !(sing && r == ny1 - 1));
    d[b] = r < ny1 ? __ldg(dv + (size_t)b * nk) : T(0);
  }
  V *e0 = reinterpret_cast<V *>(smraw), *e1 = e0 + w.NT;
  T *p0 = reinterpret_cast<T *>(e1 + w.NT), *p1 = p0 + w.NT;
  T pr = T(1);
#pragma unroll
  for (int b = 0; b < K; ++b) {
    l[b] = s + b < ny1 ? -__ldg(ayp + 3 * b) * dp : T(0);
    pr *= l[b];
    dp = d[b];
  }
  e0[t] = forward_end<K, 1, T>(y, l);
  p0[t] = pr;
  __syncthreads();
  forward_from<K, 1, T>(y, l, chunk_carry<T>(e0 + t - w.L, -w.L, p0 + t - w.L, -w.L, q));
  pr = T(1);
#pragma unroll
  for (int b = 0; b < K; ++b) {  // l holds u from here on
    l[b] = s + b < ny1 - 1 ? __ldg(ayp + 3 * b + 2) : T(0);
    pr *= -l[b] * d[b];
  }
  e1[t] = backward_end<K, 1, T>(y, d, l);
  p1[t] = pr;
  __syncthreads();
  backward_from<K, 1, T>(y, d, l, chunk_carry<T>(e1 + t + w.L, w.L, p1 + t + w.L, w.L, C - 1 - q));
  if (!w.active) return;
#pragma unroll
  for (int b = 0; b < K; ++b)
    if (s + b < ny1) x[(size_t)b * nk] = y[b];
}

// interpyy and the solve of columns of more than 256 chunks (rows above 3840),
// which no CTA holds: a thread per mode, serial sweeps, the forward one's
// values kept in the output. Only there for their range (the boxes of a step
// end at genflu's 3227 rows).
template <typename T>
__global__ void __launch_bounds__(128) k_interpy_tall(DCoefT<T> c, InterpyArgs a) {
  using V = V2<T>;
  const int f = blockIdx.y, ny = c.ny, nk = c.nz1 >> 1, m = blockIdx.x * 128 + threadIdx.x;
  if (m >= c.nx * nk) return;
  const int i = m / nk, k = m - i * nk, which = pick3(a.which, f), jin = which == 0 ? ny + 1 : ny;
  const double2 *in = reinterpret_cast<const double2 *>(pick3(a.in, f)) + (size_t)i * jin * nk + k;
  V *o = static_cast<V *>(pick3(a.out, f)) + (size_t)i * ny * nk + k;
  const T *lu = which == 0 ? c.inyu : c.inyv, *e = which == 0 ? c.cofiuy : c.cofivy;
  auto g = [&](int r) {
    const double2 v = __ldg(in + (size_t)r * nk);
    return cmake<V>((T)v.x, (T)v.y);
  };
  const int off = which == 0 ? 0 : -1;
  V x = cmake<V>(T(0), T(0));
  for (int r = 0; r < ny; ++r) {
    V y = cmake<V>(T(0), T(0));
    if (r > 0 && r < ny - 1) {
      fma2(y, e[2 * r], g(r + off));
      fma2(y, e[2 * r + 1], g(r + off + 1));
    } else if (r > 0 || which == 1) {
      for (int q = 1; q <= 4; ++q)
        fma2(y, M4(c.inby, (r == 0 ? 3 : (which == 0 ? 1 : 4)), q), g(r == 0 ? q - 1 : jin - q));
    }
    if (r > 0) fma2(y, lu[3 * r], x);
    o[(size_t)r * nk] = x = y;
  }
  for (int r = ny - 1; r >= 0; --r) {
    V y = o[(size_t)r * nk];
    if (r < ny - 1) fma2(y, -lu[3 * r + 2], x);
    x = cmake<V>(lu[3 * r + 1] * y.x, lu[3 * r + 1] * y.y);
    o[(size_t)r * nk] = x;
  }
}

template <typename T>
__global__ void __launch_bounds__(128) k_pois_solve_tall(DCoefT<T> c, T *phi, const T *__restrict__ dinv, int k0,
                                                         int nkm) {
  using V = V2<T>;
  const int ny = c.ny, ny1 = ny - 1, nk = c.nz1 >> 1, m = blockIdx.x * 128 + threadIdx.x;
  if (m >= (c.nx - 1) * nkm) return;
  const int i = m / nkm + 2, k = k0 + m - (i - 2) * nkm;
  V *p = reinterpret_cast<V *>(phi) + (size_t)(i - 1) * ny * nk + k;
  const T *dv = dinv + (size_t)(i - 1) * ny * nk + k, *ayp = c.ayp;
  if (i == 2 && k == 0) p[(size_t)(ny1 - 1) * nk] = cmake<V>(T(0), T(0));
  V x = p[0];
  for (int r = 1; r < ny1; ++r) {
    V y = p[(size_t)r * nk];
    fma2(y, -ayp[3 * r] * dv[(size_t)(r - 1) * nk], x);
    p[(size_t)r * nk] = x = y;
  }
  for (int r = ny1 - 1; r >= 0; --r) {
    V y = p[(size_t)r * nk];
    const T d = dv[(size_t)r * nk];
    if (r < ny1 - 1) fma2(y, -ayp[3 * r + 2], x);
    x = cmake<V>(d * y.x, d * y.y);
    p[(size_t)r * nk] = x;
  }
}

// ---------------------------------------------------------------------------
// tables and launch wrappers
// ---------------------------------------------------------------------------
// Work::ytab in T: interpyy (u-type, v-type), then differzy and vistyy
// (u-type, v-type); Work::tdtab in FP64: implzy (u-type, v-type), whose l, d,
// u and products k_dt writes for the substep's dt
struct YSizes {
  int K, C[2], Ci;            // rows per chunk; chunks of the tail (u-, v-type) and of interpyy
  size_t in, tw[2], td[2];    // elements of each table
  int QS;                     // row stride of interpyy's
};
static YSizes y_sizes(int ny) {
  YSizes z;
  z.K = y_chunk(ny);
  z.Ci = (ny + z.K - 1) / z.K;
  z.QS = z.K == 7 ? 64 : 256;
  z.in = (size_t)(kYInterp * z.K + 2) * z.QS;
  for (int wh = 0; wh < 2; ++wh) {
    z.C[wh] = ((wh ? ny : ny + 1) + z.K - 1) / z.K;
    z.tw[wh] = ytab_elems(z.K, z.C[wh], kTailW, 4);
    z.td[wh] = ytab_elems(z.K, z.C[wh], kTailD, 2);
  }
  return z;
}
size_t ytab_bytes(int ny, bool mixed) {
  const YSizes z = y_sizes(ny);
  return (2 * z.in + z.tw[0] + z.tw[1]) * (mixed ? sizeof(float) : sizeof(double));
}
size_t tdtab_doubles(int ny) {
  const YSizes z = y_sizes(ny);
  return z.td[0] + z.td[1];
}

ImplzyTab implzy_tab(otbl_ctx *c, int which) {
  const YSizes z = y_sizes(c->cfg.ny);
  double *t = c->w.tdtab + (which ? z.td[0] : 0);
  return {t + 3 * z.K, t + (size_t)z.C[which] * kTailD * z.K, z.K, kTailD * z.K, z.C[which]};
}

template <typename T>
static cudaError_t y_tables(otbl_ctx *c) {
  const int ny = c->cfg.ny;
  const YSizes z = y_sizes(ny);
  const int K = z.K;
  otbl_coef_offsets o;
  otbl_coef_layout(c->cfg.nx, ny, c->cfg.nz, &o);
  std::vector<T> cf(c->coef_host.begin(), c->coef_host.end());
  auto A = [&](int id) { return cf.data() + o.off[id]; };
  std::vector<T> all(2 * z.in + z.tw[0] + z.tw[1], T(0));
  T *tab = all.data();
  for (int wh = 0; wh < 2; ++wh, tab += z.in) {
    if (z.Ci > z.QS) continue;  // k_interpy_tall reads the coefficients
    const T *e = A(wh ? OTBL_C_COFIVY : OTBL_C_COFIUY);
    auto put = [&](int i, int r, T v) { tab[(size_t)(i * K + r % K) * z.QS + r / K] = v; };
    for (int r = 1; r < ny - 1; ++r) {
      put(0, r, e[2 * r]);
      put(1, r, e[2 * r + 1]);
    }
    T *P = tab + (size_t)kYInterp * K * z.QS;
    chunk_factors<T>([&](int i, int r, T v) { put(2 + i, r, v); }, K, ny, A(wh ? OTBL_C_INYV : OTBL_C_INYU), 0, P,
                     P + z.QS);
  }
  const int S = kTailW * K;
  auto put = [&](int i, int r, T v) { tab[(size_t)(r / K) * S + i * K + r % K] = v; };
  auto ldu = [&](int at) { return [&put, at](int i, int r, T v) { put(at + i, r, v); }; };
  for (int wh = 0; wh < 2; tab += z.tw[wh], ++wh) {
    const int jee = wh ? ny : ny + 1, C = z.C[wh];
    const T *e = A(wh ? OTBL_C_COFCYV : OTBL_C_COFCYU), *ev = A(wh ? OTBL_C_COFVYV : OTBL_C_COFVYU);
    for (int r = 1; r < jee - 1; ++r) {
      put(0, r, e[2 * r]);
      put(1, r, e[2 * r + 1]);
      for (int k = 0; k < 3; ++k) put(5 + k, r, ev[3 * r + k]);
    }
    T *P = tab + (size_t)C * S;
    chunk_factors<T>(ldu(2), K, jee, A(wh ? OTBL_C_DCYV : OTBL_C_DCYU), 0, P, P + C);
    chunk_factors<T>(ldu(8), K, jee, A(wh ? OTBL_C_VIYV : OTBL_C_VIYU), 0, P + 2 * C, P + 3 * C);
  }
  std::vector<double> dt(z.td[0] + z.td[1], 0.0);
  for (int wh = 0; wh < 2; ++wh) {
    double *td = dt.data() + (wh ? z.td[0] : 0);
    const int jee = wh ? ny : ny + 1;
    const double *vyi = c->coef_host.data() + o.off[wh ? OTBL_C_VYVI : OTBL_C_VYUI];
    const double *idyy = c->coef_host.data() + o.off[OTBL_C_IDYY];
    for (int r = 0; r < jee; ++r) {
      double *row = td + (size_t)(r / K) * kTailD * K + r % K;
      if (r > 0 && r < jee - 1)
        for (int k = 0; k < 3; ++k) row[k * K] = vyi[3 * r + k];
      if (wh && r < ny) row[6 * K] = idyy[r];
    }
  }
  cudaError_t e = cudaMemcpyAsync(c->w.ytab, all.data(), all.size() * sizeof(T), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c->w.tdtab, dt.data(), dt.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream);
  return e == cudaSuccess ? cudaStreamSynchronize(c->stream) : e;
}

cudaError_t prepare_ylines(otbl_ctx *c) { return c->mixed ? y_tables<float>(c) : y_tables<double>(c); }

// tiles of a persistent launch: what `per` CTAs per SM take at once, shared by
// ncomp fields, unless there are fewer
static int y_grid(int ntile, int per, int ncomp) {
  return std::min(ntile, std::max(1, (per * sm_count() + ncomp - 1) / ncomp));
}

template <typename T>
static void interpy_t(otbl_ctx *c, const DCoefT<T> &dc, InterpyArgs &a) {
  const YSizes z = y_sizes(c->cfg.ny);
  for (int wh = 0; wh < 2; ++wh) a.tab[wh] = static_cast<const T *>(c->w.ytab) + wh * z.in;
  a.C = z.Ci;
  if (a.C > 256) {
    k_interpy_tall<T><<<dim3((c->cfg.nx * (c->dc.nz1 / 2) + 127) / 128, 3), 128, 0, c->stream>>>(dc, a);
    return;
  }
  // as wide as the threads allow, or narrower when the autotuner found that
  // faster (tune_bs 128, 64, 32)
  a.L = std::max(1, y_lanes(a.C, 256) * c->tune_bs[2] / 128);
  const int NT = y_threads(a.C, a.L), ncm = c->cfg.nx * (c->dc.nz1 / 2);
  const dim3 gr((ncm + a.L - 1) / a.L, 3);
  const size_t sm = (size_t)2 * NT * sizeof(V2<T>);
  if (z.K == 7)
    k_interpy<T, 7, 64><<<gr, NT, sm, c->stream>>>(dc, a);
  else
    k_interpy<T, 15, 256><<<gr, NT, sm, c->stream>>>(dc, a);
}

cudaError_t launch_interpy(otbl_ctx *c) {
  prof_begin(c, PK_INTERPY);
  if (ydense_ready(c)) {
    const cudaError_t e = launch_interpy_dense(c);
    prof_end(c);
    return e;
  }
  if (stream_interpy(c)) {
    const cudaError_t e = launch_interpy_stream(c);
    prof_end(c);
    c->launches += 1;
    return e;
  }
  InterpyArgs a;
  const double *ins[3] = {c->f[OTBL_F_U], c->f[OTBL_F_W], c->f[OTBL_F_V]};
  void *outs[3] = {c->w.uy, c->w.wy, c->w.vy};
  for (int f = 0; f < 3; ++f) {
    a.in[f] = ins[f];
    a.out[f] = outs[f];
    a.which[f] = f == 2;
  }
  if (c->mixed)
    interpy_t<float>(c, c->dcf, a);
  else
    interpy_t<double>(c, c->dc, a);
  prof_end(c);
  c->launches += 1;
  return cudaGetLastError();
}

// cuTensorMapEncodeTiled from the driver, looked up once (thread-safe
// initialisation of a function-local static); nullptr if unavailable
void *tensor_map_encoder() {
  static void *const fn = []() -> void * {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    cudaGetLastError();
    return p;
  }();
  return fn;
}

template <typename W>
static void tail_t(otbl_ctx *c, const DCoefT<W> &cw, unsigned comps) {
  const YSizes z = y_sizes(c->cfg.ny);
  TailArgs<W> a;
  a.u = c->f[OTBL_F_U];
  a.v = c->f[OTBL_F_V];
  a.w = c->f[OTBL_F_W];
  a.p = reinterpret_cast<const W *>(c->f[OTBL_F_P]);
  a.rhsupa = reinterpret_cast<W *>(c->f[OTBL_F_RHSUPA]);
  a.rhsvpa = reinterpret_cast<W *>(c->f[OTBL_F_RHSVPA]);
  a.rhswpa = reinterpret_cast<W *>(c->f[OTBL_F_RHSWPA]);
  a.cu = static_cast<const W *>(c->w.cu);
  a.cv = static_cast<const W *>(c->w.cv);
  a.cw = static_cast<const W *>(c->w.cw);
  a.uv = static_cast<const W *>(c->w.uv);
  a.uw = static_cast<const W *>(c->w.uw);
  a.vw = static_cast<const W *>(c->w.vw);
  a.vv = static_cast<const W *>(c->w.vv);
  a.ww = static_cast<const W *>(c->w.ww);
  a.st = c->st;
  const bool gt = y_table_global(z.K);
  int NT = 0, lmin = 32, n = 0;
  size_t tabs = 0;
  for (int wh = 0; wh < 2; ++wh) {
    a.tw[wh] = static_cast<const W *>(c->w.ytab) + 2 * z.in + (wh ? z.tw[0] : 0);
    a.td[wh] = c->w.tdtab + (wh ? z.td[0] : 0);
    a.C[wh] = z.C[wh];
    a.nw[wh] = (int)z.tw[wh];
    a.nd[wh] = (int)z.td[wh];
    a.L[wh] = y_lanes(z.C[wh], gt ? 256 : 128);
    lmin = std::min(lmin, a.L[wh]);
    NT = std::max(NT, y_threads(z.C[wh], a.L[wh]));
    if (!gt) tabs = std::max(tabs, z.td[wh] * sizeof(double) + z.tw[wh] * sizeof(W));
  }
  for (int k = 0; k < 3; ++k) a.comp[k] = 0;
  for (int k = 0; k < 3; ++k)
    if (comps & (1u << k)) a.comp[n++] = k;
  const int ncm = (c->cfg.nx - 1) * (c->dc.nz1 / 2), ntile = (ncm + lmin - 1) / lmin;
  const size_t sm = (size_t)4 * NT * 16 + (gt ? 0 : (size_t)5 * z.K * NT * sizeof(V2<W>)) + tabs;
  const int per = std::max(1, std::min((int)(233472 / (sm + 1024)), gt ? 1 : (sizeof(W) == 8 ? 256 : 384) / NT));
  auto go = [&](auto kern) {
    allow_smem(kern, sm);
    kern<<<dim3(y_grid(ntile, per, n), n), NT, sm, c->stream>>>(c->dc, cw, a);
  };
  if (z.K == 7)
    go(k_tail<W, 7>);
  else
    go(k_tail<W, 15>);
}

cudaError_t launch_final(otbl_ctx *c, unsigned comps) {
  prof_begin(c, PK_FINAL);
  if (c->mixed)
    tail_t<float>(c, c->dcf, comps);
  else
    tail_t<double>(c, c->dc, comps);
  prof_end(c);
  c->launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_pois_lu(otbl_ctx *c) {
  dim3 g((c->dc.nz2 + 1 + 127) / 128, c->cfg.nx - 1);
  k_pois_lu<<<g, 128, 0, c->stream>>>(c->dc, c->w.pois_dinv);
  c->launches += 1;
  if (c->mixed) {
    const size_t n = (size_t)c->cfg.nx * c->cfg.ny * (c->dc.nz1 / 2);
    const cudaError_t e = launch_round_f32(c, c->w.pois_dinv, c->w.pois_dinvf, n);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

// modes k0 <= k < k0 + nkm of every plane; phi holds T
template <typename T>
static void pois_solve_t(otbl_ctx *c, const DCoefT<T> &dc, T *phi, const T *dinv, int k0, int nkm) {
  const int K = c->cfg.ny - 1 <= 7 * 64 ? 7 : 15;
  const int C = (c->cfg.ny - 1 + K - 1) / K, L = std::max(1, std::min(32, 224 / C)), NT = y_threads(C, L);
  const int ncm = (c->cfg.nx - 1) * nkm, nb = (ncm + L - 1) / L;
  const size_t sm = (size_t)2 * NT * (sizeof(V2<T>) + sizeof(T));
  if (C > 256)
    k_pois_solve_tall<T><<<(ncm + 127) / 128, 128, 0, c->stream>>>(dc, phi, dinv, k0, nkm);
  else if (K == 7)
    k_pois_solve<T, 7><<<nb, NT, sm, c->stream>>>(dc, phi, dinv, k0, nkm, C, L);
  else
    k_pois_solve<T, 15><<<nb, NT, sm, c->stream>>>(dc, phi, dinv, k0, nkm, C, L);
  c->launches += 1;
}

cudaError_t launch_pois_solve(otbl_ctx *c, double *phi64, float *phi32, int kr_split) {
  const int nk = c->dc.nz1 / 2, ks = kr_split / 2;
  prof_begin(c, PK_POIS_SOLVE);
  if (ks > 0) pois_solve_t<double>(c, c->dc, phi64, c->w.pois_dinv, 0, ks);
  if (ks < nk) pois_solve_t<float>(c, c->dcf, phi32, c->w.pois_dinvf, ks, nk - ks);
  prof_end(c);
  return cudaGetLastError();
}

}  // namespace otbl
