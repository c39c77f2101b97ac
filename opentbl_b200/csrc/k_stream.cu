// The line operators as streams, one thread per line fed by TMA rings: the
// serial Thomas sweeps of lip.f90, forward with a checkpoint every few rows,
// then backward segment by segment, each recomputed from its checkpoint. They
// move 1.5-1.8x the algorithmic bytes, but with hundreds of thousands of lines
// they do it at 4.8-5.9 TB/s of DRAM traffic, and the chunked solves of
// k_xlines.cu and k_ylines.cu, which read each input once, are slower there: a
// CTA cannot hold whole lines of many neighbouring columns, so their rows are
// 64-byte pieces of planes of 0.5 MB, and few warps hide their latency. With
// fewer lines the chunked kernels are the faster ones alone (by 1.1 to 2.5), but
// they fill an SM and leave no room for kernels beside them, so the y-lines of
// well-filled column blocks are streamed on small boxes too. The rules stream_*
// say where, each with both sides measured.
//   k_xline_t            difvisxx, interpxx (mixed path)
//   k_interpy_t          interpyy
//   k_final_ta, tb, s2   the tail of rhsp (rhsp.F90:291-484)
#include <cudaTypedefs.h>

#include <algorithm>
#include <type_traits>

#include "devcommon.cuh"
#include "otbl_internal.cuh"
#include "tma.cuh"

namespace otbl {

// ---------------------------------------------------------------------------
// x-lines
// ---------------------------------------------------------------------------
struct XStream {
  const void *in[3];
  const double *in2[3];  // in2: the second input of difvisxx (velocity)
  void *out[3];
  double *ck[3];         // checkpoint scratch of each line set
  int which[3], np[3];
  CflReset reset;        // interpxx
};

// planes per segment, measured at 1025x193x512: FP64 difvisxx 6 against 4 and
// 8, 42.5, 42.7, 42.7 ms per RK3 step; FP32 8 against 12, 30.8, 30.9
template <typename T, bool DV>
constexpr int xseg() {
  return DV && sizeof(T) == 8 ? 6 : 8;
}

// ---------------------------------------------------------------------------
// A CTA owns TB = 128 consecutive lines of one field; thread 0 loads, for the next segment of K planes, boxes of 32
// lines x K+1 (K+2) planes of each input into a two-stage shared-memory ring
// counted on mbarriers (bounded waits), while every thread runs its line's
// serial sweeps from shared memory. The sequence of segments is the forward
// sweep (0..nseg-1) then the backward one (nseg-1..0). DV: difvisxx (inputs:
// the product, FP32 on the mixed path, and the FP64 velocity) or interpxx
// (input: the FP64 velocity; mixed path only).
// ---------------------------------------------------------------------------
template <typename T, bool DV>
__global__ void __launch_bounds__(128) k_xline_t(DCoefT<T> c, XStream a, int *err, const __grid_constant__ XMaps maps) {
  constexpr int K = xseg<T, DV>(), TB = 128, NB = TB / 32;
  using TG = typename std::conditional<DV, T, double>::type;
  constexpr int GR = K + 1, UR = K + 2;
  constexpr int GBYTES = NB * GR * 32 * (int)sizeof(TG);
  constexpr int GB = (GBYTES + 127) / 128 * 128;
  constexpr int UBYTES = DV ? NB * UR * 32 * 8 : 0;
  constexpr int RCB = K * 16 * (int)sizeof(T);  // the segment's coefficient rows
  constexpr int STG = GB + UBYTES + RCB;
  constexpr unsigned TX = (unsigned)(GBYTES + UBYTES + RCB);
  extern __shared__ __align__(128) unsigned char smraw[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smraw + 2 * STG);
  const int f = blockIdx.y, np = pick3(a.np, f);
  const int t = threadIdx.x, mp0 = blockIdx.x * TB;
  if (!DV && blockIdx.x == 0 && f == 0) a.reset(c.ny);
  if (mp0 >= np) return;  // the whole CTA lies past this field's lines
  const int mp = mp0 + t;
  const bool active = mp < np;
  const int mpc = active ? mp : np - 1;
  const CUtensorMap *mg = f == 0 ? &maps.g[0] : (f == 1 ? &maps.g[1] : &maps.g[2]);
  const CUtensorMap *mu = f == 0 ? &maps.u[0] : (f == 1 ? &maps.u[1] : &maps.u[2]);
  const CUtensorMap *mr = f == 0 ? &maps.r[0] : (f == 1 ? &maps.r[1] : &maps.r[2]);
  const int nx = c.nx, xr = c.xround, which = pick3(a.which, f);
  const int nseg = (nx + K - 1) / K;
  auto seg_of = [&](int it) { return it < nseg ? it : 2 * nseg - 1 - it; };
  auto issue = [&](int stg, int sg) {
    unsigned char *b = smraw + stg * STG;
    const int s0 = sg * K;
    mbar_arrive_expect_tx(&bar[stg], TX);
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      tma_load_2d(b + j * GR * 32 * (int)sizeof(TG), mg, mp0 + 32 * j, DV ? s0 - 1 : s0, &bar[stg]);
      if (DV) tma_load_2d(b + GB + j * UR * 32 * 8, mu, mp0 + 32 * j, s0 - 1, &bar[stg]);
    }
    tma_load_2d(b + GB + UBYTES, mr, 0, s0, &bar[stg]);
  };
  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncthreads();
  if (t == 0) issue(0, 0);
  T *out = static_cast<T *>(pick3(a.out, f)) + mpc;
  T *ck = reinterpret_cast<T *>(pick3(a.ck, f)) + mpc;
  const int gofs = ((t >> 5) * GR) * 32 + (t & 31), uofs = ((t >> 5) * UR) * 32 + (t & 31);
  // ---- operator setup (boundary stencils from global memory)
  T gb0, gbN, ub0 = T(0), ubN = T(0), uN = T(0), uN1 = T(0);
  const T rex = c.S[OTBL_S_REX], idx = c.S[OTBL_S_IDX], uinf = c.S[OTBL_S_UINF];
  if constexpr (DV) {
    const TG *gin = static_cast<const TG *>(pick3(a.in, f)) + mpc;
    const double *uin = pick3(a.in2, f) + mpc;
    const int chv = which == 0 ? 1 : 2, chv1 = chv + 2, ic = which == 0 ? 3 : 1;
    const T *db = c.dcbx, *vb = c.cofvbx;
    auto G = [&](int i) { return (T)rnd(__ldg(gin + (size_t)i * np), xr); };
    auto U = [&](int i) { return (T)rnd(__ldg(uin + (size_t)i * np), xr); };
    gb0 = M5(db, chv, 1) * G(0) + M5(db, chv, 2) * G(1) + M5(db, chv, 3) * G(2) + M5(db, chv, 4) * G(3);
    ub0 = M4(vb, ic, 1) * U(0) + M4(vb, ic, 2) * U(1) + M4(vb, ic, 3) * U(2) + M4(vb, ic, 4) * U(3);
    gbN = M5(db, chv1, 1) * G(nx - 1) + M5(db, chv1, 2) * G(nx - 2) + M5(db, chv1, 3) * G(nx - 3) +
          M5(db, chv1, 4) * G(nx - 4);
    uN = U(nx - 1);
    uN1 = U(nx - 2);
    ubN = M4(vb, ic + 1, 1) * uN + M4(vb, ic + 1, 2) * uN1 + M4(vb, ic + 1, 3) * U(nx - 3) +
          M4(vb, ic + 1, 4) * U(nx - 4);
  } else {
    const double *gin = static_cast<const double *>(pick3(a.in, f)) + mpc;
    const int chi = which == 0 ? 2 : 1, chi2 = which == 0 ? 3 : 4;
    const T *ib = c.inbx;
    auto G = [&](int i) { return (T)rnd(__ldg(gin + (size_t)i * np), xr); };
    gb0 = M4(ib, chi2, 1) * G(0) + M4(ib, chi2, 2) * G(1) + M4(ib, chi2, 3) * G(2) + M4(ib, chi2, 4) * G(3);
    gbN = M4(ib, chi, 1) * G(nx - 1) + M4(ib, chi, 2) * G(nx - 2) + M4(ib, chi, 3) * G(nx - 3) +
          M4(ib, chi, 4) * G(nx - 4);
  }
  // right-hand sides: interpxx e1 g_i + e2 g_{i+1}; difvisxx convective
  // e1 g_{i-1} + e2 g_i and viscous f1 u_{i+1} + f2 u_i + f3 u_{i-1}; q is
  // the plane's coefficient row in shared memory (k_x_rows' layout)
  auto rg = [&](int i, const T *q, T ga, T gb) { return i == 0 ? gb0 : (i == nx - 1 ? gbN : q[0] * ga + q[1] * gb); };
  auto ru = [&](int i, const T *q, T um, T u0, T up) {
    return i == 0 ? ub0 : (i == nx - 1 ? ubN : q[5] * up + q[6] * u0 + q[7] * um);
  };
  T yg = T(0), yu = T(0), xg = T(0), xu = T(0);
  for (int it = 0; it < 2 * nseg; ++it) {
    const int stg = it & 1;
    const bool ok = mbar_wait_bounded(&bar[stg], (it >> 1) & 1, 2000000000ull);
    if (__syncthreads_or(!ok)) {
      if (t == 0) atomicExch(err, OTBL_ERR_TIMEOUT);
      return;
    }
    if (t == 0 && it + 1 < 2 * nseg) issue(stg ^ 1, seg_of(it + 1));
    if (!active) continue;
    const int sg = seg_of(it), s0 = sg * K;
    const unsigned char *bs = smraw + stg * STG;
    const TG *gs = reinterpret_cast<const TG *>(bs) + gofs;
    const double *us = reinterpret_cast<const double *>(bs + GB) + uofs;
    const T *rcs = reinterpret_cast<const T *>(bs + GB + UBYTES);
    auto g = [&](int b) { return (T)rnd(gs[b * 32], xr); };
    auto u = [&](int b) { return (T)rnd(us[b * 32], xr); };
    if (it < nseg) {  // forward sweep, checkpoint at the segment start
      ck[(size_t)((DV ? 2 : 1) * sg) * np] = yg;
      if (DV) ck[(size_t)(2 * sg + 1) * np] = yu;
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int i = s0 + b;
        const T *q = rcs + 16 * b;
        if (i < nx) {
          yg = rg(i, q, g(b), g(b + 1)) + (i > 0 ? q[2] : T(0)) * yg;
          if (DV) yu = ru(i, q, u(b), u(b + 1), u(b + 2)) + (i > 0 ? q[8] : T(0)) * yu;
        }
      }
    } else {  // backward sweep: recompute the segment, then substitute
      T a1 = ck[(size_t)((DV ? 2 : 1) * sg) * np], a2 = DV ? ck[(size_t)(2 * sg + 1) * np] : T(0);
      T y1[K], y2[K];
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int i = s0 + b;
        const T *q = rcs + 16 * b;
        if (i < nx) {
          a1 = rg(i, q, g(b), g(b + 1)) + (i > 0 ? q[2] : T(0)) * a1;
          if (DV) a2 = ru(i, q, u(b), u(b + 1), u(b + 2)) + (i > 0 ? q[8] : T(0)) * a2;
        }
        y1[b] = a1;
        y2[b] = a2;
      }
#pragma unroll
      for (int b = K - 1; b >= 0; --b) {
        const int i = s0 + b;
        const T *q = rcs + 16 * b;
        if (i < nx) {
          xg = (y1[b] - q[4] * xg) * q[3];
          T v = xg;
          if (DV) {
            xu = (y2[b] - q[10] * xu) * q[9];
            v = i == nx - 1 ? uinf * (uN - uN1) * idx + rex * T(0) : xg + rex * xu;
          }
          out[(size_t)i * np] = (T)rnd(v, xr);
        }
      }
    }
  }
}

// One row of 16 T per plane i of each table (dv, which), dv 0 interpxx (mixed
// path) and 1 difvisxx, which 0 u-type and 1 v-type coefficients: the
// right-hand-side weights econ[2i], econ[2i+1] and the LU coefficients
// icon[3i..3i+2], then for difvisxx the viscous operator's econv[3i..3i+2] and
// iconv[3i..3i+2]. k_xline_t's ring stages a segment's rows with its line
// boxes. Entries a plane does not use are 0.
template <typename T>
__global__ void __launch_bounds__(128) k_x_rows(DCoefT<T> c, T *tab) {
  const int nx = c.nx;
  constexpr int dv0 = sizeof(T) == 8;  // the first table's
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (4 - 2 * dv0) * nx) return;
  const int dv = e / (2 * nx) + dv0, which = (e / nx) & 1, i = e % nx;
  T *q = tab + (size_t)e * 16;
  for (int k = 0; k < 16; ++k) q[k] = T(0);
  const T *icon = dv ? (which == 0 ? c.dcxu : c.dcxv) : (which == 0 ? c.inxu : c.inxv);
  const T *econ = dv ? (which == 0 ? c.cofcxu : c.cofcxv) : (which == 0 ? c.cofiux : c.cofivx);
  const bool inner = i > 0 && i < nx - 1;
  if (inner) {
    q[0] = econ[2 * i];
    q[1] = econ[2 * i + 1];
  }
  for (int k = 0; k < 3; ++k) q[2 + k] = icon[3 * i + k];
  if (dv) {
    const T *iconv = which == 0 ? c.vixu : c.vixv, *econv = which == 0 ? c.cofvxu : c.cofvxv;
    for (int k = 0; k < 3; ++k) {
      if (inner) q[5 + k] = econv[3 * i + k];
      q[8 + k] = iconv[3 * i + k];
    }
  }
}

// 2D map of one table of Work::xrowc: [nx planes][16 T], boxes of K planes
static bool encode_xrows(CUtensorMap *m, const void *base, size_t esz, int nx, int k) {
  auto fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encoder());
  if (!fn || ((uintptr_t)base) % 16 != 0) return false;
  const cuuint64_t dims[2] = {16, (cuuint64_t)nx};
  const cuuint64_t strides[1] = {16 * esz};
  const cuuint32_t box[2] = {16, (cuuint32_t)k};
  const cuuint32_t es[2] = {1, 1};
  const CUtensorMapDataType dt = esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return fn(m, dt, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- TMA descriptors (host): field [nx][np], boxes of 32 lines x rows
static bool encode_lines(CUtensorMap *m, const void *base, size_t esz, int nx, int np, int rows) {
  auto fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encoder());
  if (!fn || (np * esz) % 16 != 0 || ((uintptr_t)base) % 16 != 0) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)np, (cuuint64_t)nx};
  const cuuint64_t strides[1] = {(cuuint64_t)np * esz};
  const cuuint32_t box[2] = {32, (cuuint32_t)rows};
  const cuuint32_t es[2] = {1, 1};
  const CUtensorMapDataType dt = esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return fn(m, dt, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool build_x_maps(otbl_ctx *c) {
  const int KI = xseg<float, false>();
  const int KD = c->mixed ? xseg<float, true>() : xseg<double, true>();
  const int nx = c->cfg.nx, nz1 = c->dc.nz1, ny = c->cfg.ny;
  const int np[3] = {nz1 * (ny + 1), nz1 * ny, nz1 * (ny + 1)};
  const double *st[3] = {c->f[OTBL_F_U], c->f[OTBL_F_V], c->f[OTBL_F_W]};
  const void *pr[3] = {c->w.uu, c->w.uv, c->w.uw};
  const size_t ew = c->mixed ? sizeof(float) : sizeof(double);
  bool ok = true;
  const int which[3] = {0, 1, 1};  // u-type or v-type operator of each field
  const char *tab = static_cast<const char *>(c->w.xrowc);
  auto table = [&](int dv, int wh) { return tab + (size_t)(2 * (dv - !c->mixed) + wh) * nx * 16 * ew; };
  for (int f = 0; f < 3 && ok; ++f) {
    if (c->mixed) {
      ok = ok && encode_lines(&c->xmi.g[f], st[f], 8, nx, np[f], KI + 1);
      c->xmi.u[f] = c->xmi.g[f];  // unused by interpxx
      ok = ok && encode_xrows(&c->xmi.r[f], table(0, which[f]), ew, nx, KI);
    }
    ok = ok && encode_lines(&c->xmd.g[f], pr[f], ew, nx, np[f], KD + 1);
    ok = ok && encode_lines(&c->xmd.u[f], st[f], 8, nx, np[f], KD + 2);
    ok = ok && encode_xrows(&c->xmd.r[f], table(1, which[f]), ew, nx, KD);
  }
  c->xmaps_ok = ok;
  return ok;
}

template <typename T, bool DV>
static void xline_t_launch(otbl_ctx *c, const DCoefT<T> &dc, int reset) {
  constexpr int K = xseg<T, DV>();
  using TG = typename std::conditional<DV, T, double>::type;
  const int nz1 = c->dc.nz1, ny = c->cfg.ny, npu = nz1 * (ny + 1), npv = nz1 * ny;
  const double *st[3] = {c->f[OTBL_F_U], c->f[OTBL_F_V], c->f[OTBL_F_W]};
  const void *pr[3] = {c->w.uu, c->w.uv, c->w.uw};
  void *outs[2][3] = {{c->w.ux, c->w.vx, c->w.wx}, {c->w.cu, c->w.cv, c->w.cw}};
  double *cks[3] = {c->w.s1, c->w.s2, c->w.s3};
  XStream a;
  for (int f = 0; f < 3; ++f) {
    a.in[f] = DV ? pr[f] : st[f];
    a.in2[f] = st[f];
    a.out[f] = outs[DV][f];
    a.ck[f] = cks[f];
    a.which[f] = f == 0 ? 0 : 1;
    a.np[f] = f == 1 ? npv : npu;
  }
  if (reset) a.reset = {c->st, c->w.vm_bits};
  const int gb = (4 * (K + 1) * 32 * (int)sizeof(TG) + 127) / 128 * 128;
  const int smem = 2 * (gb + (DV ? 4 * (K + 2) * 32 * 8 : 0) + K * 16 * (int)sizeof(T)) + 128;
  allow_smem(k_xline_t<T, DV>, smem);
  k_xline_t<T, DV><<<dim3((npu + 127) / 128, 3), 128, smem, c->stream>>>(dc, a, &c->st->err, DV ? c->xmd : c->xmi);
}

// Streamed : chunked on B200, us per substep: difvisxx FP64 1025x193x512
// (fields of 541 MB) 1835 : 2253, 865x193x512 (456 MB) 1554 : 1388, 1025x140x512
// (393 MB) 1526 : 1550; mixed the same boxes 1125 : 1361, 975 : 1151, 1038 :
// 889, 1025x96x512 (270 MB) 574 : 516; interpxx mixed 710 : 888, 593 : 783, 485
// : 563, 393 : 313. FP64 interpxx was the slower one streamed at three of
// these four (1195 : 1050, 1000 : 890, 645 : 707, 520 : 420) and is not built.
bool stream_xlines(const otbl_ctx *c, bool dv) {
  const double mb = (double)otbl_field_len(c->cfg.nx, c->cfg.ny, c->cfg.nz, 1) * 8e-6;
  if (!c->xmaps_ok) return false;
  return c->mixed ? mb > (dv ? 420 : 300) : (dv && mb > 500);
}

cudaError_t launch_xlines_stream(otbl_ctx *c, bool dv, int reset) {
  if (c->mixed)
    dv ? xline_t_launch<float, true>(c, c->dcf, 0) : xline_t_launch<float, false>(c, c->dcf, reset);
  else
    xline_t_launch<double, true>(c, c->dc, 0);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// interpyy
// ---------------------------------------------------------------------------
struct StreamYArgs {
  const double *in[3];
  void *out[3];
  double *ck[3];
  int which[3];
};
constexpr int KYT = 8;  // rows per segment

// interpyy fed by TMA: a CTA owns 128 consecutive kr of one plane of one
// field; thread 0 loads, for the next segment of KYT rows, a box of 128 kr x
// KYT+2 rows of the input into a two-stage shared-memory ring on mbarriers
// (bounded waits); the segments run forward (0..nseg-1), then backward.
template <typename T>
__global__ void __launch_bounds__(128) k_interpy_t(DCoefT<T> c, StreamYArgs a, int *err,
                                                   const __grid_constant__ YMaps maps) {
  constexpr int K = KYT, TB = 128, R = K + 2;
  constexpr int RC = K * 8 * (int)sizeof(T);  // the segment's coefficient rows
  constexpr int STG = R * TB * 8 + RC;
  constexpr unsigned TX = (unsigned)STG;
  extern __shared__ __align__(128) unsigned char smraw[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smraw + 2 * STG);
  const int f = blockIdx.z;
  const int ny = c.ny, nz1 = c.nz1, ncol = c.nx * nz1;
  const int t = threadIdx.x, kr0 = blockIdx.x * TB, kr = kr0 + t, i = blockIdx.y + 1;
  const bool active = kr < nz1;
  const int krc = active ? kr : 0;
  const int which = pick3(a.which, f), jin = which == 0 ? ny + 1 : ny;
  const CUtensorMap *mg = f == 0 ? &maps.g[0] : (f == 1 ? &maps.g[1] : &maps.g[2]);
  const CUtensorMap *mr = f == 0 ? &maps.r[0] : (f == 1 ? &maps.r[1] : &maps.r[2]);
  const int nseg = (ny + K - 1) / K;
  auto seg_of = [&](int it) { return it < nseg ? it : 2 * nseg - 1 - it; };
  auto issue = [&](int stg, int sg) {
    mbar_arrive_expect_tx(&bar[stg], TX);
    tma_load_3d(smraw + stg * STG, mg, kr0, sg * K - 1, i - 1, &bar[stg]);
    tma_load_2d(smraw + stg * STG + R * TB * 8, mr, 0, sg * K, &bar[stg]);
  };
  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncthreads();
  if (t == 0) issue(0, 0);
  const size_t S = nz1;
  const int col = (i - 1) * nz1 + krc;
  const double *g = pick3(a.in, f) + (size_t)(i - 1) * jin * nz1 + krc;
  T *o = static_cast<T *>(pick3(a.out, f)) + (size_t)(i - 1) * ny * nz1 + krc;
  T *ck = reinterpret_cast<T *>(pick3(a.ck, f)) + col;
  const T *ib = c.inby;
  auto G = [&](int r) { return (T)__ldg(g + (size_t)min(max(r, 0), jin - 1) * S); };
  T b0 = T(0), bN;
  if (which == 0) {
    bN = M4(ib, 1, 1) * G(ny) + M4(ib, 1, 2) * G(ny - 1) + M4(ib, 1, 3) * G(ny - 2) + M4(ib, 1, 4) * G(ny - 3);
  } else {
    b0 = M4(ib, 3, 1) * G(0) + M4(ib, 3, 2) * G(1) + M4(ib, 3, 3) * G(2) + M4(ib, 3, 4) * G(3);
    bN = M4(ib, 4, 1) * G(ny - 1) + M4(ib, 4, 2) * G(ny - 2) + M4(ib, 4, 3) * G(ny - 3) + M4(ib, 4, 4) * G(ny - 4);
  }
  // q: the row's coefficients in shared memory (k_y_rows' layout)
  auto rhs = [&](int r, const T *q, T gm, T g0, T gp) {
    const T e1 = q[0], e2 = q[1];
    const T in = which == 0 ? e1 * g0 + e2 * gp : e2 * g0 + e1 * gm;
    return r == 0 ? b0 : (r == ny - 1 ? bN : in);
  };
  T y = T(0), x = T(0);
  for (int it = 0; it < 2 * nseg; ++it) {
    const int stg = it & 1;
    const bool ok = mbar_wait_bounded(&bar[stg], (it >> 1) & 1, 2000000000ull);
    if (__syncthreads_or(!ok)) {
      if (t == 0) atomicExch(err, OTBL_ERR_TIMEOUT);
      return;
    }
    if (t == 0 && it + 1 < 2 * nseg) issue(stg ^ 1, seg_of(it + 1));
    if (!active) continue;
    const int sg = seg_of(it), s0 = sg * K;
    const double *gs = reinterpret_cast<const double *>(smraw + stg * STG) + t;
    const T *rcs = reinterpret_cast<const T *>(smraw + stg * STG + R * TB * 8);
    auto gv = [&](int b) { return (T)gs[b * TB]; };  // row s0 - 1 + b
    if (it < nseg) {
      ck[(size_t)sg * ncol] = y;
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int r = s0 + b;
        const T *q = rcs + 8 * b;
        if (r < ny) y = rhs(r, q, gv(b), gv(b + 1), gv(b + 2)) + (r > 0 ? q[2] : T(0)) * y;
      }
    } else {
      T yy = ck[(size_t)sg * ncol], yv[K];
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int r = s0 + b;
        const T *q = rcs + 8 * b;
        if (r < ny) yy = rhs(r, q, gv(b), gv(b + 1), gv(b + 2)) + (r > 0 ? q[2] : T(0)) * yy;
        yv[b] = yy;
      }
#pragma unroll
      for (int b = K - 1; b >= 0; --b) {
        const int r = s0 + b;
        const T *q = rcs + 8 * b;
        if (r < ny) {
          x = (yv[b] - q[4] * x) * q[3];
          o[(size_t)r * S] = x;
        }
      }
    }
  }
}

// One row of 8 values per y row r of each table (which 0: u-type input, u and w;
// 1: v-type input, v): interpyy's right-hand-side weights econ[2r],
// econ[2r+1] and LU coefficients iny[3r..3r+2]; the rest 0. k_interpy_t's
// ring stages a segment's rows with its field box.
template <typename T>
__global__ void __launch_bounds__(128) k_y_rows(DCoefT<T> c, T *tab) {
  const int ny = c.ny;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * ny) return;
  const int which = e / ny, r = e - which * ny;
  const T *iny = which == 0 ? c.inyu : c.inyv, *econ = which == 0 ? c.cofiuy : c.cofivy;
  T *q = tab + (size_t)e * 8;
  q[0] = econ[2 * r];
  q[1] = econ[2 * r + 1];
  for (int k = 0; k < 3; ++k) q[2 + k] = iny[3 * r + k];
  for (int k = 5; k < 8; ++k) q[k] = T(0);
}

// a field [planes][rows][nz1] of element size esz, boxes of 128 x brows x bplanes
static bool encode_field(CUtensorMap *m, const void *base, size_t esz, int planes, int rows, int nz1, int brows,
                         int bplanes) {
  auto fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encoder());
  if (!fn || (nz1 * esz) % 16 != 0 || ((uintptr_t)base) % 16 != 0) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)nz1, (cuuint64_t)rows, (cuuint64_t)planes};
  const cuuint64_t strides[2] = {(cuuint64_t)nz1 * esz, (cuuint64_t)rows * nz1 * esz};
  const cuuint32_t box[3] = {128, (cuuint32_t)brows, (cuuint32_t)bplanes};
  const cuuint32_t es[3] = {1, 1, 1};
  const CUtensorMapDataType dt = esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return fn(m, dt, 3, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2D map of a coefficient table [rows][width elements of esz bytes], boxes
// of brows full rows
static bool encode_table(CUtensorMap *m, const void *base, size_t esz, int width, int rows, int brows) {
  auto fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encoder());
  if (!fn || ((uintptr_t)base) % 16 != 0 || (width * esz) % 16 != 0) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {width * esz};
  const cuuint32_t box[2] = {(cuuint32_t)width, (cuuint32_t)brows};
  const cuuint32_t es[2] = {1, 1};
  const CUtensorMapDataType dt = esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return fn(m, dt, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool build_y_maps(otbl_ctx *c) {
  const int K = KYT;
  const int nx = c->cfg.nx, ny = c->cfg.ny, nz1 = c->dc.nz1;
  const double *in[3] = {c->f[OTBL_F_U], c->f[OTBL_F_W], c->f[OTBL_F_V]};
  const int rows[3] = {ny + 1, ny + 1, ny};
  bool ok = true;
  const int which[3] = {0, 0, 1};
  for (int f = 0; f < 3 && ok; ++f) {
    ok = encode_field(&c->ymi.g[f], in[f], 8, nx, rows[f], nz1, K + 2, 1);
    const size_t ew = c->mixed ? sizeof(float) : sizeof(double);
    const char *tab = reinterpret_cast<const char *>(c->w.yrowc) + (size_t)which[f] * ny * 8 * ew;
    ok = ok && encode_table(&c->ymi.r[f], tab, ew, 8, ny, K);
  }
  c->ymaps_ok = ok;
  return ok;
}

// Streamed : chunked on B200, us. Alone per substep: FP64 1025x193x512 821 :
// 959, 513x129x256 177 : 164, 257x97x128 41 : 35; FP32 660 : 654, 163 : 115, 40 :
// 26. But it runs beside interpxx, so what counts is how much of the GPU it
// takes: steps of one box, and of three boxes issued in turn,
//   FP64 257x97x128 1294 : 1310, 1268 : 1312; 513x129x256 7112 : 7125, 7046 :
//   7197; 81x150x128 1006 : 985, 892 : 911; 33x100x512 1245 : 1248, 909 : 926;
//   1025x193x512 one box 38177 : 38672; nz = 64, whose 42 columns fill a third
//   of a CTA, 385x97x64 1105 : 1086, 1043 : 982
//   FP32, which gains only where the blocks of 128 columns are nearly full:
//   33x100x512 796 : 781, 626 : 676; 257x97x128 1094 : 1081, 1094 : 1085;
//   513x129x256 5149 : 5060, 5894 : 5832; 1025x193x512 26693 : 26700
bool stream_interpy(const otbl_ctx *c) {
  const int nz1 = c->dc.nz1, filled = 100 * nz1 / ((nz1 + 127) / 128 * 128);
  return c->ymaps_ok && (c->mixed ? filled > 85 : nz1 >= 84);
}

template <typename T>
static void interpy_t_launch(otbl_ctx *c, const DCoefT<T> &dc) {
  StreamYArgs a;
  const double *ins[3] = {c->f[OTBL_F_U], c->f[OTBL_F_W], c->f[OTBL_F_V]};
  void *outs[3] = {c->w.uy, c->w.wy, c->w.vy};
  double *cks[3] = {c->w.t1, c->w.t2, c->w.t3};  // interpxx beside it uses s1..s3
  for (int f = 0; f < 3; ++f) {
    a.in[f] = ins[f];
    a.out[f] = outs[f];
    a.ck[f] = cks[f];
    a.which[f] = f == 2;
  }
  const dim3 gt((c->dc.nz1 + 127) / 128, c->cfg.nx, 3);
  const int sm = 2 * ((KYT + 2) * 128 * 8 + KYT * 8 * (int)sizeof(T)) + 128;
  allow_smem(k_interpy_t<T>, sm);
  k_interpy_t<T><<<gt, 128, sm, c->stream>>>(dc, a, &c->st->err, c->ymi);
}

cudaError_t launch_interpy_stream(otbl_ctx *c) {
  if (c->mixed)
    interpy_t_launch<float>(c, c->dcf);
  else
    interpy_t_launch<double>(c, c->dc);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// tail of rhsp (rhsp.F90:291-484) for planes 2..nx, one velocity component
// per launch triple. W: element type of the difvisxx outputs, the products,
// the pressure and the RHS history and of differzy's and vistyy's arithmetic
// (float on the mixed path); everything else is FP64.
//   k_final_ta (rows ascending): the forward sweeps of differzy (of the
//     product) and vistyy (of the old velocity), a checkpoint every KF rows.
//   k_final_tb (segments descending): both forward sweeps recomputed from the
//     checkpoints, both back-substitutions, the RHS assembly, the RK3
//     combination, the new RHS history, the right-hand side of implzy and, in
//     the same descending order, its elimination with the top-down factors of
//     k_dt, written to scratch.
//   k_final_s2 (rows ascending): implzy's substitution and the new velocity.
// KF = 4: the tail 3.47 ms per FP64 substep at 1025x193x512 against 3.73 at 3,
// 3.90 at 2, 3.71 at 5 and 3.82 at 6 (mixed 2.62, 2.77, 2.87, 2.74, 2.72),
// and 3.99 with a three-stage ring.
// ---------------------------------------------------------------------------
constexpr int KFT = 4, NSTG = 2;

template <typename W>
struct FinalArgs {
  double *u, *v, *w;                 // state: old on entry, new on exit
  const W *p;                        // p and the RHS history: W as well
  W *rhsupa, *rhsvpa, *rhswpa;       // old on entry, new on exit
  const W *cu, *cv, *cw;             // difvisxx outputs
  const W *uv, *uw, *vw, *vv, *ww;
  const double *fac_u, *fac_v;
  const DState *st;
};

template <typename W>
struct FinalStream {
  FinalArgs<W> a;
  double *ck;   // checkpoints: [2*seg + op][column]
  double *yq;   // implzy right-hand side after the descending elimination: [q][column]
  double *ub;   // ub1, ubt: [2][column]
};

// implzy substitution x_q = (y_q - A_q x_{q-1}) / B'_q on the eliminated
// right-hand side of k_final_tb (rows q = 0..n-1 are velocity rows q+1),
// then the boundary rows ub1, ubt
template <int COMP>
__global__ void __launch_bounds__(128) k_final_s2(DCoef c, double *u, double *v, double *w, const double *fac_u,
                                                  const double *fac_v, const double *__restrict__ yqb,
                                                  const double *__restrict__ ub) {
  const int nx = c.nx, ny = c.ny, nz1 = c.nz1;
  const int ncol = (nx - 1) * nz1;
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= ncol) return;
  const int i = col / nz1 + 2, kr = col - (i - 2) * nz1;
  const int jee = COMP == 1 ? ny : ny + 1, n = jee - 2;
  const size_t PU = (size_t)(ny + 1) * nz1, PV = (size_t)ny * nz1;
  double *vel = (COMP == 0 ? u : (COMP == 1 ? v : w)) + (size_t)(i - 1) * (COMP == 1 ? PV : PU) + kr;
  const double *fac = COMP == 1 ? fac_v : fac_u;
  const double *yq = yqb + col;
  constexpr int K = 8;
  double x = 0.0;
  for (int q0 = 0; q0 < n; q0 += K) {
    double yv[K];
#pragma unroll
    for (int b = 0; b < K; ++b) yv[b] = yq[(size_t)min(q0 + b, n - 1) * ncol];
#pragma unroll
    for (int b = 0; b < K; ++b) {
      const int q = q0 + b;
      if (q < n) {
        x = (yv[b] - __ldg(fac + 3 * (q + 2)) * x) * __ldg(fac + 3 * (q + 2) + 1);
        vel[(size_t)(q + 1) * nz1] = x;
      }
    }
  }
  vel[0] = ub[col];
  vel[(size_t)(jee - 1) * nz1] = ub[(size_t)ncol + col];
}

// ---------------------------------------------------------------------------
// Pass B. A CTA owns 128 consecutive kr of one
// plane i (one column per thread); thread 0 loads, for the next segment of
// KF rows (descending), one box per field (the product and the velocity on
// rows s0-1..s0+KF, the difvisxx output, the kz product and the RHS history
// on rows s0..s0+KF-1, the pressure rows that component's pressure
// gradient needs)
// into a two-stage shared-memory ring, counted on one mbarrier per stage,
// while all threads work on the current segment from shared memory. Element
// (row b, column t) of a box is at b*128 + t, so each thread's reads are
// conflict-free. Rows outside the field read as 0 and are not used.
// ---------------------------------------------------------------------------
template <typename W, int COMP>
struct FinalBox {
  static constexpr int KF = KFT, T = 128, E = (int)sizeof(W);
  // pressure box: u needs planes i, i+1 on rows s0..s0+KF-1, v rows
  // s0..s0+KF of plane i, w rows s0..s0+KF-1 of plane i
  static constexpr int PR = COMP == 1 ? KF + 1 : KF, PP = COMP == 0 ? 2 : 1;
  static constexpr int r128(int b) { return (b + 127) / 128 * 128; }
  static constexpr int prod = 0;                              // W (KF+2) rows
  static constexpr int vel = prod + r128((KF + 2) * T * E);   // double (KF+2) rows
  static constexpr int cx = vel + (KF + 2) * T * 8;           // W KF rows
  static constexpr int kp = cx + r128(KF * T * E);            // W KF rows
  static constexpr int hp = kp + r128(KF * T * E);            // W KF rows
  static constexpr int p = hp + r128(KF * T * E);             // W PR x PP
  static constexpr int rc = p + r128(PR * PP * T * E);         // KF coefficient rows
  static constexpr int stage = rc + KF * 128;
  static constexpr unsigned tx =
      (unsigned)((KF + 2) * T * E + (KF + 2) * T * 8 + 3 * KF * T * E + PR * PP * T * E + KF * 128);
  static constexpr int NS = NSTG;  // ring stages
  static constexpr int smem = NS * stage + 128;    // the stages and the barriers
};

template <int COMP, typename W>
__global__ void __launch_bounds__(128) k_final_tb(DCoef c, DCoefT<W> cw, FinalStream<W> fs, int *err,
                                                  const __grid_constant__ FinalMaps maps) {
  using B = FinalBox<W, COMP>;
  constexpr int KF = B::KF, TB = B::T;
  extern __shared__ __align__(128) unsigned char smraw[];
  constexpr int NS = B::NS;
  uint64_t *full = reinterpret_cast<uint64_t *>(smraw + NS * B::stage);
  const FinalArgs<W> &a = fs.a;
  const int nx = c.nx, ny = c.ny, nz1 = c.nz1;
  const int ncol = (nx - 1) * nz1;
  const int t = threadIdx.x;
  const int i = blockIdx.y + 2, kr0 = blockIdx.x * TB, kr = kr0 + t;
  const bool active = kr < nz1;
  const int col = (i - 2) * nz1 + kr;
  const int k = kr >> 1, odd = kr & 1;
  const bool last = i == nx;
  const int jee = COMP == 1 ? ny : ny + 1, n = jee - 2;
  const int nseg = (jee + KF - 1) / KF;
  // ---- the ring: thread 0 initialises the barriers and loads segment nseg-1
  auto issue = [&](int stg, int sg) {
    unsigned char *b = smraw + stg * B::stage;
    const int s0 = sg * KF;
    mbar_arrive_expect_tx(&full[stg], B::tx);
    tma_load_3d(b + B::prod, &maps.prod, kr0, s0 - 1, i - 1, &full[stg]);
    tma_load_3d(b + B::vel, &maps.vel, kr0, s0 - 1, i - 1, &full[stg]);
    tma_load_3d(b + B::cx, &maps.cx, kr0, s0, i - 1, &full[stg]);
    tma_load_3d(b + B::kp, &maps.kp, kr0, s0, i - 1, &full[stg]);
    tma_load_3d(b + B::hp, &maps.hp, kr0, s0, i - 1, &full[stg]);
    tma_load_3d(b + B::p, &maps.p, kr0, s0, i - 1, &full[stg]);
    tma_load_2d(b + B::rc, &maps.rc, 0, s0, &full[stg]);
  };
  if (t == 0) {
    for (int q = 0; q < NS; ++q) mbar_init(&full[q], 1);
    mbar_init_fence();
  }
  __syncthreads();
  if (t == 0)  // the first NS-1 segments (descending)
    for (int q = 0; q < NS - 1 && q < nseg; ++q) issue(q, nseg - 1 - q);
  // ---- per-column setup
  const int pof = odd ? -1 : 1;
  const size_t PU = (size_t)(ny + 1) * nz1, PV = (size_t)ny * nz1;
  const size_t pl = (size_t)(i - 1) * (COMP == 1 ? PV : PU), plv = (size_t)(i - 1) * PV;
  const size_t S = nz1;
  const int krc = active ? kr : 0;  // inactive threads read a valid column and write nothing
  const W *prod = (COMP == 0 ? a.uv : (COMP == 1 ? a.vv : a.vw)) + plv + krc;
  const double *vel = (COMP == 0 ? a.u : (COMP == 1 ? a.v : a.w)) + pl + krc;
  W *hp = (COMP == 0 ? a.rhsupa : (COMP == 1 ? a.rhsvpa : a.rhswpa)) + pl + krc;
  const W *pc = a.p + plv + krc;
  const double kz = c.kaz[k], kv = c.kvis[k];
  const double var1 = a.st->var1, var3 = a.st->var3, var4 = a.st->var4;
  const double v2 = last ? 0.0 : a.st->var2;
  const double idxx = c.S[OTBL_S_IDXX];
  const double *ib = c.inby, *cc = c.ccon;
  const double sgn = odd ? 1.0 : -1.0;
  const int which = COMP == 1 ? 1 : 0;
  // differzy and vistyy run in W on the coefficient copy cw (FP32 on the
  // mixed path); the RHS assembly, RK3 combination and implzy in FP64
  // (per-row coefficients: k_tail_rows' rows, staged with each segment)
  const double *fac = COMP == 1 ? a.fac_v : a.fac_u;
  auto Pg = [&](int r) { return (double)__ldg(prod + (size_t)min(max(r, 0), ny - 1) * S); };
  auto Vg = [&](int r) { return __ldg(vel + (size_t)min(max(r, 0), jee - 1) * S); };
  // velocity after the pressure gradient (rhsp.F90:291-339), from global
  // memory (boundary rows) ...
  auto star_g = [&](int r, double o) -> double {
    const int rp = min(r, ny - 1);
    if (COMP == 0)
      return last ? o
                  : o - var1 * idxx * ((double)__ldg(pc + PV + (size_t)rp * S) - (double)__ldg(pc + (size_t)rp * S));
    if (COMP == 1)
      return o - var1 * c.idyy[r] *
                     ((double)__ldg(pc + (size_t)min(r + 1, ny - 1) * S) - (double)__ldg(pc + (size_t)rp * S));
    const double pp = (double)__ldg(pc + (size_t)rp * S + pof);
    const double av = var1 * kz;
    return o - (odd ? av * pp : -av * pp);
  };
  const int chv = which == 0 ? 3 : 1, cha = chv + 1, ic = which == 0 ? 3 : 1;
  const W *db = cw.dcby, *vb = cw.cofvby;
  W bot = W(0), top = W(0);
  if (!last) {
    bot = M4(db, chv, 1) * (W)Pg(0) + M4(db, chv, 2) * (W)Pg(1) + M4(db, chv, 3) * (W)Pg(2) + M4(db, chv, 4) * (W)Pg(3);
    top = M4(db, cha, 1) * (W)Pg(ny - 1) + M4(db, cha, 2) * (W)Pg(ny - 2) + M4(db, cha, 3) * (W)Pg(ny - 3) +
          M4(db, cha, 4) * (W)Pg(ny - 4);
  }
  const W b0 = M4(vb, ic, 1) * (W)Vg(0) + M4(vb, ic, 2) * (W)Vg(1) + M4(vb, ic, 3) * (W)Vg(2) + M4(vb, ic, 4) * (W)Vg(3);
  const W bN = M4(vb, ic + 1, 1) * (W)Vg(jee - 1) + M4(vb, ic + 1, 2) * (W)Vg(jee - 2) +
               M4(vb, ic + 1, 3) * (W)Vg(jee - 3) + M4(vb, ic + 1, 4) * (W)Vg(jee - 4);
  double ub1 = 0.0, ubt = 0.0;
  if (COMP == 1) {
    ubt = kr == 0 ? c.vmagic[i - 1] : 0.0;
  } else {
    const double s2 = star_g(1, Vg(1)), s3 = star_g(2, Vg(2)), s4 = star_g(3, Vg(3));
    const double sn = star_g(ny - 1, Vg(ny - 1)), sn1 = star_g(ny - 2, Vg(ny - 2)), sn2 = star_g(ny - 3, Vg(ny - 3));
    ub1 = -1.0 / M4(ib, 2, 1) * (M4(ib, 2, 2) * s2 + M4(ib, 2, 3) * s3 + M4(ib, 2, 4) * s4);
    ubt = -1.0 / M2(cc, 1, 1) * (M2(cc, 1, 2) * sn + M2(cc, 1, 3) * sn1 + M2(cc, 1, 4) * sn2);
  }
  // q: the row's W coefficients in shared memory (k_tail_rows' layout)
  auto rd = [&](int r, const W *q, W gm, W g0, W gp) {
    const W in = which == 0 ? q[1] * g0 + q[0] * gm : q[1] * gp + q[0] * g0;
    return r == 0 ? bot : (r == jee - 1 ? top : in);
  };
  auto rv = [&](int r, const W *q, W um, W u0, W up) {
    const W in = q[5] * up + q[6] * u0 + q[7] * um;
    return r == 0 ? b0 : (r == jee - 1 ? bN : in);
  };
  const W *ck = reinterpret_cast<const W *>(fs.ck) + (active ? col : 0);
  double *yq = fs.yq + (active ? col : 0);
  const double a1raw = fac[3 * (jee + 1)], a3raw = fac[3 * (jee + 1) + 1];
  W xd = W(0), xv = W(0);
  double R1 = 0.0, R2 = 0.0, R3 = 0.0;
  double res1 = 0.0, res2 = 0.0;
  double yel = 0.0;
  W ckd = ck[(size_t)(2 * (nseg - 1)) * ncol], ckv = ck[(size_t)(2 * (nseg - 1) + 1) * ncol];
  const int tk = t ^ 1;  // kr+1 for even kr, kr-1 for odd kr (the chunk starts even)
  for (int sg = nseg - 1, it = 0; sg >= 0; --sg, ++it) {
    const int stg = it % NS;
    const bool ok = mbar_wait_bounded(&full[stg], (it / NS) & 1, 2000000000ull);
    if (__syncthreads_or(!ok)) {  // the stage of iteration it-1 is free from here on
      if (t == 0) atomicExch(err, OTBL_ERR_TIMEOUT);
      return;
    }
    if (t == 0 && sg >= NS - 1) issue((it + NS - 1) % NS, sg - (NS - 1));
    const int s0 = sg * KF;
    const unsigned char *bs = smraw + stg * B::stage;
    const W *sp = reinterpret_cast<const W *>(bs + B::prod);
    const double *sv = reinterpret_cast<const double *>(bs + B::vel);
    const W *sc = reinterpret_cast<const W *>(bs + B::cx);
    const W *sk = reinterpret_cast<const W *>(bs + B::kp);
    const W *sh = reinterpret_cast<const W *>(bs + B::hp);
    const W *spp = reinterpret_cast<const W *>(bs + B::p);
    const double *rcs = reinterpret_cast<const double *>(bs + B::rc);
    W ad = ckd, av = ckv;
    if (sg >= 1) {  // next segment's checkpoints, ahead of use
      ckd = ck[(size_t)(2 * (sg - 1)) * ncol];
      ckv = ck[(size_t)(2 * (sg - 1) + 1) * ncol];
    }
    if (!active) continue;
    W ydv[KF], yvv[KF];
#pragma unroll
    for (int b = 0; b < KF; ++b) {
      const int r = s0 + b;
      const W *q = reinterpret_cast<const W *>(rcs + 16 * b + 5);
      if (r < jee) {
        if (!last)
          ad = rd(r, q, sp[b * TB + t], sp[(b + 1) * TB + t], sp[(b + 2) * TB + t]) + (r > 0 ? q[2] : W(0)) * ad;
        av = rv(r, q, (W)sv[b * TB + t], (W)sv[(b + 1) * TB + t], (W)sv[(b + 2) * TB + t]) +
             (r > 0 ? q[8] : W(0)) * av;
      }
      ydv[b] = ad;
      yvv[b] = av;
    }
#pragma unroll
    for (int b = KF - 1; b >= 0; --b) {
      const int r = s0 + b, j = r + 1;
      if (r >= jee) continue;
      const double *rq = rcs + 16 * b;
      const W *q = reinterpret_cast<const W *>(rq + 5);
      if (!last) xd = (ydv[b] - q[4] * xd) * q[3];
      xv = (yvv[b] - q[10] * xv) * q[9];
      // RHS assembly (rhsp.F90:164-169, 181-204, 351-418, 423-445)
      const double d1 = last ? 0.0 : (double)xd;
      const double u0 = sv[(b + 1) * TB + t];
      double R = (double)sc[b * TB + t];
      const double kzt = sgn * kz * ((!last && (COMP != 2 || r < ny)) ? (double)sk[b * TB + tk] : 0.0);
      if (COMP == 0) {
        if (!last) {
          R = (d1 + kzt) + R;
          if (j >= 2 && j <= ny) R = R - u0 * kv;
        }
      } else if (COMP == 1) {
        if (!last) {
          if (j >= 2 && j <= ny - 1) R = R - u0 * kv;
          R = R + kzt;
          R = R + d1;
        }
        if (j == 1 || j == ny) R = 0.0;
      } else {
        if (!last) {
          if (j >= 2 && j <= ny) R = R - u0 * kv;
          R = R + d1;
          if (j <= ny) R = R + kzt;
        }
      }
      if (COMP != 1) {  // wall and top rows of the u,w RHS (rhsp.F90:438-442)
        if (r == jee - 1) R = 0.0;
        if (r == 0) R = -1.0 / M4(ib, 2, 1) * (M4(ib, 2, 2) * R1 + M4(ib, 2, 3) * R2 + M4(ib, 2, 4) * R3);
        if (r == 3) R3 = R;
        if (r == 2) R2 = R;
        if (r == 1) R1 = R;
      }
      // RK3 combination and the new RHS history (rhsp.F90:448-475); rows
      // 1..jee-2 of the pressure box (no clamp needed there)
      double st;
      if (r == 0) {
        st = ub1;
      } else if (r == jee - 1) {
        st = ubt;
      } else if (COMP == 0) {
        st = last ? u0 : u0 - var1 * idxx * ((double)spp[(B::PR + b) * TB + t] - (double)spp[b * TB + t]);
      } else if (COMP == 1) {
        st = u0 - var1 * rq[4] * ((double)spp[(b + 1) * TB + t] - (double)spp[b * TB + t]);
      } else {
        const double pp = (double)spp[b * TB + tk];
        const double avz = var1 * kz;
        st = u0 - (odd ? avz * pp : -avz * pp);
      }
      const double res = st - (var3 * R + v2 * (double)xv + var4 * (double)sh[b * TB + t]);
      hp[(size_t)r * S] = (W)R;
      if (r < n) {
        double v = rq[1] * res + rq[2] * res1 + rq[3] * res2;
        if (r == 0) v = v - a1raw * ub1;
        if (r == n - 1) v = v - a3raw * ubt;
        yel = v + rq[0] * yel;
        yq[(size_t)r * ncol] = yel;
      }
      res2 = res1;
      res1 = res;
    }
  }
  if (active) {
    fs.ub[col] = ub1;
    fs.ub[(size_t)ncol + col] = ubt;
  }
}

// Pass A: the same ring as k_final_tb, ascending,
// with boxes of 128 columns x KA+2 rows of the product and the velocity
// (KA = 8 rows per stage); the checkpoints are still written every KF rows
// of k_final_tb's segments.
template <int COMP, typename W>
__global__ void __launch_bounds__(128) k_final_ta(DCoef c, DCoefT<W> cw, FinalStream<W> fs, int *err,
                                                  const __grid_constant__ FinalMaps maps) {
  constexpr int KF = KFT, KA = 8, TB = 128, R = KA + 2;
  constexpr int PB = (R * TB * (int)sizeof(W) + 127) / 128 * 128;
  constexpr int STG = PB + R * TB * 8 + KA * 128;  // + the KA coefficient rows
  constexpr unsigned TX = (unsigned)(R * TB * sizeof(W) + R * TB * 8 + KA * 128);
  extern __shared__ __align__(128) unsigned char smraw[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smraw + 2 * STG);
  const FinalArgs<W> &a = fs.a;
  const int nx = c.nx, ny = c.ny, nz1 = c.nz1;
  const int ncol = (nx - 1) * nz1;
  const int t = threadIdx.x;
  const int i = blockIdx.y + 2, kr0 = blockIdx.x * TB, kr = kr0 + t;
  const bool active = kr < nz1;
  const int krc = active ? kr : 0;
  const int col = (i - 2) * nz1 + krc;
  const bool last = i == nx;
  const int jee = COMP == 1 ? ny : ny + 1;
  const int nst = (jee + KA - 1) / KA;
  auto issue = [&](int stg, int sa) {
    unsigned char *b = smraw + stg * STG;
    mbar_arrive_expect_tx(&bar[stg], TX);
    tma_load_3d(b, &maps.prod_a, kr0, sa * KA - 1, i - 1, &bar[stg]);
    tma_load_3d(b + PB, &maps.vel_a, kr0, sa * KA - 1, i - 1, &bar[stg]);
    tma_load_2d(b + PB + R * TB * 8, &maps.rc_a, 0, sa * KA, &bar[stg]);
  };
  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  __syncthreads();
  if (t == 0) issue(0, 0);
  const size_t PU = (size_t)(ny + 1) * nz1, PV = (size_t)ny * nz1;
  const size_t pl = (size_t)(i - 1) * (COMP == 1 ? PV : PU), plv = (size_t)(i - 1) * PV;
  const size_t S = nz1;
  const W *prod = (COMP == 0 ? a.uv : (COMP == 1 ? a.vv : a.vw)) + plv + krc;
  const double *vel = (COMP == 0 ? a.u : (COMP == 1 ? a.v : a.w)) + pl + krc;
  const int which = COMP == 1 ? 1 : 0;
  // the sweeps run in W on the coefficient copy cw (FP32 on the mixed path);
  // the per-row coefficients come staged with the boxes (k_tail_rows' rows)
  auto Pg = [&](int r) { return (W)__ldg(prod + (size_t)min(max(r, 0), ny - 1) * S); };
  auto Vg = [&](int r) { return (W)__ldg(vel + (size_t)min(max(r, 0), jee - 1) * S); };
  const int chv = which == 0 ? 3 : 1, cha = chv + 1, ic = which == 0 ? 3 : 1;
  const W *db = cw.dcby, *vb = cw.cofvby;
  W bot = W(0), top = W(0);
  if (!last) {
    bot = M4(db, chv, 1) * Pg(0) + M4(db, chv, 2) * Pg(1) + M4(db, chv, 3) * Pg(2) + M4(db, chv, 4) * Pg(3);
    top = M4(db, cha, 1) * Pg(ny - 1) + M4(db, cha, 2) * Pg(ny - 2) + M4(db, cha, 3) * Pg(ny - 3) +
          M4(db, cha, 4) * Pg(ny - 4);
  }
  const W b0 = M4(vb, ic, 1) * Vg(0) + M4(vb, ic, 2) * Vg(1) + M4(vb, ic, 3) * Vg(2) + M4(vb, ic, 4) * Vg(3);
  const W bN = M4(vb, ic + 1, 1) * Vg(jee - 1) + M4(vb, ic + 1, 2) * Vg(jee - 2) +
               M4(vb, ic + 1, 3) * Vg(jee - 3) + M4(vb, ic + 1, 4) * Vg(jee - 4);
  auto rd = [&](int r, const W *q, W gm, W g0, W gp) {
    const W in = which == 0 ? q[1] * g0 + q[0] * gm : q[1] * gp + q[0] * g0;
    return r == 0 ? bot : (r == jee - 1 ? top : in);
  };
  auto rv = [&](int r, const W *q, W um, W u0, W up) {
    const W in = q[5] * up + q[6] * u0 + q[7] * um;
    return r == 0 ? b0 : (r == jee - 1 ? bN : in);
  };
  W *ck = reinterpret_cast<W *>(fs.ck) + col;  // checkpoints in W, read back by k_final_tb
  W yd = W(0), yv = W(0);
  for (int sa = 0; sa < nst; ++sa) {
    const int stg = sa & 1;
    const bool ok = mbar_wait_bounded(&bar[stg], (sa >> 1) & 1, 2000000000ull);
    if (__syncthreads_or(!ok)) {
      if (t == 0) atomicExch(err, OTBL_ERR_TIMEOUT);
      return;
    }
    if (t == 0 && sa + 1 < nst) issue(stg ^ 1, sa + 1);
    if (!active) continue;
    const W *sp = reinterpret_cast<const W *>(smraw + stg * STG) + t;
    const double *sv = reinterpret_cast<const double *>(smraw + stg * STG + PB) + t;
    const double *rcs = reinterpret_cast<const double *>(smraw + stg * STG + PB + R * TB * 8);
    const int s0 = sa * KA;
#pragma unroll
    for (int b = 0; b < KA; ++b) {
      const int r = s0 + b;
      const W *q = reinterpret_cast<const W *>(rcs + 16 * b + 5);
      if (r % KF == 0 && r < jee) {  // y of row r-1 at the start of segment r/KF
        ck[(size_t)(2 * (r / KF)) * ncol] = yd;
        ck[(size_t)(2 * (r / KF) + 1) * ncol] = yv;
      }
      if (r < jee) {
        if (!last) yd = rd(r, q, sp[b * TB], sp[(b + 1) * TB], sp[(b + 2) * TB]) + (r > 0 ? q[2] : W(0)) * yd;
        yv = rv(r, q, (W)sv[b * TB], (W)sv[(b + 1) * TB], (W)sv[(b + 2) * TB]) + (r > 0 ? q[8] : W(0)) * yv;
      }
    }
  }
}

template <typename W>
static bool build_maps_t(otbl_ctx *c) {
  constexpr int KF = KFT;
  const int nx = c->cfg.nx, ny = c->cfg.ny, nz1 = c->dc.nz1;
  const size_t ew = sizeof(W);
  bool ok = nz1 >= 2;
  for (int comp = 0; comp < 3 && ok; ++comp) {
    FinalMaps &m = c->fmaps[comp];
    const int jee = comp == 1 ? ny : ny + 1;
    const void *prod = comp == 0 ? c->w.uv : (comp == 1 ? c->w.vv : c->w.vw);
    const void *kp = comp == 0 ? c->w.uw : (comp == 1 ? c->w.vw : c->w.ww);
    const int kprows = comp == 0 ? ny + 1 : ny;
    const double *vel = c->f[comp == 0 ? OTBL_F_U : (comp == 1 ? OTBL_F_V : OTBL_F_W)];
    const void *cx = comp == 0 ? c->w.cu : (comp == 1 ? c->w.cv : c->w.cw);
    const void *hp = c->f[comp == 0 ? OTBL_F_RHSUPA : (comp == 1 ? OTBL_F_RHSVPA : OTBL_F_RHSWPA)];
    ok = ok && encode_field(&m.prod, prod, ew, nx, ny, nz1, KF + 2, 1);
    ok = ok && encode_field(&m.prod_a, prod, ew, nx, ny, nz1, 8 + 2, 1);
    ok = ok && encode_field(&m.vel_a, vel, 8, nx, jee, nz1, 8 + 2, 1);
    ok = ok && encode_field(&m.kp, kp, ew, nx, kprows, nz1, KF, 1);
    ok = ok && encode_field(&m.vel, vel, 8, nx, jee, nz1, KF + 2, 1);
    ok = ok && encode_field(&m.cx, cx, ew, nx, jee, nz1, KF, 1);
    ok = ok && encode_field(&m.hp, hp, ew, nx, jee, nz1, KF, 1);
    ok = ok && encode_field(&m.p, c->f[OTBL_F_P], ew, nx, ny, nz1, comp == 1 ? KF + 1 : KF, comp == 0 ? 2 : 1);
    ok = ok && encode_table(&m.rc, c->w.rowc + (comp == 1 ? (size_t)16 * (ny + 2) : 0), 8, 16, ny + 2, KF);
    ok = ok && encode_table(&m.rc_a, c->w.rowc + (comp == 1 ? (size_t)16 * (ny + 2) : 0), 8, 16, ny + 2, 8);
  }
  return ok;
}

// One 128-byte row per y row r and tail kind (table 0: the u and w tails,
// u-type coefficients; table 1: the v tail): the FP64 values fac[3(r+2)+2]
// (the implzy factor of the descending elimination), vyi[3(r+1)+0..2] and
// idyy[r], then in W ecd[2r+0..1], dcy[3r+0..2], ecv[3r+0..2],
// viy[3r+0..2] (differzy's and vistyy's right-hand-side and LU
// coefficients). k_final_tb's ring stages a segment's rows with its field
// boxes, so its sweeps read them from shared memory as broadcasts. Entries
// that a row does not use are 0.
template <typename W>
__global__ void __launch_bounds__(128) k_tail_rows(DCoef c, DCoefT<W> cw, const double *fac_u, const double *fac_v,
                                                   double *rowc) {
  const int ny = c.ny, R = ny + 2;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * R) return;
  const int which = e / R, r = e - which * R;
  const int jee = which == 1 ? ny : ny + 1, n = jee - 2;
  double *row = rowc + (size_t)e * 16;
  const double *fac = which == 1 ? fac_v : fac_u;
  const double *vyi = which == 0 ? c.vyui : c.vyvi;
  row[0] = r < n ? fac[3 * (r + 2) + 2] : 0.0;
  for (int q = 0; q < 3; ++q) row[1 + q] = r < n ? vyi[3 * (r + 1) + q] : 0.0;
  row[4] = (which == 1 && r < ny) ? c.idyy[r] : 0.0;
  W *q = reinterpret_cast<W *>(row + 5);
  constexpr int NW = (int)((128 - 5 * sizeof(double)) / sizeof(W));
  for (int k = 0; k < NW; ++k) q[k] = W(0);
  if (r < jee) {
    const W *dcy = which == 0 ? cw.dcyu : cw.dcyv, *ecd = which == 0 ? cw.cofcyu : cw.cofcyv;
    const W *viy = which == 0 ? cw.viyu : cw.viyv, *ecv = which == 0 ? cw.cofvyu : cw.cofvyv;
    q[0] = ecd[2 * r];
    q[1] = ecd[2 * r + 1];
    for (int k = 0; k < 3; ++k) {
      q[2 + k] = dcy[3 * r + k];
      q[5 + k] = ecv[3 * r + k];
      q[8 + k] = viy[3 * r + k];
    }
  }
}

cudaError_t launch_tail_rows(otbl_ctx *c) {
  const int n = 2 * (c->cfg.ny + 2);
  if (c->mixed)
    k_tail_rows<float><<<(n + 127) / 128, 128, 0, c->stream>>>(c->dc, c->dcf, c->w.fac_u, c->w.fac_v, c->w.rowc);
  else
    k_tail_rows<double><<<(n + 127) / 128, 128, 0, c->stream>>>(c->dc, c->dc, c->w.fac_u, c->w.fac_v, c->w.rowc);
  c->launches += 1;
  return cudaGetLastError();
}

// Streamed : chunked on B200, us. The kernels alone per substep:
// 1025x193x512 (174 thousand modes) FP64 3470 : 4863, mixed 2625 : 3368;
// 1025x140x512 2557 : 3168, mixed 1916 : 2171; 257x193x512 (44 thousand) 1053 :
// 1226, mixed 838 : 870; 513x129x256 (44 thousand) 882 : 827; 1025x48x512 mixed
// 754 : 611; 513x65x128 (22 thousand) 311 : 182, mixed 222 : 146; 257x97x128
// 277 : 163, mixed 264 : 116. But the chunked tail's CTAs fill an SM's
// registers, so that no other kernel runs beside it: steps of one box, and of
// three boxes issued in turn (/ three with the tail that both replaced):
//   mixed 65x150x512 2048 : 2105, 1558 : 1778 / 1574; 97x133x512 2440 : 2319,
//   2076 : 2392 / 2010; 193x150x512 4500 : 4781, 4379 : 5448 / 4209; 321x97x512
//   4582 : 4475, 4571 : 5160 / 4413; 33x100x512 (5 thousand modes) 1006 : 793,
//   646 : 627 / 722
//   FP64 65x92x256 1102 : 1024, 782 : 855 / 778; 193x73x256 1802 : 1742, 1681 :
//   1793 / 1646; 193x150x256 3452 : 3620, 3214 : 3654 / 3313; 513x129x256 6662 :
//   7120, 6532 : 7019 / 7116; 33x60x256 580 : 374, 337 : 292 / 388; 1025x60x256
//   6571 : 6225, 6475 : 6385 / 7174; 33x100x512 1240 : 1123, 909 : 962 / 916
//   FP64 nz = 128 (one block of 84 columns): 513x97x128 2627 : 2467, 2287 :
//   2411 / 3177; 769x65x128 2541 : 2438, 2431 : 2363 / 3281
// So a box whose rows take several blocks of 128 columns is streamed unless it
// is low (FP64, nz = 256) or has few modes, and one whose columns fill less
// than a block only when it is large.
bool stream_tail(const otbl_ctx *c) {
  const int modes = (c->cfg.nx - 1) * (c->dc.nz1 / 2), ny = c->cfg.ny;
  if (!c->fmaps_ok || ny > 447) return false;
  const int nz1 = c->dc.nz1, filled = 100 * nz1 / ((nz1 + 127) / 128 * 128);
  if (c->mixed) return (modes > 50000 && ny > 110) || (filled > 85 && modes > 10000);
  return modes > 50000 || (modes > 30000 && ny > 150) || filled > 85 || (nz1 > 128 && modes > 5000 && ny > 70);
}

template <typename W>
static int final_t(otbl_ctx *c, const DCoefT<W> &cw, unsigned comps, cudaEvent_t before_vel, bool second_scratch) {
  FinalStream<W> fs;
  FinalArgs<W> &a = fs.a;
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
  a.fac_u = c->w.fac_u;
  a.fac_v = c->w.fac_v;
  a.st = c->st;
  const int ncol = (c->cfg.nx - 1) * c->dc.nz1;
  fs.ck = second_scratch ? c->w.t1 : c->w.s1;
  fs.yq = second_scratch ? c->w.t2 : c->w.s2;
  fs.ub = second_scratch ? c->w.t3 : c->w.s3;
  const dim3 g((ncol + 127) / 128);
  double *U = c->f[OTBL_F_U], *V = c->f[OTBL_F_V], *Wv = c->f[OTBL_F_W];
  const dim3 gt((c->dc.nz1 + 127) / 128, c->cfg.nx - 1);
  auto comp = [&](auto C) {
    constexpr int K = decltype(C)::value;
    constexpr int sma = 2 * ((10 * 128 * (int)sizeof(W) + 127) / 128 * 128 + 10 * 128 * 8 + 8 * 128) + 128;
    constexpr int smb = FinalBox<W, K>::smem;
    allow_smem(k_final_ta<K, W>, sma);
    k_final_ta<K, W><<<gt, 128, sma, c->stream>>>(c->dc, cw, fs, &c->st->err, c->fmaps[K]);
    allow_smem(k_final_tb<K, W>, smb);
    k_final_tb<K, W><<<gt, 128, smb, c->stream>>>(c->dc, cw, fs, &c->st->err, c->fmaps[K]);
    if (before_vel) {  // the first velocity write waits for this event
      cudaStreamWaitEvent(c->stream, before_vel, 0);
      before_vel = nullptr;
    }
    k_final_s2<K><<<g, 128, 0, c->stream>>>(c->dc, U, V, Wv, c->w.fac_u, c->w.fac_v, fs.yq, fs.ub);
  };
  int n = 0;
  if (comps & 1) comp(std::integral_constant<int, 0>{}), ++n;
  if (comps & 2) comp(std::integral_constant<int, 1>{}), ++n;
  if (comps & 4) comp(std::integral_constant<int, 2>{}), ++n;
  return 3 * n;
}

cudaError_t launch_final_stream(otbl_ctx *c, unsigned comps, cudaEvent_t before_vel, bool second_scratch) {
  prof_begin(c, PK_FINAL);
  const int nl = c->mixed ? final_t<float>(c, c->dcf, comps, before_vel, second_scratch)
                          : final_t<double>(c, c->dc, comps, before_vel, second_scratch);
  prof_end(c);
  c->launches += nl;
  return cudaGetLastError();
}

void build_stream_maps(otbl_ctx *c) {
  build_x_maps(c);
  build_y_maps(c);
  c->fmaps_ok = c->mixed ? build_maps_t<float>(c) : build_maps_t<double>(c);
}

// the per-plane and per-row coefficient tables of the rings
cudaError_t prepare_stream(otbl_ctx *c) {
  const int n = (c->mixed ? 4 : 2) * c->cfg.nx, m = 2 * c->cfg.ny;
  if (c->mixed) {
    k_x_rows<float><<<(n + 127) / 128, 128, 0, c->stream>>>(c->dcf, static_cast<float *>(c->w.xrowc));
    k_y_rows<float><<<(m + 127) / 128, 128, 0, c->stream>>>(c->dcf, reinterpret_cast<float *>(c->w.yrowc));
  } else {
    k_x_rows<double><<<(n + 127) / 128, 128, 0, c->stream>>>(c->dc, static_cast<double *>(c->w.xrowc));
    k_y_rows<double><<<(m + 127) / 128, 128, 0, c->stream>>>(c->dc, c->w.yrowc);
  }
  c->launches += 2;
  return cudaGetLastError();
}

}  // namespace otbl
