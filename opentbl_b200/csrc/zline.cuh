// z-line transforms (fourxz, ffts.f90:27-67), one warp per line, shared by
// the products (kernels.cu) and the statistics (k_stats.cu).
#pragma once
#include <cuda_runtime.h>

#include "fft.cuh"

namespace otbl {

// z-line transforms (fourxz, ffts.f90:27-67), one warp per line, in the
// arithmetic type T (double, or float on the mixed path). Fields of element
// type TI/TO are read and written with conversion to and from T.
// ---------------------------------------------------------------------------
template <typename T>
struct ZTabT {
  const V2<T> *tw;   // exp(-2 pi i t/M), t < M
  const V2<T> *tw2;  // exp(-2 pi i t/nz), t < M
  int M, nz, nz2;
};
using ZTab = ZTabT<double>;

// complex element k of a field of element type TI, as V2<T>
template <typename T, typename TI>
__device__ __forceinline__ V2<T> ldcx(const TI *__restrict__ f, int k) {
  const V2<TI> a = __ldg(reinterpret_cast<const V2<TI> *>(f) + k);
  return cmake<V2<T>>((T)a.x, (T)a.y);
}
template <typename TO, typename V>
__device__ __forceinline__ void stcx(TO *__restrict__ f, int k, V v) {
  reinterpret_cast<V2<TO> *>(f)[k] = cmake<V2<TO>>((TO)v.x, (TO)v.y);
}

// c2r of fou (nz2+1 complex modes, global) into buf (M complex = nz reals)
template <typename T, typename TI>
__device__ __forceinline__ void line_c2r(const ZTabT<T> &z, const TI *__restrict__ fou, V2<T> *buf, int lane) {
  using V = V2<T>;
  const int M = z.M, nz2 = z.nz2;
  for (int k = lane; k < M; k += 32) {
    V a = k <= nz2 ? ldcx<T>(fou, k) : cmake<V>(T(0), T(0));
    if (k == 0) a.y = T(0);  // c2r ignores Im X[0]
    const int km = M - k;
    V b = km <= nz2 ? ldcx<T>(fou, km) : cmake<V>(T(0), T(0));
    b.y = -b.y;
    const V s = cadd(a, b), d = csub(a, b);
    const V t = cmul(cconj(__ldg(z.tw2 + k)), d);  // W^{-k} d
    buf[k] = cmake<V>(s.x - t.y, s.y + t.x);      // s + i t
  }
  __syncwarp();
  warp_fft<1>(buf, M, z.tw, lane);
}

// r2c of buf (nz reals packed as M complex) into fou (modes 0..nz2) x 1/nz
template <typename T, typename TO>
__device__ __forceinline__ void line_r2c(const ZTabT<T> &z, V2<T> *buf, TO *__restrict__ fou, int lane) {
  using V = V2<T>;
  const int M = z.M, nz2 = z.nz2;
  warp_fft<-1>(buf, M, z.tw, lane);
  const T dnf = T(1) / (T)z.nz;
  for (int k = lane; k <= nz2; k += 32) {
    const V zk = buf[k];
    const V zc = cconj(buf[(M - k) & (M - 1)]);
    const V e = cmake<V>(T(0.5) * (zk.x + zc.x), T(0.5) * (zk.y + zc.y));
    const V d = csub(zk, zc);
    const V o = cmake<V>(T(0.5) * d.y, T(-0.5) * d.x);  // -i d / 2
    const V xk = cadd(e, cmul(__ldg(z.tw2 + k), o));
    stcx(fou, k, cmake<V>(dnf * xk.x, dnf * xk.y));
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// The same transforms with a line kept in the registers of G lanes, E = M/G
// elements each: layout L, lane t of the group holds complex element n = t + G
// m in v[m]. Two Stockham passes, radix E (the lane's own elements) and radix G
// (E / G butterflies per lane), with one exchange through a shared buffer of
// the group between them; the second one's outputs are in layout L again.
//   M = 256: 16 lanes, 16 x 16; 128: 8 lanes, 16 x 8; 64: 8, 8 x 8; 32: 4,
//   8 x 4; 16: 4, 4 x 4
// A warp works on 32 / G lines. The buffer's element i sits at i + i / E: the
// lanes of a write are E + 1 elements apart and those of a read neighbours,
// both without bank conflicts in 8- and 16-byte elements. The mirrored element
// Z[M-k] of the real-to-complex step comes from the lane that holds it.
// Bound: the L1/shared-memory unit. Against a whole warp per line (8 elements
// a lane, radix 8, 8, 4 with two exchanges) a transform of M = 256 takes about
// 155 wavefronts instead of 245.
// ---------------------------------------------------------------------------
template <int M>
struct ZGroup {
  static_assert(M == 256 || M == 128 || M == 64 || M == 32 || M == 16, "M = 16..256");
  static constexpr int G = M == 256 ? 16 : (M >= 64 ? 8 : 4), E = M / G, NB = E / G;
  static constexpr int LW = 32 / G;          // lines per warp
  static constexpr int BUF = G * (E + 1);    // buffer elements per line
};
template <typename V>
__device__ __forceinline__ V shfl_cx(V v, int src) {
  V r;
  r.x = __shfl_sync(0xffffffffu, v.x, src);
  r.y = __shfl_sync(0xffffffffu, v.y, src);
  return r;
}

// inverse (SIGN = +1) or forward (SIGN = -1) FFT of a line in layout L
template <int M, int SIGN, typename V>
__device__ __forceinline__ void zfft_group(V (&L)[ZGroup<M>::E], V *buf, const V *__restrict__ tw, int t) {
  constexpr int G = ZGroup<M>::G, E = ZGroup<M>::E, NB = ZGroup<M>::NB;
  dft_small<E, SIGN>(L);
#pragma unroll
  for (int r = 0; r < E; ++r) buf[t * (E + 1) + r] = L[r];
  __syncwarp();
#pragma unroll
  for (int it = 0; it < NB; ++it) {
    const int j = t + G * it;
    V v[G];
#pragma unroll
    for (int r = 0; r < G; ++r) v[r] = buf[j + r * (E + 1)];
#pragma unroll
    for (int r = 1; r < G; ++r) {
      V w = __ldg(&tw[r * j]);
      if (SIGN > 0) w.y = -w.y;
      v[r] = cmul(v[r], w);
    }
    dft_small<G, SIGN>(v);
#pragma unroll
    for (int r = 0; r < G; ++r) L[it + r * NB] = v[r];
  }
  __syncwarp();
}

// c2r of fou (modes 0..nz2, global) into layout L (physical values packed as
// complex), line_c2r's pre-step followed by the inverse FFT
template <int M, typename T, typename TI>
__device__ __forceinline__ void zc2r_group(const ZTabT<T> &z, const TI *__restrict__ fou, V2<T> (&L)[ZGroup<M>::E],
                                           V2<T> *buf, int t) {
  using V = V2<T>;
  constexpr int G = ZGroup<M>::G, E = ZGroup<M>::E;
  const int nz2 = z.nz2;
  V b[E];
#pragma unroll
  for (int m = 0; m < E; ++m) {  // modes above nz2 are not read (they are 0)
    const int k = t + G * m, km = M - k;
    L[m] = k <= nz2 ? ldcx<T>(fou, k) : cmake<V>(T(0), T(0));
    b[m] = km <= nz2 ? ldcx<T>(fou, km) : cmake<V>(T(0), T(0));
  }
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int k = t + G * m;
    if (k == 0) L[m].y = T(0);  // c2r ignores Im X[0]
    b[m].y = -b[m].y;
    const V s = cadd(L[m], b[m]), d = csub(L[m], b[m]);
    const V tt = cmul(cconj(__ldg(z.tw2 + k)), d);  // W^{-k} d
    L[m] = cmake<V>(s.x - tt.y, s.y + tt.x);       // s + i t
  }
  zfft_group<M, 1>(L, buf, z.tw, t);
}

// r2c of layout L (physical values packed as complex) into fou (modes 0..nz2)
// x 1/nz: forward FFT, then line_r2c's post-step; stores only when `store`
template <int M, typename T, typename TO>
__device__ __forceinline__ void zr2c_group(const ZTabT<T> &z, V2<T> (&L)[ZGroup<M>::E], TO *__restrict__ fou,
                                           V2<T> *buf, int t, bool store) {
  using V = V2<T>;
  constexpr int G = ZGroup<M>::G, E = ZGroup<M>::E;
  zfft_group<M, -1>(L, buf, z.tw, t);
  const int nz2 = z.nz2, src = (threadIdx.x & 31 & ~(G - 1)) + ((G - t) & (G - 1));
  const T dnf = T(1) / (T)z.nz;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    // Z[(M - k) mod M], k = t + G m: lane G - t's L[E - 1 - m] for t >= 1, this
    // lane's own L[(E - m) mod E] for t = 0
    const V other = shfl_cx(L[E - 1 - m], src);
    const V zm = t == 0 ? L[(E - m) % E] : other;
    const int k = t + G * m;
    if (k <= nz2 && store) {
      const V zk = L[m];
      const V zc = cconj(zm);
      const V e = cmake<V>(T(0.5) * (zk.x + zc.x), T(0.5) * (zk.y + zc.y));
      const V d = csub(zk, zc);
      const V o = cmake<V>(T(0.5) * d.y, T(-0.5) * d.x);  // -i d / 2
      const V xk = cadd(e, cmul(__ldg(z.tw2 + k), o));
      stcx(fou, k, cmake<V>(dnf * xk.x, dnf * xk.y));
    }
  }
}

}  // namespace otbl
