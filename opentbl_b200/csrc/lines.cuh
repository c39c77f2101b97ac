// Chunked tridiagonal solves: a line of n rows is cut into C chunks of K
// rows, a thread holds one chunk of two neighbouring lines in registers, and
// the chunks of a line sit in one CTA. With A = L U factored in advance,
//   forward   y_r = b_r + l_r y_{r-1},  backward  x_r = (y_r - u_r x_{r+1}) d_r,
// each thread first sweeps its rows as if the neighbouring chunk's value were
// 0, keeping only its last (first) value, leaves that in shared memory, and
// after one CTA barrier forms the carry c from the neighbouring chunks and
// sweeps its rows again, now from c. The carry into chunk q is the sum
// Y_{q-1} + P_{q-1} Y_{q-2} + P_{q-1} P_{q-2} Y_{q-3} + ..., P a chunk's
// whole product of l (-u d). It ends once the product of the P is below 2^-60
// (FP32: 2^-32), a part of the result's last bit; systems that do not decay
// take all chunks.
// The second sweep is the serial recurrence, operation for operation, and so
// are its roundings. One sweep that is kept and corrected by the carry times
// the products of l (-u d), with -u d rounded once, is K operations shorter in
// series (step of 257x97x128 1251 against 1266 us, the 12-box mixed ensemble
// 16.29 against 16.45 ms, others equal) but less accurate: the solves end
// 10-20% further from the exact ones than a serial sweep in the same
// precision, and after a mixed step of 129x65x64 the median error of u over 12
// states was 2.10e-8, where serial sweeps gave 1.79e-8 and these give 1.74e-8.
//
// Against one thread per line with checkpoints every few rows (read the
// inputs twice, 1.5-1.8x the algorithmic bytes, a serial chain as long as the
// line) this reads each input once and the chain is 2 K rows and two barriers.
//
// Where they exceed a few KB, the coefficients are staged in shared memory,
// coefficient i of row s + b of chunk q at tab[q S + i K + b], S the number of
// coefficients times K (an odd number of values, so that neighbouring chunks
// fall on different banks and all offsets are constants). Read through L1
// instead, they were evicted by the fields (1025x49x512 interpxx: half of the
// table's sectors missed, a warp waited 22 cycles between its instructions).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "fft.cuh"

namespace otbl {

// y += a x for the two lines of a thread
template <typename T>
__device__ __forceinline__ void fma2(V2<T> &y, T a, V2<T> x) {
  y.x += a * x.x;
  y.y += a * x.y;
}

// p ? a : b by components (a conditional store to an unrolled array element
// would be turned into an indexed one and the array put in local memory)
template <typename V>
__device__ __forceinline__ V select2(bool p, V a, V b) {
  return cmake<V>(p ? a.x : b.x, p ? a.y : b.y);
}

// The sweeps of a chunk; l, d, u point at its entries, LS apart per row.
// *_end: the last (first) value of a sweep that starts from 0; *_from: the
// sweep in place from the neighbouring chunk's value. backward_end carries
// x_r / d_r, whose chain is one multiply-add a row.
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ V2<T> forward_end(const V2<T> (&y)[K], TP l) {
  V2<T> x = y[0];
#pragma unroll
  for (int b = 1; b < K; ++b) {
    V2<T> v = y[b];
    fma2(v, l[b * LS], x);
    x = v;
  }
  return x;
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void forward_from(V2<T> (&y)[K], TP l, V2<T> c) {
#pragma unroll
  for (int b = 0; b < K; ++b) fma2(y[b], l[b * LS], b == 0 ? c : y[b == 0 ? 0 : b - 1]);
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ V2<T> backward_end(const V2<T> (&y)[K], TP d, TP u) {
  V2<T> x = y[K - 1];
#pragma unroll
  for (int b = K - 2; b >= 0; --b) {
    V2<T> v = y[b];
    fma2(v, -u[b * LS] * d[(b + 1) * LS], x);
    x = v;
  }
  return cmake<V2<T>>(d[0] * x.x, d[0] * x.y);
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void backward_from(V2<T> (&y)[K], TP d, TP u, V2<T> g) {
#pragma unroll
  for (int b = K - 1; b >= 0; --b) {
    const T w = d[b * LS];
    fma2(y[b], -u[b * LS], b == K - 1 ? g : y[b == K - 1 ? b : b + 1]);
    y[b].x *= w;
    y[b].y *= w;
  }
}
// the sum over n neighbouring chunks, the nearest first: their values at ex,
// ex + step, ..., their products at P, P + pstep, ...
template <typename T, typename TP>
__device__ __forceinline__ V2<T> chunk_carry(const V2<T> *ex, int step, TP P, int pstep, int n) {
  constexpr T tiny = sizeof(T) == 8 ? (T)8.673617379884035e-19 : (T)2.3283064365386963e-10;  // 2^-60, 2^-32
  V2<T> c = cmake<V2<T>>(T(0), T(0));
  T w = T(1);
  for (int k = 0; k < n; ++k) {
    fma2(c, w, *ex);
    w *= *P;
    if (fabs(w) < tiny) break;
    ex += step;
    P += pstep;
  }
  return c;
}
// whole sweeps with their barrier; P and Q are the line's chunk products, q
// this chunk, slot its place in ex, L the lanes of a chunk
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void chunk_forward(V2<T> (&y)[K], TP l, TP P, V2<T> *ex, int q, int slot, int L) {
  ex[slot] = forward_end<K, LS, T>(y, l);
  __syncthreads();
  forward_from<K, LS, T>(y, l, chunk_carry<T>(ex + slot - L, -L, P + (q - 1), -1, q));
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void chunk_backward(V2<T> (&y)[K], TP d, TP u, TP Q, V2<T> *ex, int q, int C, int slot,
                                               int L) {
  ex[slot] = backward_end<K, LS, T>(y, d, u);
  __syncthreads();
  backward_from<K, LS, T>(y, d, u, chunk_carry<T>(ex + slot + L, L, Q + (q + 1), 1, C - 1 - q));
}

// asynchronous global -> shared copy of one value, zeros when !valid
template <typename V>
__device__ __forceinline__ void cp_async_v(V *s, const V *g, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  const int sz = valid ? (int)sizeof(V) : 0;
  if constexpr (sizeof(V) == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(g), "r"(sz) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;\n" ::"r"(sa), "l"(g), "r"(sz), "n"(sizeof(V))
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---- tables (host) ----
// One operator's factors over n rows, from the reference's icon(3, n) (l,
// 1/pivot, upper), starting at row `first`: put(0, r, l), put(1, r, d),
// put(2, r, u), and the chunk products to P and Q.
template <typename T, typename F>
void chunk_factors(F put, int K, int n, const T *icon, int first, T *P, T *Q) {
  const int C = (n + K - 1) / K;
  for (int q = 0; q < C; ++q) {
    const int s = q * K, t = std::min(s + K, n) - 1;
    double p = 1.0;
    for (int r = s; r <= t; ++r) {
      const double l = r <= first ? 0.0 : (double)icon[3 * r];
      p *= l;
      put(0, r, (T)l);
      put(1, r, icon[3 * r + 1]);
    }
    P[q] = t == s + K - 1 ? (T)p : T(0);
    p = 1.0;
    for (int r = t; r >= s; --r) {
      const T u = r == n - 1 || r < first ? T(0) : icon[3 * r + 2];
      p *= -(double)u * (double)icon[3 * r + 1];
      put(2, r, u);
    }
    Q[q] = (T)p;
  }
}

}  // namespace otbl
