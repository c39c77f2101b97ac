// Chunked tridiagonal solves: a line of n rows is cut into C chunks of K
// rows, a thread holds one chunk of two neighbouring lines in registers, and
// the chunks of a line sit in one CTA. With A = L U factored in advance,
//   forward   y_r = b_r + l_r y_{r-1},  backward  x_r = d_r y_r + e_r x_{r+1},
// each thread sweeps its rows as if the neighbouring chunk's value were 0,
// leaves its last (first) value in shared memory, and after one CTA barrier
// adds the missing carry times the products of l (e) along its rows:
//   y_r += (l_s ... l_r) c,   x_r += (e_r ... e_t) g
// (s, t the chunk's first and last row). The carry into chunk q is the sum
// Y_{q-1} + P_{q-1} Y_{q-2} + P_{q-1} P_{q-2} Y_{q-3} + ..., P a chunk's
// whole product. It ends once the product of the P is below 2^-60 (FP32:
// 2^-32), a part of the result's last bit; systems that do not decay take all
// chunks.
//
// Against one thread per line with checkpoints every few rows (read the
// inputs twice, 1.5-1.8x the algorithmic bytes, a serial chain as long as the
// line) this reads each input once and the chain is K rows and two barriers.
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

// The sweeps of a chunk in place (forward: right-hand side to y, backward: y
// to x). l, d, e point at the chunk's entries, LS apart per row; after the
// local sweep the chunk's last (first) value goes to ex[slot], and the carry
// follows after a CTA barrier.
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void forward_local(V2<T> (&y)[K], TP l) {
#pragma unroll
  for (int b = 1; b < K; ++b) fma2(y[b], l[b * LS], y[b - 1]);
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void backward_local(V2<T> (&y)[K], TP d, TP e) {
#pragma unroll
  for (int b = K - 1; b >= 0; --b) {
    const T w = d[b * LS];
    y[b].x *= w;
    y[b].y *= w;
    if (b < K - 1) fma2(y[b], e[b * LS], y[b + 1]);
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
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void forward_fix(V2<T> (&y)[K], TP l, V2<T> c) {
  T p = T(1);
#pragma unroll
  for (int b = 0; b < K; ++b) {
    p *= l[b * LS];
    fma2(y[b], p, c);
  }
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void backward_fix(V2<T> (&y)[K], TP e, V2<T> g) {
  T p = T(1);
#pragma unroll
  for (int b = K - 1; b >= 0; --b) {
    p *= e[b * LS];
    fma2(y[b], p, g);
  }
}
// whole sweeps with their barrier; P and Q are the line's chunk products, q
// this chunk, slot its place in ex, L the lanes of a chunk
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void chunk_forward(V2<T> (&y)[K], TP l, TP P, V2<T> *ex, int q, int slot, int L) {
  forward_local<K, LS, T>(y, l);
  ex[slot] = y[K - 1];
  __syncthreads();
  if (q > 0) forward_fix<K, LS, T>(y, l, chunk_carry<T>(ex + slot - L, -L, P + (q - 1), -1, q));
}
template <int K, int LS, typename T, typename TP>
__device__ __forceinline__ void chunk_backward(V2<T> (&y)[K], TP d, TP e, TP Q, V2<T> *ex, int q, int C, int slot,
                                               int L) {
  backward_local<K, LS, T>(y, d, e);
  ex[slot] = y[0];
  __syncthreads();
  if (q < C - 1) backward_fix<K, LS, T>(y, e, chunk_carry<T>(ex + slot + L, L, Q + (q + 1), 1, C - 1 - q));
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
// put(2, r, e), and the chunk products to P and Q.
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
      const double e = r == n - 1 || r < first ? 0.0 : -(double)icon[3 * r + 2] * (double)icon[3 * r + 1];
      p *= e;
      put(2, r, (T)e);
    }
    Q[q] = (T)p;
  }
}

}  // namespace otbl
