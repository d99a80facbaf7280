// heom_tl_term.cuh -- the time-local truncation term of one ADO element
// (internal; shared by the tiled and the node stage kernels).
//
// For an independent bath m on site m, IndependentBath::DoTimelocal
// (hierarchy_updater.cc:171-190) forms X_m = Q_m X - X Q_m^+ and adds its
// column m and subtracts its row m, so element (i, j) of the derivative of a
// deepest-tier ADO X gains X_j[i][j] - X_i[i][j].  With D = Q_j - Q_i and X
// Hermitian that is
//     (D X)_ij - conj((D X)_ji),
// the same shape as the commutator with H; for i == j it vanishes.  Either a
// thread evaluates a pair (tl_pair_term), or each element adds its own product
// (tl_half_term) before the transposed elements are exchanged.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace phi {

// An element of Q.  Q is rewritten between stages, so it is not read through the
// read-only path, and a volatile load stays behind the stage's pdl_wait.
__device__ __forceinline__ double2 ld_q(const double2 *p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// Q: nb*N*N sums Q_m, column-major per bath (a few KB for the sizes the tile
// kernel serves).  X: the ADO, column-major.  The loop stays rolled so that,
// inlined into a stage kernel, it holds few registers.
template <class TX>
static __device__ __forceinline__ TX tl_pair_term(const TX *X, const double2 *Q, int N, int i, int j) {
  using R = decltype(X->x);
  const size_t E = (size_t)N * N;
  const double2 *Qi = Q + (size_t)i * E, *Qj = Q + (size_t)j * E;
  R ar = 0, ai = 0, br = 0, bi = 0;
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    const double2 qji = ld_q(Qj + i + k * N), qii = ld_q(Qi + i + k * N);
    const double2 qjj = ld_q(Qj + j + k * N), qij = ld_q(Qi + j + k * N);
    const R dir = (R)(qji.x - qii.x), dii = (R)(qji.y - qii.y);  // D[i][k]
    const R djr = (R)(qjj.x - qij.x), dji = (R)(qjj.y - qij.y);  // D[j][k]
    const TX xkj = X[k + j * N], xki = X[k + i * N];
    ar = fma(dir, xkj.x, ar);
    ar = fma(-dii, xkj.y, ar);
    ai = fma(dir, xkj.y, ai);
    ai = fma(dii, xkj.x, ai);
    br = fma(djr, xki.x, br);
    br = fma(-dji, xki.y, br);
    bi = fma(djr, xki.y, bi);
    bi = fma(dji, xki.x, bi);
  }
  TX out;
  out.x = ar - br;  // a - conj(b)
  out.y = ai + bi;
  return out;
}

// ((Q_j - Q_i) X)_ij: added to its conjugate transpose over the pair, the term
// above (element (j, i) has -D).
template <class TX>
static __device__ __forceinline__ TX tl_half_term(const TX *X, const double2 *Q, int N, int i, int j) {
  using R = decltype(X->x);
  const size_t E = (size_t)N * N;
  const double2 *Qi = Q + (size_t)i * E + i, *Qj = Q + (size_t)j * E + i;
  const TX *Xj = X + j * N;
  TX g;
  g.x = g.y = 0;
#pragma unroll 4
  for (int k = 0; k < N; ++k) {
    const double2 qj = ld_q(Qj + k * N), qi = ld_q(Qi + k * N);
    const R dr = (R)(qj.x - qi.x), di = (R)(qj.y - qi.y);
    const TX x = Xj[k];
    g.x = fma(dr, x.x, g.x);
    g.x = fma(-di, x.y, g.x);
    g.y = fma(dr, x.y, g.y);
    g.y = fma(di, x.x, g.y);
  }
  return g;
}

}  // namespace phi
