// heom_small.cu -- the whole RK4 run of a small hierarchy in one CTA.
//
// A hierarchy of a few hundred elements (PHI's spin-boson configuration has
// 11 nodes of 2 x 2) gives each stage kernel a handful of warps of work, so
// a run of four launches per step is bound by launch and memory latency,
// not by the SMs.  Here one CTA loops over every step of the run on the
// device.  With a thread per upper-triangle (node, pair) item the state, the RK4
// accumulator and the item's coefficients are in registers, only the stage
// inputs in shared memory, and a stage has one barrier; larger hierarchies keep
// all of it in shared memory, a stage being one pass over the items and one
// element-wise combine, separated by block barriers.  The arithmetic is that of the node kernel
// (heom_kernels.cu) for IndependentBath and DiagonalBath couplings:
// HierarchyUpdater::Get (hierarchy_updater.h:36-75, hierarchy_updater.cc
// :84-127, :216-254) and the RK4 combines of Rk4Integrate
// (hierarchy_integrator.cc:2705-2826); every derivative ADO is evaluated on
// its upper triangle and mirrored.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "heom_device.cuh"
#include "heom_kernels.h"
#include "heom_tile.h"

namespace phi {
namespace {

constexpr int kSmallThreads = 256;  // at most; register rows need one thread per item

__device__ __forceinline__ double2 s_conj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 s_axpy(double2 a, double2 b, double s) {
  return make_double2(fma(b.x, s, a.x), fma(b.y, s, a.y));
}

struct SmallRk4Params {
  HeomConsts c;
  double2 *y;     // hierarchy state (global), read at the start, written at the end
  double dt;
  long long steps;
  Rk4Ctl *rk4;    // step / output bookkeeping, as the stage kernels keep it
  double2 *traj;  // rho_0 rows (may be null)
};

// The derivative of node n's ADO at an upper-triangle pair (i, j) is a
// fixed linear combination of stage-input elements (every stage input is
// exactly Hermitian).  Each item's combination -- element offsets and complex
// coefficients -- is built once per launch into shared memory, so a stage
// is R complex multiply-adds from shared memory per item:
//   -i/hbar [H, X]_ij = sum_k (-i/hbar) H_ik X_kj + (i/hbar) conj(H_jk) X_ik
//   -(dephasing_n + Matsubara_ij) X_ij
//   IndependentBath (hierarchy_updater.cc:216-254), site m = j: +i p X+_ij,
//     +i sp conj(c) X-_ij; site m = i: -i p X+_ij, -i sp c X-_ij; i = j = m:
//     2 sp Im(c) X-_mm (the next terms cancel);
//   DiagonalBath (:105-127): -i (V_i - V_j) X+_ij, -i n (c V_i - c* V_j) X-_ij.
struct RowBuilder {
  int *idx;
  double2 *coef;
  int n = 0;
  __device__ void add(long long e, double2 cf) {
    idx[n] = (int)e;
    coef[n] = cf;
    ++n;
  }
};

template <int KIND>
__device__ int build_row(const HeomConsts &c, const double2 *Hs, long long n, int i, int j, int *idx,
                         double2 *coef) {
  const int N = c.N, E = N * N, T = c.T, L2 = c.L + 2;
  const double ih = c.inv_hbar;
  RowBuilder r{idx, coef};
  const long long base = n * E;
  for (int k = 0; k < N; ++k) {
    const double2 h1 = Hs[i + k * N], h2 = Hs[j + k * N];
    r.add(base + k + j * N, make_double2(h1.y * ih, -h1.x * ih));   // -i ih H_ik
    r.add(base + i + k * N, make_double2(h2.y * ih, h2.x * ih));    // +i ih conj(H_jk)
  }
  if (c.vacuum) return r.n;
  double deph = 0.0;  // sum_t n_t nu_t in term order
  for (int t = 0; t < T; ++t) deph += __ldg(c.mi + n * T + t) * __ldg(c.nu + t);
  r.add(base + i + j * N, make_double2(-(deph + __ldg(c.mats_elem + i + j * N)), 0.0));
  if (KIND == kIndependent) {
    for (int side = 0; side < 2; ++side) {
      const int site = side == 0 ? j : i;
      for (int q = __ldg(c.site_ptr + site); q < __ldg(c.site_ptr + site + 1); ++q) {
        const int t = __ldg(c.site_terms + q);
        const int nt = __ldg(c.mi + n * T + t);
        const int nx = __ldg(c.next + n * T + t), pv = __ldg(c.prev + n * T + t);
        const double sn = __ldg(c.sq_next + t * L2 + nt), sp = __ldg(c.sq_prev + t * L2 + nt);
        const double2 ct = __ldg(c.corr + t);
        const long long off = (long long)i + (long long)j * N;
        if (i == j) {
          if (side == 1 && pv >= 0) r.add((long long)pv * E + off, make_double2(2.0 * sp * ct.y, 0.0));
          continue;
        }
        if (side == 0) {
          if (nx >= 0) r.add((long long)nx * E + off, make_double2(0.0, sn));
          if (pv >= 0) r.add((long long)pv * E + off, make_double2(sp * ct.y, sp * ct.x));   // i sp conj(c)
        } else {
          if (nx >= 0) r.add((long long)nx * E + off, make_double2(0.0, -sn));
          if (pv >= 0) r.add((long long)pv * E + off, make_double2(sp * ct.y, -sp * ct.x));  // -i sp c
        }
      }
    }
  } else {
    for (int s2 = 0; s2 < 2 * T; ++s2) {
      const bool is_next = s2 < T;
      const int t = is_next ? s2 : s2 - T;
      const int id = is_next ? __ldg(c.next + n * T + t) : __ldg(c.prev + n * T + t);
      if (id < 0) continue;
      const double *V = c.bath_V + (size_t)__ldg(c.term_site + t) * N;
      const double vi = __ldg(V + i), vj = __ldg(V + j);
      double2 f;
      if (is_next) {
        f = make_double2(0.0, -(vi - vj));
      } else {
        const double2 ct = __ldg(c.corr + t);
        const int nt = __ldg(c.mi + n * T + t);
        const double re = ct.x * vi - ct.x * vj;
        const double im = ct.y * vi + ct.y * vj;
        f = make_double2(im * nt, -re * nt);
      }
      r.add((long long)id * E + i + (long long)j * N, f);
    }
  }
  return r.n;
}

// Entries of one item's row, an upper bound: the commutator (2N), the decay,
// and the neighbour terms (IndependentBath: next and prev of the terms of
// sites i and j; DiagonalBath: next and prev of every term).
__host__ __device__ inline int small_row_max(const HeomConsts &c) {
  return 2 * c.N + 1 + (c.kind == kIndependent ? 4 * c.T : 2 * c.T);
}

// Number of an item's entries with a purely imaginary coefficient (2 of the 4
// products): the commutator of a real H and the next terms.
__host__ __device__ inline int small_imag_max(const HeomConsts &c) {
  return (c.h_real ? 2 * c.N : 0) + (c.kind == kIndependent ? 2 * c.T : c.T);
}

// Moves up to `most` entries with a zero real coefficient to the front of an
// item's row (other entries can have one too); returns their number.
__device__ int partition_row(int n, int most, int *idx, double2 *coef) {
  int front = 0;
  for (int r = 0; r < n && front < most; ++r) {
    if (coef[r].x != 0.0) continue;
    const double2 cf = coef[front];
    const int e = idx[front];
    coef[front] = coef[r];
    idx[front] = idx[r];
    coef[r] = cf;
    idx[r] = e;
    ++front;
  }
  return front;
}

// RI + RC > 0: every thread owns at most one item and keeps its row in
// registers for the whole run -- up to RI imaginary and RC complex entries,
// padded with zero coefficients -- with the state and the accumulator of its
// element and of the mirrored one.  A stage is then the gather of the row from
// one of two shared stage inputs, its products, the combine, and one barrier:
// stage 0 reads buffer 0 (y) and writes 1, stage 1 the reverse, and so on.
// Bound by that chain of latencies (11-node spin-boson, 2 warps): with the
// state in shared memory and every entry complex a stage took 0.267 us.
// RI = RC = 0: rows stay in shared memory and threads loop over items.
template <int KIND, int RI, int RC>
__global__ void __launch_bounds__(kSmallThreads, 1) heom_small_rk4_kernel(SmallRk4Params p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool REG = RI + RC > 0;
  const HeomConsts &c = p.c;
  const int N = c.N, E = N * N, P = N * (N + 1) / 2;
  const long long M = c.M, ME = M * E, items = M * P;
  const int R = small_row_max(c);
  const int tid = threadIdx.x, nth = blockDim.x;
  double2 *Hs = reinterpret_cast<double2 *>(smem_raw);
  double2 *Y = Hs + E;
  double2 *ACC = Y + ME;
  double2 *X = ACC + ME;
  double2 *K = X + ME;
  double2 *coef = K + ME;                                 // items * R
  int *idx = reinterpret_cast<int *>(coef + items * R);   // items * R
  int *cnt = idx + items * R;                             // items
  for (int e = tid; e < E; e += nth) Hs[e] = c.H[e];
  for (long long e = tid; e < ME; e += nth) Y[e] = p.y[e];
  __syncthreads();
  for (long long u = tid; u < items; u += nth) {
    const long long n = u / P;
    const int q = (int)(u - n * P);
    cnt[u] = build_row<KIND>(c, Hs, n, __ldg(c.pair_i + q), __ldg(c.pair_j + q), idx + u * R, coef + u * R);
  }
  __syncthreads();
  const double dt = p.dt;
  Rk4Ctl *rc = p.rk4;
  long long step = rc->step, nout = rc->nout;
  const long long out_factor = rc->out_factor, capacity = rc->capacity;
  if constexpr (REG) {
    int i_idx[RI], c_idx[RC];
    double i_cf[RI];
    double2 c_cf[RC];
    const long long u = tid;
    const bool own = u < items;
    int nr = 0, ni = 0, e0 = -1, e1 = -1;  // the item's element and its mirror (-1: none)
    if (own) {
      nr = cnt[u];
      ni = partition_row(nr, RI, idx + u * R, coef + u * R);
      const long long n = u / P;
      const int q = (int)(u - n * P);
      const int i = __ldg(c.pair_i + q), j = __ldg(c.pair_j + q);
      e0 = (int)(n * E + i + j * N);
      e1 = i == j ? -1 : (int)(n * E + j + i * N);
    }
#pragma unroll
    for (int r = 0; r < RI; ++r) {
      i_idx[r] = r < ni ? idx[u * R + r] : 0;
      i_cf[r] = r < ni ? coef[u * R + r].y : 0.0;
    }
#pragma unroll
    for (int r = 0; r < RC; ++r) {
      c_idx[r] = ni + r < nr ? idx[u * R + ni + r] : 0;
      c_cf[r] = ni + r < nr ? coef[u * R + ni + r] : make_double2(0.0, 0.0);
    }
    const double2 zero = make_double2(0.0, 0.0);
    double2 y0 = own ? Y[e0] : zero, y1 = e1 >= 0 ? Y[e1] : zero, a0 = zero, a1 = zero;
    for (long long it = 0; it < p.steps; ++it) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const double a = s == 2 ? dt : dt / 2;
        const double w = (s == 0 || s == 3) ? dt / 6 : dt / 3;
        const double2 *in = s & 1 ? X : Y;
        double2 *out = s & 1 ? Y : X;
        double2 xi[RI], xc[RC];
#pragma unroll
        for (int r = 0; r < RI; ++r) xi[r] = in[i_idx[r]];
#pragma unroll
        for (int r = 0; r < RC; ++r) xc[r] = in[c_idx[r]];
        // Two chains per component: the imaginary entries and the complex ones.
        double2 v = zero, z = zero;
#pragma unroll
        for (int r = 0; r < RI; ++r) {
          v.x = fma(-i_cf[r], xi[r].y, v.x);
          v.y = fma(i_cf[r], xi[r].x, v.y);
        }
#pragma unroll
        for (int r = 0; r < RC; ++r) {
          z.x = fma(c_cf[r].x, xc[r].x, z.x);
          z.x = fma(-c_cf[r].y, xc[r].y, z.x);
          z.y = fma(c_cf[r].x, xc[r].y, z.y);
          z.y = fma(c_cf[r].y, xc[r].x, z.y);
        }
        v.x += z.x;
        v.y = e1 < 0 ? 0.0 : v.y + z.y;
        double2 x0, x1;
        if (s < 3) {
          x0 = s_axpy(y0, v, a);
          x1 = s_axpy(y1, s_conj(v), a);
          a0 = s_axpy(s == 0 ? y0 : a0, v, w);
          a1 = s_axpy(s == 0 ? y1 : a1, s_conj(v), w);
        } else {
          x0 = y0 = s_axpy(a0, v, w);
          x1 = y1 = s_axpy(a1, s_conj(v), w);
        }
        if (own) out[e0] = x0;
        if (e1 >= 0) out[e1] = x1;
        __syncthreads();
      }
      // rho_0 row after step `step` when step % out_factor == 0 (:2858).
      if (out_factor > 0 && step % out_factor == 0) {
        if (p.traj && nout < capacity) {
          if (own && e0 < E) p.traj[nout * E + e0] = y0;
          if (e1 >= 0 && e1 < E) p.traj[nout * E + e1] = y1;
        }
        ++nout;
      }
      ++step;
    }
    if (own) p.y[e0] = y0;
    if (e1 >= 0) p.y[e1] = y1;
  } else {
    for (long long it = 0; it < p.steps; ++it) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const double a = s == 2 ? dt : dt / 2;
        const double w = (s == 0 || s == 3) ? dt / 6 : dt / 3;
        const double2 *in = s == 0 ? Y : X;
        for (long long u = tid; u < items; u += nth) {
          const int *ri = idx + u * R;
          const double2 *rcf = coef + u * R;
          double2 v = make_double2(0.0, 0.0);
          for (int r = 0; r < cnt[u]; ++r) {
            const double2 cf = rcf[r], x = in[ri[r]];
            v.x = fma(cf.x, x.x, v.x);
            v.x = fma(-cf.y, x.y, v.x);
            v.y = fma(cf.x, x.y, v.y);
            v.y = fma(cf.y, x.x, v.y);
          }
          const long long n = u / P;
          const int q = (int)(u - n * P);
          const int i = __ldg(c.pair_i + q), j = __ldg(c.pair_j + q);
          if (i == j) {
            v.y = 0.0;
            K[n * E + i + j * N] = v;
          } else {
            K[n * E + i + j * N] = v;
            K[n * E + j + i * N] = s_conj(v);
          }
        }
        __syncthreads();
        for (long long e = tid; e < ME; e += nth) {
          const double2 kv = K[e];
          if (s == 0) {
            const double2 ys = Y[e];
            X[e] = s_axpy(ys, kv, a);
            ACC[e] = s_axpy(ys, kv, w);
          } else if (s < 3) {
            X[e] = s_axpy(Y[e], kv, a);
            ACC[e] = s_axpy(ACC[e], kv, w);
          } else {
            Y[e] = s_axpy(ACC[e], kv, w);
          }
        }
        __syncthreads();
      }
      if (out_factor > 0 && step % out_factor == 0) {
        if (p.traj && nout < capacity)
          for (int e = tid; e < E; e += nth) p.traj[nout * E + e] = Y[e];
        ++nout;
      }
      ++step;
    }
    for (long long e = tid; e < ME; e += nth) p.y[e] = Y[e];
  }
  if (tid == 0) {
    rc->step = step;
    rc->nout = nout;
  }
}

size_t small_smem(const HeomConsts &c) {
  const size_t E = (size_t)c.N * c.N, items = (size_t)c.M * (c.N * (c.N + 1) / 2);
  const size_t R = (size_t)small_row_max(c);
  return (E + 4 * (size_t)c.M * E) * sizeof(double2) + items * R * (sizeof(double2) + sizeof(int)) +
         items * sizeof(int);
}

// Threads of the launch: enough for the larger of the item and element
// loops, in whole warps, at most kSmallThreads (fewer warps make the two
// barriers of a stage cheaper).
int small_threads(const HeomConsts &c) {
  const long long work = std::max<long long>(c.M * (c.N * (c.N + 1) / 2), c.M * c.N * c.N);
  const long long w = (work + 31) / 32 * 32;
  return (int)std::min<long long>(kSmallThreads, std::max<long long>(32, w));
}

template <int KIND, int RI, int RC>
cudaError_t launch_small_variant(const SmallRk4Params &p, size_t smem, int threads, cudaStream_t stream) {
  static thread_local int raised[kSmemLimitDevices] = {};
  cudaError_t e = raise_smem_limit(heom_small_rk4_kernel<KIND, RI, RC>, smem, raised);
  if (e != cudaSuccess) return e;
  heom_small_rk4_kernel<KIND, RI, RC><<<1, threads, smem, stream>>>(p);
  return cudaGetLastError();
}

// Register rows when every item has its own thread and the bounds on its
// imaginary and complex entries fit one of the compiled sizes.
template <int KIND>
cudaError_t launch_small_kind(const SmallRk4Params &p, size_t smem, cudaStream_t stream) {
  const HeomConsts &c = p.c;
  const int threads = small_threads(c);
  if (c.M * (c.N * (c.N + 1) / 2) <= kSmallThreads) {
    const int ri = small_imag_max(c), total = small_row_max(c);
    const int rc = total - ri;
    if (ri <= 6 && rc <= 2) return launch_small_variant<KIND, 6, 2>(p, smem, threads, stream);
    if (ri <= 8 && rc <= 4) return launch_small_variant<KIND, 8, 4>(p, smem, threads, stream);
    if (ri <= 12 && rc <= 4) return launch_small_variant<KIND, 12, 4>(p, smem, threads, stream);
    if (ri <= 8 && rc <= 8) return launch_small_variant<KIND, 8, 8>(p, smem, threads, stream);
    if (ri <= 16 && rc <= 8) return launch_small_variant<KIND, 16, 8>(p, smem, threads, stream);
  }
  return launch_small_variant<KIND, 0, 0>(p, smem, threads, stream);
}

}  // namespace

bool small_rk4_eligible(const HeomConsts &c) {
  if (c.kind != kIndependent && c.kind != kDiagonal) return false;
  // Problems the tiled kernel takes stay on it: a batch of such instances
  // is then bit-identical to each instance run alone.
  if (tile_kernel_available(c)) return false;
  if (c.filtered || c.time_local) return false;
  return (size_t)c.M * c.N * c.N <= kSmallMaxElements && small_smem(c) <= kSmallMaxSmem;
}

cudaError_t launch_small_rk4(const HeomConsts &c, double2 *y, double dt, long long steps, Rk4Ctl *rk4,
                             double2 *traj, cudaStream_t stream) {
  if (!small_rk4_eligible(c) || steps <= 0) return cudaErrorInvalidValue;
  SmallRk4Params p;
  p.c = c;
  p.y = y;
  p.dt = dt;
  p.steps = steps;
  p.rk4 = rk4;
  p.traj = traj;
  const size_t smem = small_smem(c);
  return c.kind == kIndependent ? launch_small_kind<kIndependent>(p, smem, stream)
                                : launch_small_kind<kDiagonal>(p, smem, stream);
}

}  // namespace phi
