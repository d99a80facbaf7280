// heom_kernels.cu -- the Liouvillian and the fused RK stages for every bath
// coupling at any N (FP64); identity-site independent baths of the tiled sizes
// run on heom_tile.cu instead.
//
// A CTA owns a tile of nt consecutive nodes.  Thread t < CS * N works on row
// i = t % N of the tile's columns t / N, t / N + CS, ... (elements t, t + CS N,
// ... of the tile), so its reads of ADOs -- its own tile's and the linked
// ones -- run along contiguous memory.  Per element
//   B_ij = -i/hbar (H X)_ij + sum_b (V_b M_b)_ij
//   M_b  = sum_k (-i s X+ - i c sp X-)  over the K + 1 terms of bath b
//          (+ Delta_b [X, V_b] for full couplings: FullBath::DoMatsubara)
// and, every ADO being Hermitian,
//   dX_ij = B_ij + conj(B_ji) - (dephasing + Matsubara_ij) X_ij :
// PHI's commutators -i/hbar [H, X], -p [V, X+], -pr V X- - pc X- V and
// -Delta [V, [V, X]] are each a product plus its Hermitian conjugate, and the
// two factors of a term differ only in V's side, so the terms of a bath are
// summed before the one product with V_b (a 3-bath full coupling with K = 1
// takes 10 products per node instead of 37).  An independent bath's V_b is
// |m><m|: V_b M_b is row m of M_b, the conjugate of its column m, so element
// (i, j) adds the terms of site j; a diagonal V_b scales row i.  The tile
// exchanges B through shared memory; the RK stage combine follows in
// registers.
//
// What bounds it (B200): latency.  A stage of these hierarchies is a few
// thousand nodes or fewer, i.e. one chain of node records -> gathers ->
// products -> exchange -> combine per CTA.  So the records are read before
// the wait on the previous stage's kernel (programmatic dependent launch:
// they are constant), the combine's operands are copied to shared memory
// asynchronously while the derivative runs, and tiles are cut down until
// there are two CTAs per SM.
//
// Reference: HierarchyUpdater::Get and the IndependentBath / DiagonalBath /
// FullBath / Vacuum terms (hierarchy_updater.h:36-75,
// hierarchy_updater.cc:10-144, :216-254), the RK4 stage combines
// (hierarchy_integrator.cc:2705-2826) and the RKF45 combines, error and
// control (:2010-2482).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "heom_device.cuh"
#include "heom_kernels.h"
#include "heom_tile.h"
#include "heom_tl_term.cuh"

namespace phi {
namespace {

__device__ __forceinline__ double2 c_axpy(double2 a, double2 b, double s) {
  return make_double2(fma(b.x, s, a.x), fma(b.y, s, a.y));
}
// Data that a preceding stage kernel wrote.
__device__ __forceinline__ double2 ld_global(const double2 *p) { return __ldcg(p); }
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
constexpr int kNodeThreads = 512;   // at most
constexpr int kNodeRounds = 2;      // elements of a thread whose neighbour sums stay in registers
constexpr int kNodeMaxOps = 5;      // combine operands

// Shape of a launch and its shared-memory plan (bytes, every region 16-byte
// aligned).
struct NodePlan {
  int threads;   // CTA size
  int nt;        // nodes per tile
  int cs;        // columns per round: threads / N
  int bc;        // full couplings: baths whose M_b are in shared memory at once
  int stage_ops; // combine operands staged in shared memory (0: read directly)
  uint32_t x, u, m, v, ops, cf, ids, bytes;
  int vb;        // full couplings: baths whose V_b are in shared memory at once (all, or bc)
};

struct StageParams {
  HeomConsts c;
  NodePlan plan;
  int mode;          // StageMode
  int stage;         // RK stage index
  const double2 *x;  // stage input (node-major)
  double2 *out;      // apply output / next stage input
  // RK4
  double2 *y;
  double2 *acc;
  double a_next;     // X_{s+1} = y + a_next * k
  double w_acc;      // accumulator weight
  Rk4Ctl *rk4;
  double2 *traj;
  // RKF45
  double2 *k[5];
  double2 *ybuf[2];
  Rkf45Ctl *ctl;
  // Combine operands in the order the epilogue reads them; RKF45's operand 0
  // is the state, chosen on the device.
  int nops;
  const double2 *op[kNodeMaxOps];
  // filtering (see StageLaunch)
  uint8_t *act[2];
  int act_par;
  // apply mode, gridDim.y > 1: block row y applies to x + y * x_bstride and
  // writes out + y * out_bstride (many inputs of one operator per launch)
  long long x_bstride, out_bstride;
};

// s: next prefactor magnitude; a = (previous scale) * c_t.
struct alignas(16) NodeCoef {
  double s, pad, ax, ay;
};

// What a kernel of its own keeps out of the others (registers and 0.6 % of a
// 6-state full coupling):
//   kTimeLocal  time-local runs of independent baths from 9 sites on, where each
//               element adds its own product of the term before the exchange;
//               the pair's term at both of its elements is twice the work (48
//               sites 27.3 ms for 32 RK4 steps, 13.1 so; 20 sites 3.79 and
//               2.18), which a few sites do not notice.
//   kVPerPass   full couplings whose V_b do not all fit (NodePlan::vb = bc).
enum NodeVariant : int { kPlain = 0, kTimeLocal = 1, kVPerPass = 2 };

template <int KIND, int VARIANT>
__global__ void __launch_bounds__(kNodeThreads) heom_node_kernel(const __grid_constant__ StageParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const HeomConsts &c = p.c;
  const NodePlan &pl = p.plan;
  const int N = c.N, E = N * N, T = c.T, tid = threadIdx.x, nth = blockDim.x;
  constexpr bool TL = VARIANT == kTimeLocal, VP = VARIANT == kVPerPass;
  const int NP = N | 1;  // odd column stride of the exchange tile: transposed reads in distinct banks
  double2 *Hs = reinterpret_cast<double2 *>(smem_raw);
  double2 *Xs = reinterpret_cast<double2 *>(smem_raw + pl.x);
  double2 *Us = reinterpret_cast<double2 *>(smem_raw + pl.u);
  double2 *Ms = reinterpret_cast<double2 *>(smem_raw + pl.m);
  double *Vs = reinterpret_cast<double *>(smem_raw + pl.v);
  double2 *Ops = reinterpret_cast<double2 *>(smem_raw + pl.ops);
  NodeCoef *cfs = reinterpret_cast<NodeCoef *>(smem_raw + pl.cf);
  int2 *ids = reinterpret_cast<int2 *>(smem_raw + pl.ids);

  const long long n0 = (long long)blockIdx.x * pl.nt;
  const int nt = (int)(c.M - n0 < pl.nt ? c.M - n0 : pl.nt);
  const int ncols = nt * N, tile = nt * E, step = pl.cs * N;
  const bool nb = !c.vacuum;
  if (c.filtered) pdl_wait();  // the records read the previous stage's flags
  const uint8_t *act_in = nullptr;
  if (c.filtered) act_in = p.act[p.mode == kModeRkf45 ? *(volatile int *)&p.ctl->ycur : p.act_par];
  // Records: neighbour ids (-1 absent; an inactive neighbour contributes
  // nothing, hierarchy_updater.cc:256-303) and coefficients.
  if (nb) {
    for (int q = tid; q < nt * T; q += nth) {
      const int t = q % T;
      int nx = __ldg(c.next + n0 * T + q), pv = __ldg(c.prev + n0 * T + q);
      const int occ = __ldg(c.mi + n0 * T + q);
      const double2 ct = __ldg(c.corr + t);
      if (act_in) {
        if (nx >= 0 && !__ldcg(act_in + nx)) nx = -1;
        if (pv >= 0 && !__ldcg(act_in + pv)) pv = -1;
      }
      // DiagonalBath is unnormalised (hierarchy_updater.cc:105-127).
      const double s = KIND == kDiagonal ? 1.0 : __ldg(c.sq_next + t * (c.L + 2) + occ);
      const double sp = KIND == kDiagonal ? (double)occ : __ldg(c.sq_prev + t * (c.L + 2) + occ);
      ids[q] = make_int2(nx, pv);
      cfs[q] = NodeCoef{s, 0.0, sp * ct.x, sp * ct.y};
    }
  }
  if (!c.filtered) pdl_wait();
  // One dependent in flight, not a chain of them: 924-node diagonal couplings
  // RK4 1.63 -> 1.53 ms (64 steps) against letting it go before the wait.
  pdl_launch_dependents();

  int ycur = 0;
  if (p.mode == kModeRkf45) {
    if (*(volatile int *)&p.ctl->done) return;  // uniform for the whole grid
    ycur = *(volatile int *)&p.ctl->ycur;
  }
  const double2 *xin = (p.mode == kModeRkf45 && p.stage == 0) ? p.ybuf[ycur] : p.x + blockIdx.y * p.x_bstride;
  // This thread's elements: e0 + r * step, row i, first column c0.
  const int i = tid % N, c0 = tid / N;
  const bool live = c0 < pl.cs;
  for (int e = tid; e < tile; e += nth) cp_async16(Xs + e, xin + n0 * E + e);
  if (pl.stage_ops && live) {
    for (int o = 0; o < p.nops; ++o) {
      const double2 *src = (p.mode == kModeRkf45 && o == 0) ? p.ybuf[ycur] : p.op[o];
      double2 *dst = Ops + (size_t)o * pl.nt * E;
      for (int e = tid; e < tile; e += step) cp_async16(dst + e, src + n0 * E + e);
    }
  }
  // An annealing run rewrites H (and V) between stages.
  double *Hr = reinterpret_cast<double *>(Hs);
  if (c.h_real) {
    for (int e = tid; e < E; e += nth) Hr[e] = __ldcg(c.H + e).x;
  } else {
    for (int e = tid; e < E; e += nth) Hs[e] = __ldcg(c.H + e);
  }
  if (KIND == kFull && nb)
    for (int e = tid; e < (VP ? pl.vb : c.nb) * E; e += nth) Vs[e] = __ldcg(c.bath_V + e);
  __syncthreads();  // records

  // The tile's X (and H) before the first read of them.
  bool have_x = false;
  auto need_x = [&]() {
    if (have_x) return;
    have_x = true;
    cp_async_wait();
    __syncthreads();
  };
  const double ih = c.inv_hbar;
  const int rounds = (ncols + pl.cs - 1) / pl.cs;
  const int K1 = c.K1;
  // The linked ADOs' values at offset off for `count` term records, four
  // terms' loads in flight at a time: use(n, X+, X-, record n's coefficients),
  // absent ADOs as zeros.
  auto gather = [&](int count, int off, auto record, bool with_next, auto use) {
    for (int n0t = 0; n0t < count; n0t += 4) {
      double2 g[4], h[4];
      int q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool on = n0t + u < count;
        q[u] = on ? record(n0t + u) : -1;
        const int2 id = on ? ids[q[u]] : make_int2(-1, -1);
        g[u] = with_next && id.x >= 0 ? ld_global(xin + (long long)id.x * E + off) : make_double2(0.0, 0.0);
        h[u] = id.y >= 0 ? ld_global(xin + (long long)id.y * E + off) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q[u] >= 0) use(n0t + u, g[u], h[u], cfs[q[u]]);
    }
  };
  // m += -i (s X+ + a X-)
  auto add_term = [](double2 &m, double2 g, double2 h, const NodeCoef &f) {
    m.x = fma(f.s, g.y, m.x);
    m.y = fma(-f.s, g.x, m.y);
    m.x = fma(f.ax, h.y, fma(f.ay, h.x, m.x));
    m.y = fma(f.ay, h.y, fma(-f.ax, h.x, m.y));
  };
  // (Q X - X Q^+)_ij of the deepest tier's time-local matrix Q_b.
  auto tl_deepest = [&](int nd) {
    int tier = 0;
    for (int t = 0; t < T; ++t) tier += __ldg(c.mi + (n0 + nd) * T + t);
    return tier == c.L;
  };
  auto tl_commutator = [&](int b, const double2 *X, int j) {
    const double2 *Q = c.tl_q + (size_t)b * E;
    double2 w = make_double2(0.0, 0.0);
    for (int k = 0; k < N; ++k) {
      const double2 qi = __ldcg(Q + i + k * N), qj = __ldcg(Q + j + k * N), xk = X[k + j * N], xi = X[i + k * N];
      w.x += qi.x * xk.x - qi.y * xk.y - (xi.x * qj.x + xi.y * qj.y);
      w.y += qi.x * xk.y + qi.y * xk.x - (xi.y * qj.x - xi.x * qj.y);
    }
    return w;
  };

  // Full couplings: the neighbour terms of baths b0 .. b0 + bn - 1 into Ms.
  auto full_terms = [&](int b0, int bn) {
    for (int r = 0; r < rounds; ++r) {
      const int col = c0 + r * pl.cs;
      if (!live || col >= ncols) continue;
      const int nd = col / N, off = i + (col - nd * N) * N;
      double2 m = make_double2(0.0, 0.0);
      int left = K1, b = 0;
      gather(bn * K1, off, [&](int n) { return nd * T + b0 * K1 + n; }, true,
             [&](int, double2 g, double2 h, const NodeCoef &f) {
               add_term(m, g, h, f);
               if (--left == 0) {
                 Ms[b * pl.nt * E + col * N + i] = m;
                 m = make_double2(0.0, 0.0);
                 left = K1;
                 ++b;
               }
             });
    }
  };
  if (KIND == kFull && nb) full_terms(0, c.nb < pl.bc ? c.nb : pl.bc);

  for (int r0 = 0; r0 < rounds; r0 += kNodeRounds) {
    double2 acc[kNodeRounds];
#pragma unroll
    for (int r = 0; r < kNodeRounds; ++r) {
      acc[r] = make_double2(0.0, 0.0);
      const int col = c0 + (r0 + r) * pl.cs;
      if (KIND == kFull || !nb || !live || col >= ncols) continue;
      const int nd = col / N, j = col - nd * N, off = i + j * N;
      if (KIND == kIndependent) {
        // Column j of the ADOs linked by the baths on site j: + i s X+ and
        // + i conj(c) sp X- (the next terms cancel on the diagonal).
        const int q0 = __ldg(c.site_ptr + j), nq = __ldg(c.site_ptr + j + 1) - q0;
        gather(nq, off, [&](int n) { return nd * T + __ldg(c.site_terms + q0 + n); }, i != j,
               [&](int, double2 g, double2 h, const NodeCoef &f) {
                 acc[r].x = fma(-f.s, g.y, acc[r].x);
                 acc[r].y = fma(f.s, g.x, acc[r].y);
                 acc[r].x = fma(f.ay, h.x, fma(-f.ax, h.y, acc[r].x));
                 acc[r].y = fma(f.ax, h.x, fma(f.ay, h.y, acc[r].y));
               });
      } else {
        gather(T, off, [&](int n) { return nd * T + n; }, true,
               [&](int n, double2 g, double2 h, const NodeCoef &f) {
                 double2 m = make_double2(0.0, 0.0);
                 add_term(m, g, h, f);
                 acc[r] = c_axpy(acc[r], m, __ldg(c.bath_V + (size_t)(n / K1) * N + i));
               });
      }
    }
    need_x();
    // A = H X: one H_ik serves the round's elements (elements past the tile
    // repeat its last column).
    int xo[kNodeRounds];
    double2 a[kNodeRounds];
#pragma unroll
    for (int r = 0; r < kNodeRounds; ++r) {
      const int col = c0 + (r0 + r) * pl.cs;
      xo[r] = (col < ncols ? col : ncols - 1) * N;
      a[r] = make_double2(0.0, 0.0);
    }
    if (c.h_real) {
#pragma unroll 4
      for (int k = 0; k < N; ++k) {
        const double h = Hr[i + k * N];
#pragma unroll
        for (int r = 0; r < kNodeRounds; ++r) {
          const double2 x = Xs[xo[r] + k];
          a[r].x = fma(h, x.x, a[r].x);
          a[r].y = fma(h, x.y, a[r].y);
        }
      }
    } else {
#pragma unroll 4
      for (int k = 0; k < N; ++k) {
        const double2 h = Hs[i + k * N];
#pragma unroll
        for (int r = 0; r < kNodeRounds; ++r) {
          const double2 x = Xs[xo[r] + k];
          a[r].x = fma(h.x, x.x, fma(-h.y, x.y, a[r].x));
          a[r].y = fma(h.x, x.y, fma(h.y, x.x, a[r].y));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kNodeRounds; ++r) {
      const int col = c0 + (r0 + r) * pl.cs;
      if (!live || col >= ncols) continue;
      if (KIND == kDiagonal && c.time_local && nb) {
        const int nd = col / N, j = col - nd * N;
        if (tl_deepest(nd))
          for (int b = 0; b < c.nb; ++b)
            acc[r] = c_axpy(acc[r], tl_commutator(b, Xs + nd * E, j), -__ldg(c.bath_V + (size_t)b * N + i));
      }
      Us[col * NP + i] = make_double2(fma(a[r].y, ih, acc[r].x), fma(-a[r].x, ih, acc[r].y));
    }
  }
  if (TL) {
    for (int r = 0; r < rounds; ++r) {
      const int col = c0 + r * pl.cs, nd = col / N, j = col - nd * N;
      if (!live || col >= ncols || i == j || !tl_deepest(nd)) continue;
      const double2 g = tl_half_term<double2>(Xs + nd * E, c.tl_q, N, i, j);
      double2 &u = Us[col * NP + i];
      u = make_double2(u.x + g.x, u.y + g.y);
    }
  }
  if (KIND == kFull && nb) {
    // M_b of up to bc baths at a time, then B += V_b M_b.
    for (int b0 = 0; b0 < c.nb; b0 += pl.bc) {
      const int bn = c.nb - b0 < pl.bc ? c.nb - b0 : pl.bc;
      if (b0 > 0) {
        __syncthreads();  // the previous baths' M_b (and V_b) are read
        if (VP)
          for (int e = tid; e < bn * E; e += nth) Vs[e] = __ldcg(c.bath_V + (size_t)b0 * E + e);
        full_terms(b0, bn);
        if (VP) __syncthreads();
      }
      for (int r = 0; r < rounds; ++r) {
        const int col = c0 + r * pl.cs;
        if (!live || col >= ncols) continue;
        const int nd = col / N, j = col - nd * N;
        const double2 *X = Xs + nd * E;
        const bool tl = c.time_local && tl_deepest(nd);
        for (int b = 0; b < bn; ++b) {
          // + Delta_b [X, V_b]
          const double *V = Vs + (size_t)(VP ? b : b0 + b) * E;
          double2 w = make_double2(0.0, 0.0), z = w;
#pragma unroll 4
          for (int k = 0; k < N; ++k) {
            w = c_axpy(w, X[i + k * N], V[k + j * N]);
            z = c_axpy(z, X[k + j * N], V[i + k * N]);
          }
          double2 &m = Ms[b * pl.nt * E + col * N + i];
          double2 v = c_axpy(m, make_double2(w.x - z.x, w.y - z.y), __ldg(c.mats_bath + b0 + b));
          if (tl) v = c_axpy(v, tl_commutator(b0 + b, X, j), -1.0);
          m = v;
        }
      }
      __syncthreads();
      for (int r = 0; r < rounds; ++r) {
        const int col = c0 + r * pl.cs;
        if (!live || col >= ncols) continue;
        double2 u = Us[col * NP + i], w = make_double2(0.0, 0.0);
        for (int b = 0; b < bn; ++b) {
          const double *V = Vs + (size_t)(VP ? b : b0 + b) * E + i;
          const double2 *M = Ms + b * pl.nt * E + col * N;
          int k = 0;
#pragma unroll 2
          for (; k + 1 < N; k += 2) {
            u = c_axpy(u, M[k], V[k * N]);
            w = c_axpy(w, M[k + 1], V[(k + 1) * N]);
          }
          if (k < N) u = c_axpy(u, M[k], V[k * N]);
        }
        Us[col * NP + i] = make_double2(u.x + w.x, u.y + w.y);
      }
    }
  }
  __syncthreads();

  // dX of each element and its combine.
  const double *coef = p.mode == kModeRkf45 ? p.ctl->coef : nullptr;
  auto cf = [&](int q) { return __ldcg(coef + q); };
  auto operand = [&](int o, int e) -> double2 {
    if (pl.stage_ops) return Ops[(size_t)o * pl.nt * E + e];
    const double2 *src = (p.mode == kModeRkf45 && o == 0) ? p.ybuf[ycur] : p.op[o];
    return ld_global(src + n0 * E + e);
  };
  const bool flags = c.filtered && ((p.mode == kModeRk4 && p.stage == 3) || (p.mode == kModeRkf45 && p.stage == 5));
  long long row = -1;  // rho_0 row this step writes
  if (p.mode == kModeRk4 && p.stage == 3 && n0 == 0 && p.traj) {
    const volatile Rk4Ctl *rc = p.rk4;
    if (rc->out_factor > 0 && rc->step % rc->out_factor == 0 && rc->nout < rc->capacity) row = rc->nout;
  }
  double emax = 0.0;
  for (int r = 0; r < rounds; ++r) {
    const int col = c0 + r * pl.cs;
    if (!live || col >= ncols) continue;
    const int nd = col / N, j = col - nd * N, e = tid + r * step;
    const long long g = n0 * E + e;
    const double2 *X = Xs + nd * E;
    const double2 b = Us[col * NP + i], bt = Us[(nd * N + i) * NP + j];
    double2 kv = make_double2(b.x + bt.x, i == j ? 0.0 : b.y - bt.y);
    if (nb) {
      // The upper triangle's X (a lower element is its conjugate).
      const double2 x = X[i <= j ? i + j * N : j + i * N];
      const double fac = __ldg(c.deph_node + n0 + nd) + __ldg(c.mats_elem + i + j * N);
      kv.x = fma(-fac, x.x, kv.x);
      kv.y = fma(i == j ? 0.0 : (i < j ? -fac : fac), x.y, kv.y);
    }
    if (KIND == kIndependent && !TL && c.time_local && i != j && tl_deepest(nd)) {
      const double2 tv = tl_pair_term<double2>(X, c.tl_q, N, i < j ? i : j, i < j ? j : i);
      kv.x += tv.x;
      kv.y += i < j ? tv.y : -tv.y;
    }
    double2 yn = kv;  // the new state, in the stages that write it
    if (p.mode == kModeApply) {
      p.out[blockIdx.y * p.out_bstride + g] = kv;
    } else if (p.mode == kModeRk4) {
      const int s = p.stage;
      if (s < 3) {
        const double2 ys = s == 0 ? X[i + j * N] : operand(0, e);
        p.out[g] = c_axpy(ys, kv, p.a_next);
        p.acc[g] = c_axpy(s == 0 ? ys : operand(1, e), kv, p.w_acc);
      } else {
        yn = c_axpy(operand(0, e), kv, p.w_acc);
        p.y[g] = yn;
        if (row >= 0 && e < E) p.traj[row * E + e] = yn;
      }
    } else if (p.stage < 5) {
      // X_{s+1} = y + sum_{r<=s} b_{s+1,r} k_r  (left to right, :2015-2200)
      const int s = p.stage, co = s * (s + 1) / 2;
      p.k[s][g] = kv;
      double2 xv = s == 0 ? X[i + j * N] : operand(0, e);
      for (int q = 0; q < s; ++q) xv = c_axpy(xv, operand(1 + q, e), cf(co + q));
      p.out[g] = c_axpy(xv, kv, cf(co + s));
    } else {
      const double2 ys = operand(0, e), k0 = operand(1, e), k2 = operand(2, e), k3 = operand(3, e),
                    k4 = operand(4, e);
      double2 y4 = c_axpy(ys, k0, cf(15));
      y4 = c_axpy(y4, k2, cf(16));
      y4 = c_axpy(y4, k3, cf(17));
      y4 = c_axpy(y4, k4, cf(18));
      yn = c_axpy(ys, k0, cf(19));
      yn = c_axpy(yn, k2, cf(20));
      yn = c_axpy(yn, k3, cf(21));
      yn = c_axpy(yn, k4, cf(22));
      yn = c_axpy(yn, kv, cf(23));
      p.ybuf[ycur ^ 1][g] = yn;
      const double err = hypot(y4.x - yn.x, y4.y - yn.y);
      emax = (err > emax || err != err) ? err : emax;
    }
    // X's own slot is free: no other thread reads it after the exchange
    // barrier except as the upper triangle above, so the norms wait below.
    if (flags) Ops[e] = make_double2(fma(yn.x, yn.x, yn.y * yn.y), 0.0);
  }
  if (p.mode == kModeRk4 && p.stage == 3 && n0 == 0 && p.traj) {
    __syncthreads();
    if (tid == 0) {
      Rk4Ctl *rc = p.rk4;
      if (row >= 0) rc->nout = rc->nout + 1;
      rc->step = rc->step + 1;
    }
  }
  if (flags) {
    // New flags of the state just written (hierarchy_integrator.cc:2827-2850,
    // :2359-2384): below the tolerance -> inactive, above -> active, equal
    // -> unchanged.  A NaN never wins the `>`, as in PHI's scan.
    __syncthreads();
    const int ap = p.mode == kModeRkf45 ? ycur : p.act_par;
    for (int nd = tid >> 5; nd < nt; nd += nth >> 5) {
      double m = 0.0;
      for (int w = tid & 31; w < E; w += 32) {
        const double v = Ops[nd * E + w].x;
        m = v > m ? v : m;
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, m, o);
        m = v > m ? v : m;
      }
      if ((tid & 31) == 0) {
        const double mx = sqrt(m);
        p.act[ap ^ 1][n0 + nd] =
            mx < c.filter_tol ? (uint8_t)0 : (mx > c.filter_tol ? (uint8_t)1 : __ldcg(p.act[ap] + n0 + nd));
      }
    }
  }
  if (p.mode == kModeRkf45 && p.stage == 5) {
    // max-reduce |y4 - y5| (hierarchy_integrator.cc:2317-2351); the bit
    // pattern of a non-negative double orders like the value (NaN above inf).
    // One atomic per CTA.
    unsigned long long bits = (unsigned long long)__double_as_longlong(emax);
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, bits, off);
      bits = o > bits ? o : bits;
    }
    __shared__ unsigned long long wmax[kNodeThreads / 32];
    if ((tid & 31) == 0) wmax[tid >> 5] = bits;
    __syncthreads();
    if (tid == 0) {
      unsigned long long m = wmax[0];
      for (int w = 1; w < nth / 32; ++w) m = wmax[w] > m ? wmax[w] : m;
      if (m) atomicMax(&p.ctl->err_bits, m);
    }
  }
}

// Accept/reject and step-size control of Rkf45Integrate
// (hierarchy_integrator.cc:2355-2482), one thread.  The accept test uses the
// step size the attempt was made with.
__global__ void rkf45_control_kernel(Rkf45Ctl *ctl) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (ctl->done) {
    ctl->tl_pending = 0;
    return;
  }
  ctl->tl_pending = 0;
  const double err = __longlong_as_double((long long)ctl->err_bits);
  ctl->err_bits = 0ull;
  const long long attempt = ctl->steps;
  if (ctl->err_trace && attempt < ctl->trace_cap) ctl->err_trace[attempt] = err;
  ctl->steps += 1;
  if (!(err == err) || err > 1.0e300) {
    ctl->nonfinite = 1;
    ctl->done = 1;
    ctl->status = 2;
    return;
  }
  bool accept = err < ctl->tol || ctl->dt * ctl->dtdn < ctl->min_dt;
  bool grow = err < ctl->tol / 10;
  if (ctl->forced && attempt < ctl->forced_len) {
    accept = ctl->forced[attempt] != 0;
    grow = ctl->forced[attempt] == 2;
  }
  if (accept) {
    // Time-local matrices advance by the rest of this attempt (dt - a5).
    ctl->tl_h_accept = ctl->dt - ctl->a[4];
    ctl->tl_pending = 1;
    ctl->ycur ^= 1;
    ctl->time += ctl->dt;
    ctl->accepted += 1;
    if (err > ctl->max_error) ctl->max_error = err;
    bool update = grow;
    if (ctl->time + ctl->dt > ctl->end_time) {
      update = true;
      ctl->dtup = (ctl->end_time - ctl->time) / ctl->dt;
    }
    if (update) {
      ctl->dt *= ctl->dtup;
      for (int q = 0; q < 24; ++q) ctl->coef[q] *= ctl->dtup;
      for (int q = 0; q < 5; ++q) ctl->a[q] *= ctl->dtup;
    }
  } else {
    ctl->dt *= ctl->dtdn;
    for (int q = 0; q < 24; ++q) ctl->coef[q] *= ctl->dtdn;
    for (int q = 0; q < 5; ++q) ctl->a[q] *= ctl->dtdn;
    ctl->tl_pending = 2;
  }
  if (!(ctl->time < ctl->end_time)) ctl->done = 1;
  if (!ctl->done && ctl->steps >= ctl->max_steps) {
    ctl->done = 1;
    ctl->status = 1;
  }
}

constexpr uint32_t kNodeMaxSmem = 224 * 1024;
// What one CTA can be given: 227 KiB less the kernel's static shared memory.
constexpr uint32_t kNodeSmemLimit = 227 * 1024 - 128;

uint32_t align16(uint32_t b) { return (b + 15u) & ~15u; }

// Shared-memory plan of nt nodes per tile with the combine's nops operands
// staged (or not) and bc baths' M_b at once.
void node_layout(const HeomConsts &c, int nops, bool flags, NodePlan *pl) {
  const uint32_t E = c.N * c.N, tile = (uint32_t)pl->nt * E * 16;
  uint32_t b = E * 16;  // H
  pl->x = b;
  b += tile;
  pl->u = b;
  b += (uint32_t)pl->nt * c.N * (c.N | 1) * 16;
  pl->m = b;
  if (c.kind == kFull && !c.vacuum) b += (uint32_t)pl->bc * tile;
  pl->v = b;
  if (c.kind == kFull && !c.vacuum) b += align16((uint32_t)pl->vb * E * 8);
  pl->ops = b;
  b += std::max<uint32_t>(pl->stage_ops ? nops : 0, flags ? 1 : 0) * tile;
  pl->cf = b;
  b += (uint32_t)pl->nt * c.T * sizeof(NodeCoef);
  pl->ids = b;
  b += align16((uint32_t)pl->nt * c.T * sizeof(int2));
  pl->bytes = b;
}

// Tile and CTA size: the cheapest of whole rounds of elements per thread (1 to
// 4) and CTA sizes under
//   waves * (2 + rounds) + CTAs per SM * (threads * rounds / 512 + 1/2):
// a CTA's chain of latencies (a round takes about as long as half the fixed
// part), the SM's element slots, and a CTA's fixed work.  Fitted to a sweep of
// 17 problems on B200 (N = 3 .. 20, 84 to 20,000 nodes): within 10 % of the
// best shape of the sweep, where a fixed 256-thread tile was up to 1.6 times
// slower.  The V_b of all baths are loaded once where that fits; where it does
// not with any shape (N = 48 with 5 baths, 30 with 32), those of each pass over bc
// baths are.  threads = 0: nothing fits.
NodePlan node_plan(const HeomConsts &c, int nops, bool flags, int num_sms) {
  const int N = c.N;
  NodePlan best{};
  double best_cost = 1e300;
  const auto search = [&](bool all_v) {
    for (int threads = 64; threads <= kNodeThreads; threads += 32) {
      const int cs = threads / N;
      if (cs < 1) continue;
      for (int want = 1; want <= 4; ++want) {
        NodePlan pl{};
        pl.nt = std::max(1, std::min<int>(want * cs / N, 64));
        const int rounds = (pl.nt * N + cs - 1) / cs;
        if (rounds < want && want > 1) continue;
        pl.threads = threads;
        pl.cs = cs;
        pl.bc = std::min(c.nb, 8);
        pl.vb = all_v ? c.nb : pl.bc;
        pl.stage_ops = nops > 0;
        node_layout(c, nops, flags, &pl);
        // Larger nodes: first read the operands directly, then take fewer
        // baths at once.
        if (pl.bytes > kNodeMaxSmem / 2 && pl.stage_ops) {
          pl.stage_ops = 0;
          node_layout(c, nops, flags, &pl);
        }
        while (pl.bytes > kNodeMaxSmem && pl.bc > 1 && c.kind == kFull) {
          --pl.bc;
          if (!all_v) pl.vb = pl.bc;
          node_layout(c, nops, flags, &pl);
        }
        if (pl.bytes > (pl.nt > 1 ? kNodeMaxSmem : kNodeSmemLimit)) continue;
        const int resident = std::max(1, std::min<int>(768 / threads, (int)(kNodeMaxSmem / pl.bytes)));
        const double tiles = (double)((c.M + pl.nt - 1) / pl.nt);
        const double per_sm = std::ceil(tiles / num_sms);
        const double cost = std::ceil(per_sm / resident) * (2.0 + rounds) + per_sm * (threads * rounds / 512.0 + 0.5);
        if (cost < best_cost) {
          best_cost = cost;
          best = pl;
        }
      }
    }
  };
  search(true);
  if (best.threads == 0 && c.kind == kFull) search(false);
  return best;
}

template <int KIND, int VARIANT = kPlain>
cudaError_t launch_node(const StageParams &p, int batch, cudaStream_t stream) {
  auto kern = heom_node_kernel<KIND, VARIANT>;
  static thread_local int raised[kSmemLimitDevices] = {};
  cudaError_t e = raise_smem_limit(kern, p.plan.bytes, raised);
  if (e != cudaSuccess) return e;
  return launch_dependent(true, kern, dim3((unsigned)((p.c.M + p.plan.nt - 1) / p.plan.nt), batch), dim3(p.plan.threads),
                          p.plan.bytes, stream, p);
}

}  // namespace

cudaError_t launch_stage(const StageLaunch &L, cudaStream_t stream) {
  if (!L.generic && tile_kernel_available(L.c)) {
    if (L.xv || L.outv || L.mixed) return launch_tile_stage(L, stream);
    StageLaunch T = L;  // complex128 caller: the typed pointers are the storage
    T.xv = L.x;
    T.outv = L.out;
    for (int i = 0; i < 5; ++i) T.kv[i] = L.k[i];
    return launch_tile_stage(T, stream);
  }
  if (L.mixed) return cudaErrorInvalidValue;  // mixed precision needs the tiled kernel
  StageParams p;
  p.c = L.c;
  p.mode = L.mode;
  p.stage = L.stage;
  p.x = L.x;
  p.out = L.out;
  p.y = L.y;
  p.acc = L.acc;
  p.a_next = L.a_next;
  p.w_acc = L.w_acc;
  p.rk4 = L.rk4;
  p.traj = L.traj;
  for (int i = 0; i < 5; ++i) p.k[i] = L.k[i];
  p.ybuf[0] = L.ybuf[0];
  p.ybuf[1] = L.ybuf[1];
  p.ctl = L.ctl;
  p.act[0] = L.act[0];
  p.act[1] = L.act[1];
  p.act_par = L.act_par;
  p.x_bstride = L.x_bstride;
  p.out_bstride = L.out_bstride;
  const int batch = L.batch;
  if (batch < 1 || batch > 65535 || (batch > 1 && L.mode != kModeApply)) return cudaErrorInvalidValue;
  // The combine's operands (see the kernel's epilogue).
  p.nops = 0;
  if (L.mode == kModeRk4) {
    if (L.stage == 1 || L.stage == 2) {
      p.op[p.nops++] = L.y;
      p.op[p.nops++] = L.acc;
    } else if (L.stage == 3) {
      p.op[p.nops++] = L.acc;
    }
  } else if (L.mode == kModeRkf45 && L.stage > 0) {
    p.op[p.nops++] = nullptr;  // the current state
    if (L.stage < 5)
      for (int r = 0; r < L.stage; ++r) p.op[p.nops++] = L.k[r];
    else
      for (int r : {0, 2, 3, 4}) p.op[p.nops++] = L.k[r];
  }
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return cudaErrorInvalidDevice;
  const bool flags = L.c.filtered && L.mode != kModeApply;
  p.plan = node_plan(L.c, p.nops, flags, sms);
  if (p.plan.threads == 0) return cudaErrorInvalidValue;
  switch (L.c.kind) {
    case kIndependent:
      return p.c.time_local && p.c.N > 8 ? launch_node<kIndependent, kTimeLocal>(p, batch, stream)
                                         : launch_node<kIndependent>(p, batch, stream);
    case kDiagonal: return launch_node<kDiagonal>(p, batch, stream);
    default:
      return p.plan.vb < p.c.nb ? launch_node<kFull, kVPerPass>(p, batch, stream) : launch_node<kFull>(p, batch, stream);
  }
}

namespace {
__global__ void to_c64_kernel(const double2 *in, float2 *out, long long M, int E, int EP) {
  const long long total = M * EP;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / EP;
    const int w = (int)(i - n * EP);
    const double2 v = w < E ? in[n * E + w] : make_double2(0.0, 0.0);
    out[i] = make_float2((float)v.x, (float)v.y);
  }
}
__global__ void to_c128_kernel(const float2 *in, double2 *out, long long M, int E, int EP) {
  const long long total = M * E;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / E;
    const int w = (int)(i - n * E);
    const float2 v = in[n * EP + w];
    out[i] = make_double2(v.x, v.y);
  }
}
int conv_blocks(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 148 * 16 ? 148 * 16 : b));
}
}  // namespace

cudaError_t launch_to_c64(const double2 *in, float2 *out, long long M, int E, int padded, cudaStream_t s) {
  to_c64_kernel<<<conv_blocks(M * padded), 256, 0, s>>>(in, out, M, E, padded);
  return cudaGetLastError();
}

cudaError_t launch_to_c128(const float2 *in, double2 *out, long long M, int E, int padded, cudaStream_t s) {
  to_c128_kernel<<<conv_blocks(M * E), 256, 0, s>>>(in, out, M, E, padded);
  return cudaGetLastError();
}

cudaError_t launch_rkf45_control(Rkf45Ctl *ctl, cudaStream_t stream) {
  rkf45_control_kernel<<<1, 32, 0, stream>>>(ctl);
  return cudaGetLastError();
}

}  // namespace phi
