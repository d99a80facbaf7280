// heom_tile_body.cuh -- the tiled IndependentBath stage (one tile of one
// hierarchy) shared by the single-instance kernel (heom_tile.cu) and the
// batched persistent kernel (heom_tile_batch.cu).  Internal header.
//
// The stage serves the IndependentBath model (PHI's default;
// hierarchy_updater.cc:129-144, :216-254) with a compile-time system size N,
// in two arithmetics:
//
//   FP64   every buffer complex128 (the path PHI computes).
//   MIXED  stage inputs X_s and stage derivatives k_s stored as complex64 and
//          the Liouvillian evaluated in FP32, and with it the next stage
//          input (X_{s+1} = y + sum b k) of RK4 stages 0-2 and RKF45
//          stages 0-4, which is stored as complex64; the state y, the RK4
//          accumulator, the fourth/fifth-order solutions, the RKF45 error
//          norm and the step control stay FP64.  A complex64 copy of y
//          (y32) is the stage-0 input.  complex64 buffers pad every node
//          to an even number of elements so each node range is 16-byte
//          aligned.
//
// A CTA of BT threads (kTileThreads = 256, or what the single-instance
// launch picks) owns a tile of NT consecutive nodes.  Everything the tile
// reads of its own nodes is contiguous in HBM and arrives by TMA bulk copies:
// its stage input X_s, its neighbour records and every epilogue operand
// (state y, RK4 accumulator, RKF45 k_r).  Per tile:
//
//   phase 1  neighbour records: element offsets and coefficients per (node,
//            term).
//   phase 2  (tile_derivative) A = H X from shared memory ([H, X] = A - A^+),
//            dephasing + Matsubara factor, and the neighbour terms from the
//            linked ADOs, gathered from L2 with independent predicated loads.
//            Only column m of an ADO linked by a bath on site m is read: the
//            row m of a Hermitian ADO is its conjugate.
//   phase 3  (tile_epilogue) plain store, RK4 or RKF45 stage combine, RKF45
//            error max; operands from shared memory.
//
// What bounds it (B200): latency -- shared-memory and L2 round trips and the
// tile's barriers at 20 to 32 warps per SM, issue slots 40-45 % used -- and
// the shared-memory pipe (60-69 % of peak in the 7-site kernel), not DRAM.
// Mapping the products and, outside the RKF45 stages of few sites, the
// neighbour terms by element instead of by upper-triangle pair measured:
// 16-site FP64 RK4 stage 37 -> 20 us, 24-site FP64 61 -> 45 us, 8-site mixed
// 9.1 -> 6.5 us, 4-site K = 2 FP64 apply 49 -> 36 us, 48 uneven instances in
// mixed precision 2.55 -> 1.76 ms per RK4 step.
//
// Stores of the next stage input use the default cache policy (its neighbour
// gathers in the next stage should hit L2); k and accumulator stores stream.
// This kernel serves PHI's identity site map (bath m on |m><m|, terms of site
// m are m*(K+1) .. m*(K+1)+K) with K+1 <= 3; other maps use the node
// kernel of heom_kernels.cu (FP64 only).
//
// Every mbarrier wait is bounded: after kMaxPolls polls the kernel records the
// failure in HeomConsts::err_flag, waits (bounded again) for its own copies,
// and returns; the host reports PHI_E_TIMEOUT.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "heom_device.cuh"
#include "heom_kernels.h"
#include "heom_tile.h"
#include "heom_tl_term.cuh"

namespace phi {
namespace tile_detail {

constexpr int kTileThreads = 256;             // threads per CTA
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kMaxPre = 5;  // epilogue operand buffers per launch
constexpr long long kMaxPolls = 1ll << 22;

struct TileParams {
  HeomConsts c;
  int mode;
  int stage;
  const void *x;        // stage input (TX)
  void *out;            // apply output / next stage input (TX)
  double2 *y;           // RK4 state
  double2 *acc;         // RK4 accumulator
  void *y32;            // MIXED RK4: complex64 copy of y (written at stage 3)
  double a_next;
  double w_acc;
  Rk4Ctl *rk4;
  double2 *traj;
  void *k[5];           // RKF45 k0..k4 (TX)
  double2 *ybuf[2];     // RKF45 state ping-pong
  void *y32buf[2];      // MIXED RKF45: complex64 copies of ybuf
  Rkf45Ctl *ctl;
  uint8_t *act[2];               // filtering: active flags (see StageLaunch)
  int act_par;
  const double2 *dot_w;          // FP64 apply: <dot_w, out> per CTA (see StageLaunch)
  double *dot_part;
  int dot_slots;
  int dependent;                 // launched as a dependent of the previous kernel
  int npre;                      // epilogue operands prefetched
  const void *pre[kMaxPre];      // sources; slot 0 of RKF45 is chosen on the device
  int pre_bytes[kMaxPre];        // 16 (complex128) or 8 (complex64)
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// One contiguous global -> shared copy (sizes and addresses multiples of 16 B).
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// A hint: the contiguous global range [src, src + bytes) is brought into L2
// (16-byte aligned address, size a multiple of 16 bytes); nothing waits on it.
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase with the given parity of `bar` to complete;
// false if it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  long long polls = kMaxPolls) {
  for (long long i = 0; i < polls; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Initialises the two mbarriers at the start of dynamic shared memory (one
// thread) and makes them visible to the CTA.
__device__ __forceinline__ void tile_init_barriers(unsigned char *smem_raw) {
  if (threadIdx.x == 0) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw);
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

// complex helpers over double2 / float2
__device__ __forceinline__ double2 to_d2(double2 v) { return v; }
__device__ __forceinline__ double2 to_d2(float2 v) { return make_double2(v.x, v.y); }
template <class TX> __device__ __forceinline__ TX from_d2(double2 v);
template <> __device__ __forceinline__ double2 from_d2<double2>(double2 v) { return v; }
template <> __device__ __forceinline__ float2 from_d2<float2>(double2 v) {
  return make_float2((float)v.x, (float)v.y);
}
template <class TX> __device__ __forceinline__ TX mk(double re, double im);
template <> __device__ __forceinline__ double2 mk<double2>(double re, double im) { return make_double2(re, im); }
template <> __device__ __forceinline__ float2 mk<float2>(double re, double im) {
  return make_float2((float)re, (float)im);
}
__device__ __forceinline__ double2 cfma(double2 acc, double2 b, double s) {
  return make_double2(fma(b.x, s, acc.x), fma(b.y, s, acc.y));
}
template <class TX> __device__ __forceinline__ void st_stream(TX *p, TX v) { __stcs(p, v); }

// Which kernel a tile shape is for: the single-instance apply and RK4 stages,
// the RKF45 stages, the batched stages, the resident RK4 run with one element
// per thread or several.
enum TileKind : int { kTileRk4 = 0, kTileRkf45 = 1, kTileBatch = 2, kTileResident = 3, kTileResidentWide = 4 };
constexpr bool tile_resident(int kind) { return kind == kTileResident || kind == kTileResidentWide; }

template <int N, bool MIXED, int KT, int BT = kTileThreads, int ST = kTileRk4>
struct TileShape {
  static constexpr int E = N * N;
  static constexpr int EP = E + (E & 1);  // complex64 node stride (16-byte aligned nodes)
  static constexpr int ES = MIXED ? EP : E;  // node stride of X / k buffers
  static constexpr int P = N * (N + 1) / 2;
  // How the neighbour terms are mapped (tile_derivative): by upper-triangle
  // pair, or by element.
  static constexpr bool kPairs = ST == kTileRkf45 && N < 10;
  // Thread t < CS * N works on row t % N of the tile's columns t / N, t / N +
  // CS, ...: one H_ik serves all of a thread's elements, and a warp's
  // gathers and stores run along whole columns.
  static constexpr int CS = BT / N;
  // Nodes per tile: one pair per thread, or 32 bytes of elements per thread
  // and operand.  A single hierarchy halves tiles of more than 40 nodes
  // (few sites), which would leave a small one too few CTAs (84-node trimer,
  // 256 RK4 steps: FP64 4.35 -> 3.80 ms, mixed 4.83 -> 4.07; 4-site mixed
  // apply over 125,970 nodes 29.9 -> 26.9 us); a batch has tiles enough and
  // takes the large ones (48 instances: 30.1 -> 28.1 ms).
  static constexpr int R1 = MIXED ? 4 : 2;
  static constexpr int kRounds = ST == kTileResident       ? 1
                                 : ST == kTileResidentWide ? R1
                                 : ST == kTileBatch        ? (!MIXED && R1 * CS / N > 40 ? 1 : R1)
                                 : R1 * CS / N <= 40       ? R1
                                 : 2 * CS / N <= 40        ? 2
                                                           : 1;
  static constexpr int NT0 = kPairs ? BT / P : kRounds * CS / N;
  static constexpr int NT = NT0 < 1 ? 1 : (NT0 > 64 ? 64 : NT0);
  static constexpr int RR = (NT * N + CS - 1) / CS;  // elements per thread
  static constexpr int PR = (NT * P + BT - 1) / BT;  // pairs per thread
  // The exchange tile's column stride is odd, so the transposed (j, i) reads
  // of one warp fall in distinct banks; an odd N shares X's offsets.
  static constexpr int NP = (N & 1) ? N : N + 1;
  static constexpr int EU = (N & 1) ? ES : N * NP;
};

template <int N, bool MIXED, int KT, int BT = kTileThreads, int ST = kTileRk4>
struct TileLayout {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  static constexpr int ES = S::ES;
  static constexpr int XB = MIXED ? 8 : 16;        // bytes per element of X / k
  // byte offsets in dynamic shared memory
  static constexpr size_t kBars = 0;
  static constexpr size_t kX = 128;
  static constexpr size_t kXBytes = ((size_t)S::NT * ES * XB + 127) / 128 * 128;
  static constexpr size_t kU = kX + kXBytes;
  static constexpr size_t kUBytes = ((size_t)S::NT * S::EU * XB + 127) / 128 * 128;
  static constexpr size_t kPre = kU + kUBytes;
};

// Resident warps per SM the register budget is fitted to: 24 (80 registers)
// unless 32 (64 registers) hold the shape without many spills and pay.  Timed
// 32 against 24: FP64 elements with one term per site 2.53 and 2.68 ms (16-site
// RK4, 32 steps), 9.65 and 9.82 (24-site, 64 steps), but 1.14 and 1.09 (7-site
// with 3,432 nodes); mixed pairs with two terms per site from 6 sites on 8.1 and
// 8.8 ms (7-site RKF45, 38,760 nodes; 3 to 5 % the other way below 1,000
// nodes).  Elsewhere 32 is slower, by up to 1.6 (mixed RK4 with two or three
// terms per site, which spill).
template <int N, int KT, bool MIXED, int BT, bool PAIRS>
struct TileMinBlocks {
  static constexpr int warps = MIXED ? (PAIRS && KT == 2 && N >= 6 ? 32 : 24) : (KT == 1 && !PAIRS ? 32 : 24);
  static constexpr int value = warps / (BT / 32);
};

// New filter flags of a tile's nodes from |y_new|^2 staged in the first 8
// bytes of each exchange-tile slot (slot bytes apart, column stride NP, node
// stride EU):
// one warp per node; below the tolerance -> inactive, above -> active, equal
// -> unchanged (hierarchy_integrator.cc:2827-2850, :2359-2384).  A NaN never
// wins the `>`, as in PHI's scan.  Kept out of line so its registers do not
// add to the tile body's.
static __device__ __noinline__ void tile_filter_flags(const unsigned char *us, int slot, int N, int NP, int EU, int nt_here,
                                               const uint8_t *act_in, uint8_t *act_out, double tol,
                                               int warps) {
  const int E = N * N, lane = threadIdx.x & 31;
  for (int nd = threadIdx.x >> 5; nd < nt_here; nd += warps) {
    double m = 0.0;
    for (int w = lane; w < E; w += 32) {
      const int col = w / N;
      const double v = *reinterpret_cast<const double *>(us + (size_t)(nd * EU + (w - col * N) + col * NP) * slot);
      m = v > m ? v : m;
    }
    for (int off = 16; off > 0; off >>= 1) {
      const double o = __shfl_xor_sync(0xffffffffu, m, off);
      m = o > m ? o : m;
    }
    if (lane == 0) {
      const double mx = sqrt(m);
      act_out[nd] = mx < tol ? (uint8_t)0 : (mx > tol ? (uint8_t)1 : act_in[nd]);
    }
  }
}

template <bool MIXED>
struct TileArith {
  using TX = typename std::conditional<MIXED, float2, double2>::type;
  using R = typename std::conditional<MIXED, float, double>::type;
};

// ---- the parts of one tile shared by the kernels ----
// One (node, term): prefactor magnitude s of the next ADO; the previous
// one's scale sp and c_t (pairs), or a = sp * c_t (elements).
template <class R, bool PAIRS>
struct TileCoef;
template <>
struct alignas(16) TileCoef<float, true> {
  float s, sp, cx, cy;
};
template <>
struct alignas(16) TileCoef<double, true> {  // c_t from its table: half the shared memory
  double s, sp;
};
template <class R>
struct alignas(16) TileCoef<R, false> {
  R s, pad, ax, ay;
};
template <class C, class R>
__device__ __forceinline__ C tile_coef(R s, R sp, double2 c) {
  C f;
  f.s = s;
  if constexpr (std::is_same<C, TileCoef<R, true>>::value) {
    f.sp = sp;
    if constexpr (std::is_same<R, float>::value) {
      f.cx = (R)c.x;
      f.cy = (R)c.y;
    }
  } else {
    f.pad = 0;
    f.ax = sp * (R)c.x;
    f.ay = sp * (R)c.y;
  }
  return f;
}
// Reserved per-warp words (even, so what follows stays 16-byte aligned).
__host__ __device__ constexpr int tile_warp_slots(int threads) { return (threads / 32 + 1) & ~1; }

// This thread's share of a tile, the same in every tile: element r is row i
// of column j of node nd.  Offsets of elements past the tile repeat its last
// column, so every read stays inside the tile's buffers.
template <int N, int KT, bool MIXED, int BT, int ST>
struct TileMap {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  int i;
  int xo[S::RR];   // element in X (and k buffers): nd * ES + i + j * N
  int ut[S::RR];   // its transpose in the exchange tile
  int rec[S::RR];  // nd * T + j * KT, the first record of site j
  unsigned live;   // bit r: the element is in the (full) tile
  // kPairs: upper-triangle pairs i | j << 8 | node << 16 (node NT: none).
  int ij[S::kPairs ? S::PR : 1];
  __device__ __forceinline__ explicit TileMap(const HeomConsts &c) {
    if constexpr (S::kPairs) {
#pragma unroll
      for (int r = 0; r < S::PR; ++r) {
        const int it = (int)threadIdx.x + r * BT;
        const int nd = it / S::P, u = it - nd * S::P;
        ij[r] = nd < S::NT ? (int)__ldg(c.pair_i + u) | (int)__ldg(c.pair_j + u) << 8 | nd << 16 : S::NT << 16;
      }
    }
    i = (int)threadIdx.x % N;
    const int c0 = (int)threadIdx.x / N;
    live = 0;
#pragma unroll
    for (int r = 0; r < S::RR; ++r) {
      int col = c0 + r * S::CS;
      if (c0 < S::CS && col < S::NT * N) live |= 1u << r;
      col = col < S::NT * N ? col : S::NT * N - 1;
      const int nd = col / N, j = col - nd * N;
      xo[r] = nd * S::ES + i + j * N;
      ut[r] = nd * S::EU + j + i * S::NP;
      rec[r] = col * KT;
    }
  }
  __device__ __forceinline__ bool on(int r, int nt_here) const {
    return ((live >> r) & 1u) && xo[r] < nt_here * S::ES;
  }
  __device__ __forceinline__ int j(int r) const { return rec[r] / KT % N; }
  __device__ __forceinline__ int nd(int r) const { return rec[r] / KT / N; }
  // its own offset in the exchange tile
  __device__ __forceinline__ int uo(int r) const { return (N & 1) ? xo[r] : rec[r] / KT * S::NP + i; }
  // its offset in complex128 buffers
  __device__ __forceinline__ int eo(int r) const { return S::ES == S::E ? xo[r] : xo[r] - nd(r); }
};
// A = H X of this thread's elements, from shared memory: k runs outside, so
// one H_ik serves all of the thread's elements and a warp's reads of X are
// broadcasts along its columns.
template <int N, int KT, bool MIXED, int BT, int ST>
__device__ __forceinline__ void tile_products(const HeomConsts &c, const TileMap<N, KT, MIXED, BT, ST> &m,
                                              const typename TileArith<MIXED>::TX *Xs,
                                              const typename TileArith<MIXED>::TX *Hs,
                                              typename TileArith<MIXED>::TX (&a)[TileShape<N, MIXED, KT, BT, ST>::RR]) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using TX = typename TileArith<MIXED>::TX;
  using R = typename TileArith<MIXED>::R;
#pragma unroll
  for (int r = 0; r < S::RR; ++r) a[r] = mk<TX>(0.0, 0.0);
  const TX *Xc = Xs - m.i;
  if (c.h_real) {
    const R *Hr = reinterpret_cast<const R *>(Hs) + m.i;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const R h = Hr[k * N];
#pragma unroll
      for (int r = 0; r < S::RR; ++r) {
        const TX x = Xc[m.xo[r] + k];
        a[r].x = fma(h, x.x, a[r].x);
        a[r].y = fma(h, x.y, a[r].y);
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const TX h = Hs[m.i + k * N];
#pragma unroll
      for (int r = 0; r < S::RR; ++r) {
        const TX x = Xc[m.xo[r] + k];
        a[r].x = fma(h.x, x.x, a[r].x);
        a[r].x = fma(-h.y, x.y, a[r].x);
        a[r].y = fma(h.x, x.y, a[r].y);
        a[r].y = fma(h.y, x.x, a[r].y);
      }
    }
  }
}

// An element of a linked ADO; a resident run reads what other CTAs of its
// launch wrote, past L1.
template <int ST, class TX>
__device__ __forceinline__ TX ld_neighbour(const TX *p) {
  return tile_resident(ST) ? __ldcg(p) : *p;
}

// What a tile's derivative is computed from (shared memory, except xin).
template <int N, int KT, bool MIXED, int BT, int ST>
struct TileIn {
  using TX = typename TileArith<MIXED>::TX;
  using R = typename TileArith<MIXED>::R;
  using C = TileCoef<R, TileShape<N, MIXED, KT, BT, ST>::kPairs>;
  const TX *Xs;         // the tile's stage input
  TX *Us;               // exchange tile
  const TX *Hs;         // H
  const R *mats;        // Matsubara factor per element
  const int2 *ids;      // neighbour element offsets (next, prev), -1 absent
  const C *cfs;         // neighbour coefficients
  const double2 *ccs;   // c_t (FP64 pairs)
  const double *deph;   // dephasing rates
  const uint8_t *mi;    // occupations (time-local truncation)
  const TX *xin;        // the stage input of every node (HBM)
  int nt_here;
  const int *next;      // next ids of the tile's nodes (the time-local kernels)
};

// The deepest tier's time-local term of element (i, j), i < j, of node nd.
template <int N, int KT, bool MIXED, int BT, int ST>
__device__ __forceinline__ bool tile_time_local(const HeomConsts &c, const TileIn<N, KT, MIXED, BT, ST> &in, int nd, int i,
                                                int j, typename TileArith<MIXED>::TX &tv) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  int tier = 0;  // deepest tier only (is_timelocal_truncated)
  for (int t = 0; t < N * KT; ++t) tier += in.mi[nd * N * KT + t];
  if (tier != c.L) return false;
  tv = tl_pair_term<typename TileArith<MIXED>::TX>(in.Xs + nd * S::ES, c.tl_q, N, i, j);
  return true;
}

// The time-local share of B, ((Q_j - Q_i) X)_ij (zero above the deepest tier,
// whose nodes alone have no next ones), of this thread's elements (TileMap's)
// into their places of the exchange tile, one product per element.
template <class TX>
__device__ __forceinline__ void tile_time_local_half(TX *Us, const TX *Xs, const int *next, const double2 *Q, int N, int T,
                                                     int ES, int EU, int NP, int CS, int ncols) {
  const int i = threadIdx.x % N, c0 = threadIdx.x / N;
  if (c0 >= CS) return;
  for (int col = c0; col < ncols; col += CS) {
    const int nd = col / N, j = col - nd * N;
    TX g;
    g.x = g.y = 0;
    if (i != j && next[nd * T] < 0) g = tl_half_term<TX>(Xs + nd * ES, Q, N, i, j);
    Us[nd * EU + i + j * NP] = g;
  }
}

// Whether the time-local truncation of a shape's stages has kernels of its own
// (TL below): elements, from 4 sites on.  With two or three sites, and by
// pairs, the general kernels add the pair's term, which costs little there.
constexpr bool tile_tl_kernels(int N, bool rkf45) { return N >= (rkf45 ? 10 : 4); }

// Phase 2: the derivative dx of this thread's elements of a tile.
//
// By element (kPairs off).  With
//   B_ij = -i/hbar (H X)_ij + sum_q (i s X+_ij + i conj(c) sp X-_ij)
// over the terms q of site j (column j of the linked ADOs), the derivative of
// a Hermitian ADO is dX_ij = B_ij + conj(B_ji) - (dephasing + Matsubara_ij)
// X_ij: the row parts of PHI's DoNext / DoPrevious are the conjugates of the
// transposed element's column parts.  Each thread forms B of its elements --
// a warp's gathers run along whole columns of the neighbours -- and the tile
// exchanges B through Us.
//
// By pair (RKF45 stages below N = 10).  The products go through Us, then a
// thread evaluates pair (i, j), both neighbour parts included, with the
// operations and in the order of the first such kernel: the error estimate
// of a stiff hierarchy (7 sites, K = 1, depth 6) is rounding amplified in the
// deep tiers, so another order of this sum accepts and rejects other steps,
// and a run can then end past t_end instead of at it (PHI's clamp does not
// see a grown step): 2 of 16 seeds in mixed precision.  From 10 sites on the
// order does not matter so: over 10 to 24 sites, K = 0 and 1, depths 2 to 6, both
// arithmetics and three seeds, 107 of 108 runs take the steps of the pair order
// (one 24-site mixed run 87 instead of 86) and all end at t_end.  There the pair
// mapping would take, over K = 0 to 2 and both arithmetics, 0.80 to 1.06 times the
// element mapping's time at 10 sites, 0.84 to 1.21 at 12, 1.01 to 1.38 at 16 and
// 0.90 to 1.23 at 24.
//
// Barriers: every thread of the CTA calls; Us must be free on entry, and is
// free again after the CTA's next barrier.
//
// TL: a time-local run of a shape with tile_tl_kernels.  The pair's term at both
// of its elements is twice the work (16-site mixed RK4 at 153 nodes 3.76 ms for
// 32 steps, 1.56 so), and the products in the general kernel cost the runs
// without them registers (10-site mixed RK4 at K = 2 up to 15 %).
template <int N, int KT, bool MIXED, int BT, int ST, bool TL = false>
__device__ __forceinline__ void tile_derivative(const HeomConsts &c, const TileMap<N, KT, MIXED, BT, ST> &m,
                                                const TileIn<N, KT, MIXED, BT, ST> &in,
                                                typename TileArith<MIXED>::TX (&dx)[TileShape<N, MIXED, KT, BT, ST>::RR]) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using TX = typename TileArith<MIXED>::TX;
  using R = typename TileArith<MIXED>::R;
  constexpr int ES = S::ES, NP = S::NP, EU = S::EU, RR = S::RR, T = N * KT;
  const R ih = (R)c.inv_hbar;
  const bool nb = !c.vacuum;
  const TX zero = mk<TX>(0.0, 0.0);
  TX *Us = in.Us;
  if constexpr (S::kPairs) {
    // FP64 of few sites: each pair forms its two products itself, which costs
    // less than the exchange and its barrier (6-site RKF45 2.85 -> 2.37 ms).
    constexpr bool kDirect = !MIXED && N <= 6;
    auto coupling = [&](int t, const auto &f) {  // c_t
      if constexpr (MIXED) return mk<TX>(f.cx, f.cy);
      else return in.ccs[t];
    };
    // Every neighbour value the pairs need, as independent predicated loads,
    // in mixed precision issued before the products, whose work hides their
    // latency (FP64 would spill).
    constexpr bool kHoist = MIXED;
    TX gn_c[S::PR][KT], gp_c[S::PR][KT], gn_r[S::PR][KT], gp_r[S::PR][KT];
    auto gather = [&](int r) {
      const int i = m.ij[r] & 255, j = m.ij[r] >> 8 & 255, nd = m.ij[r] >> 16;
      const bool on = nb && nd < in.nt_here;
      const int oij = i + j * N, oji = j + i * N, ndr = nd < S::NT ? nd : 0;
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        const int2 idj = in.ids[ndr * T + j * KT + q], idi = in.ids[ndr * T + i * KT + q];
        gn_c[r][q] = (on && idj.x >= 0 && i != j) ? *(in.xin + idj.x + oij) : zero;
        gp_c[r][q] = (on && idj.y >= 0 && i != j) ? *(in.xin + idj.y + oij) : zero;
        gn_r[r][q] = (on && idi.x >= 0 && i != j) ? *(in.xin + idi.x + oji) : zero;
        gp_r[r][q] = (on && idi.y >= 0) ? *(in.xin + idi.y + oji) : zero;
      }
    };
    if constexpr (kHoist) {
#pragma unroll
      for (int r = 0; r < S::PR; ++r) gather(r);
    }
    if constexpr (!kDirect) {
      tile_products<N, KT, MIXED, BT, ST>(c, m, in.Xs, in.Hs, dx);
#pragma unroll
      for (int r = 0; r < RR; ++r)
        if ((m.live >> r) & 1u) Us[m.uo(r)] = dx[r];
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < S::PR; ++r) {
      const int i = m.ij[r] & 255, j = m.ij[r] >> 8 & 255, nd = m.ij[r] >> 16;
      if (nd >= in.nt_here) continue;
      const int uij = nd * EU + i + j * NP, uji = nd * EU + j + i * NP;
      TX a = zero, b = zero;  // A_ij, A_ji
      if constexpr (!kDirect) {
        a = Us[uij];
        b = Us[uji];
      } else {
        const TX *X = in.Xs + nd * ES;
        if (c.h_real) {
          const R *Hr = reinterpret_cast<const R *>(in.Hs);
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const R hik = Hr[i + k * N], hjk = Hr[j + k * N];
            const TX xkj = X[k + j * N], xik = X[i + k * N];  // X_ki = conj(X_ik)
            a.x = fma(hik, xkj.x, a.x);
            a.y = fma(hik, xkj.y, a.y);
            b.x = fma(hjk, xik.x, b.x);
            b.y = fma(-hjk, xik.y, b.y);
          }
        } else {
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const TX hik = in.Hs[i + k * N], xkj = X[k + j * N];
            const TX hjk = in.Hs[j + k * N], xik = X[i + k * N];
            a.x = fma(hik.x, xkj.x, a.x);
            a.x = fma(-hik.y, xkj.y, a.x);
            a.y = fma(hik.x, xkj.y, a.y);
            a.y = fma(hik.y, xkj.x, a.y);
            b.x = fma(hjk.x, xik.x, b.x);
            b.x = fma(hjk.y, xik.y, b.x);
            b.y = fma(-hjk.x, xik.y, b.y);
            b.y = fma(hjk.y, xik.x, b.y);
          }
        }
      }
      if constexpr (!kHoist) gather(r);
      // -i/hbar (A_ij - conj(A_ji))
      R vx = (a.y + b.y) * ih, vy = -(a.x - b.x) * ih;
      if (nb) {
        const TX xij = in.Xs[nd * ES + i + j * N];
        const R fac = (R)in.deph[nd] + in.mats[i + j * N];
        vx = fma(-fac, xij.x, vx);
        vy = fma(-fac, xij.y, vy);
        if (i != j) {
#pragma unroll
          for (int q = 0; q < KT; ++q) {
            const auto fj = in.cfs[nd * T + j * KT + q], fi = in.cfs[nd * T + i * KT + q];
            const TX cj = coupling(j * KT + q, fj), ci = coupling(i * KT + q, fi);
            // column part: + p X+_ij (p = i s), + i conj(c) sp X-_ij
            vx = fma(-fj.s, gn_c[r][q].y, vx);
            vy = fma(fj.s, gn_c[r][q].x, vy);
            const TX g = gp_c[r][q];
            const R re = cj.x * g.x + cj.y * g.y, im = cj.x * g.y - cj.y * g.x;
            vx = fma(-fj.sp, im, vx);
            vy = fma(fj.sp, re, vy);
            // row part: - p conj(X+_ji), - i c sp conj(X-_ji)
            vx = fma(-fi.s, gn_r[r][q].y, vx);
            vy = fma(-fi.s, gn_r[r][q].x, vy);
            const TX h = gp_r[r][q];
            const R re2 = ci.x * h.x + ci.y * h.y, im2 = ci.y * h.x - ci.x * h.y;
            vx = fma(fi.sp, im2, vx);
            vy = fma(-fi.sp, re2, vy);
          }
        } else {
          // diagonal: next terms cancel; prev gives 2 sp Im(c) X-_mm
#pragma unroll
          for (int q = 0; q < KT; ++q) {
            const auto fi = in.cfs[nd * T + i * KT + q];
            vx = fma((R)2 * fi.sp * coupling(i * KT + q, fi).y, gp_r[r][q].x, vx);
          }
        }
      }
      TX v = mk<TX>(vx, vy);
      if (c.time_local && i != j) {
        TX tv;
        if (tile_time_local<N, KT, MIXED, BT, ST>(c, in, nd, i, j, tv)) {
          v.x += tv.x;
          v.y += tv.y;
        }
      }
      if (i == j) v.y = 0;
      Us[uij] = v;
      if (i != j) Us[uji] = mk<TX>(v.x, -v.y);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RR; ++r) dx[r] = Us[m.uo(r)];
  } else {
    const int i = m.i;
    if constexpr (TL) tile_time_local_half(Us, in.Xs, in.next, c.tl_q, N, T, ES, EU, NP, S::CS, in.nt_here * N);
    // The gathers before the products, whose work hides their latency, where the
    // registers allow.  After them instead: mixed RK4 3 to 29 % slower at one or
    // two terms per site (3 to 10 % faster at three from 16 sites on), FP64 of one
    // term 1 to 16 % slower.  FP64 RK4 of two or three terms would spill: 24 sites
    // 5.00 -> 6.44 ms, 5 to 8 sites at three 10 to 19 % (4 sites at two gain 10 %).
    // FP64 RKF45 of two is within 1 % either way at 10 to 16 sites; 24 sites take
    // 2.01 ms so and 1.74 after.
    constexpr bool kHoist = MIXED || KT == 1 || tile_resident(ST) || (KT == 2 && ST == kTileRkf45);
    TX gn[RR][KT], gp[RR][KT];
    auto gather = [&](int r) {
      const bool on = nb && m.on(r, in.nt_here);
      const int off = m.xo[r] - m.nd(r) * ES;
      const bool diag = m.j(r) == i;
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        const int2 id = in.ids[m.rec[r] + q];
        gn[r][q] = (on && id.x >= 0 && !diag) ? ld_neighbour<ST>(in.xin + id.x + off) : zero;
        gp[r][q] = (on && id.y >= 0) ? ld_neighbour<ST>(in.xin + id.y + off) : zero;
      }
    };
    if constexpr (kHoist) {
#pragma unroll
      for (int r = 0; r < RR; ++r) gather(r);
    }
    tile_products<N, KT, MIXED, BT, ST>(c, m, in.Xs, in.Hs, dx);
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      if constexpr (!kHoist) gather(r);
      R bx = dx[r].y * ih, by = -dx[r].x * ih;  // -i/hbar A
      if (nb) {
#pragma unroll
        for (int q = 0; q < KT; ++q) {
          const auto f = in.cfs[m.rec[r] + q];
          bx = fma(-f.s, gn[r][q].y, bx);
          by = fma(f.s, gn[r][q].x, by);
          bx = fma(f.ay, gp[r][q].x, bx);
          bx = fma(-f.ax, gp[r][q].y, bx);
          by = fma(f.ax, gp[r][q].x, by);
          by = fma(f.ay, gp[r][q].y, by);
        }
      }
      if (TL && m.on(r, in.nt_here)) {
        const TX g = Us[m.uo(r)];
        bx += g.x;
        by += g.y;
      }
      dx[r] = mk<TX>(bx, by);
      if ((m.live >> r) & 1u) Us[m.uo(r)] = dx[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const TX bt = Us[m.ut[r]];
      const int j = m.j(r);
      R vx = dx[r].x + bt.x, vy = i == j ? (R)0 : dx[r].y - bt.y;
      if (nb) {
        // The upper triangle's X (a lower element is its conjugate).
        const int nd = m.nd(r);
        const TX x = in.Xs[i <= j ? m.xo[r] : nd * ES + j + i * N];
        const R fac = (R)in.deph[nd] + in.mats[i + j * N];
        vx = fma(-fac, x.x, vx);
        vy = fma(i == j ? (R)0 : (i < j ? -fac : fac), x.y, vy);
      }
      dx[r] = mk<TX>(vx, vy);
    }
    if (!TL && c.time_local) {
#pragma unroll 1
      for (int r = 0; r < RR; ++r) {
        int j = 0, nd = 0;
#pragma unroll
        for (int q = 0; q < RR; ++q)
          if (q == r) {
            j = m.j(q);
            nd = m.nd(q);
          }
        TX tv;
        if (i == j || !tile_time_local<N, KT, MIXED, BT, ST>(c, in, nd, i < j ? i : j, i < j ? j : i, tv)) continue;
#pragma unroll
        for (int q = 0; q < RR; ++q)
          if (q == r) {
            dx[q].x += tv.x;
            dx[q].y += i < j ? tv.y : -tv.y;
          }
      }
    }
  }
}

// Byte offset of prefetched epilogue operand b: operand 0, then the others,
// one size apart (each padded to 128 bytes).
template <int N, int KT, bool MIXED, int BT, int ST>
__host__ __device__ __forceinline__ uint32_t tile_pre_size(int bytes) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  return ((uint32_t)S::NT * (bytes == 16 ? S::E : S::ES) * bytes + 127) / 128 * 128;
}
template <int N, int KT, bool MIXED, int BT, int ST>
__host__ __device__ __forceinline__ uint32_t tile_pre_off(const TileParams &p, int b) {
  return b == 0 ? 0
                : tile_pre_size<N, KT, MIXED, BT, ST>(p.pre_bytes[0]) + (b - 1) * tile_pre_size<N, KT, MIXED, BT, ST>(p.pre_bytes[1]);
}

// Phase 3: the epilogue of this thread's elements (plain store, RK4 or RKF45
// stage combine) from its derivatives dx and the prefetched operands at
// Pre; the RKF45 stage-5 error is folded into emax (max of |y4 - y5|, or of
// its square in mixed precision), an apply's inner product added to it.  coef holds the 24 RKF45 coefficients in
// FP64 followed by the same 24 in FP32.
template <int N, int KT, bool MIXED, int BT, int ST>
__device__ __forceinline__ void tile_epilogue(const TileParams &p, const TileMap<N, KT, MIXED, BT, ST> &m,
                                              const TileIn<N, KT, MIXED, BT, ST> &in, const unsigned char *Pre,
                                              const double *coef, long long n0, int ycur, double &emax,
                                              const typename TileArith<MIXED>::TX (&dx)[TileShape<N, MIXED, KT, BT, ST>::RR]) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using TX = typename TileArith<MIXED>::TX;
  using R = typename TileArith<MIXED>::R;
  constexpr int E = S::E, ES = S::ES, RR = S::RR;
  constexpr bool RKF = ST == kTileRkf45;
  const int tid = threadIdx.x;
  // Element r of this thread: m.xo[r] in the tile's X / k ranges, m.eo(r) in
  // its complex128 ranges (and in the operands staged from either).
  const long long gx0 = n0 * ES, gd0 = n0 * E;
  const uint32_t off1 = tile_pre_off<N, KT, MIXED, BT, ST>(p, 1);
  const uint32_t offs = tile_pre_size<N, KT, MIXED, BT, ST>(p.pre_bytes[1]);
  const double2 *pre0d = reinterpret_cast<const double2 *>(Pre);
  const TX *pre0x = reinterpret_cast<const TX *>(Pre);
  // New filter flags follow: |y_new|^2 of every element goes to its slot of
  // the exchange tile once every thread has read its transposed elements.
  const bool flags = p.c.filtered && p.stage == (RKF ? 5 : 3) && (RKF || p.mode == kModeRk4);
  if (flags) __syncthreads();
  auto fl_put = [&](int r, double2 v) {
    *reinterpret_cast<double *>(&in.Us[m.uo(r)]) = fma(v.x, v.x, v.y * v.y);
  };
  if (!RKF && p.mode == kModeApply) {
    TX *out = static_cast<TX *>(p.out) + gx0;
    bool dot = false;
    if constexpr (!MIXED) dot = p.dot_w != nullptr;
    if (!dot) {
#pragma unroll
      for (int r = 0; r < RR; ++r)
        if (m.on(r, in.nt_here)) st_stream(out + m.xo[r], dx[r]);
    } else if constexpr (!MIXED) {
      // Steady-state solve: the output's element (0,0) of node 0 is the
      // eliminated unknown (zero), and this thread's share of <dot_w, out>
      // (the real inner product of Hermitian states; pre = {dot_w}) is added
      // up over the CTA's tiles -- the inner product the solver would
      // otherwise read the vector for.
#pragma unroll
      for (int r = 0; r < RR; ++r)
        if (m.on(r, in.nt_here)) {
          TX v = dx[r];
          if (gx0 + m.xo[r] == 0) v = mk<TX>(0.0, 0.0);
          st_stream(out + m.xo[r], v);
          const double2 w = pre0d[m.xo[r]];
          emax = fma(w.x, v.x, fma(w.y, v.y, emax));
        }
    }
  } else if (!RKF) {  // RK4
    const int s = p.stage;
    TX *out = static_cast<TX *>(p.out) + gx0;
    long long row = -1;
    if (s == 3 && n0 == 0 && p.traj) {
      const Rk4Ctl *rc = p.rk4;
      if (rc->out_factor > 0 && rc->step % rc->out_factor == 0 && rc->nout < rc->capacity) row = rc->nout;
    }
    const double2 *pre1d = reinterpret_cast<const double2 *>(Pre + off1);
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      if (!m.on(r, in.nt_here)) continue;
      const int x = m.xo[r], e = m.eo(r);
      const TX kx = dx[r];
      if (MIXED && s < 3) {
        // Mixed: the complex64 stage input y32 + a k in FP32 (stage 0: y32
        // is the input; stages 1-2: pre = {y32, acc}); the accumulator in
        // FP64 (stage 0: pre = {y}).
        const float af = (float)p.a_next;
        const TX ys = s == 0 ? in.Xs[x] : pre0x[x];
        out[x] = mk<TX>(fmaf((float)kx.x, af, (float)ys.x), fmaf((float)kx.y, af, (float)ys.y));
        st_stream(p.acc + gd0 + e, cfma((s == 0 ? pre0d : pre1d)[e], to_d2(kx), p.w_acc));
      } else if (s == 0) {  // FP64: pre = {} (y is the input)
        const double2 ys = to_d2(in.Xs[x]);
        out[x] = from_d2<TX>(cfma(ys, to_d2(kx), p.a_next));
        st_stream(p.acc + gd0 + e, cfma(ys, to_d2(kx), p.w_acc));
      } else if (s < 3) {  // pre = {y, acc}
        out[x] = from_d2<TX>(cfma(pre0d[e], to_d2(kx), p.a_next));
        st_stream(p.acc + gd0 + e, cfma(pre1d[e], to_d2(kx), p.w_acc));
      } else {             // pre = {acc}
        const double2 yn = cfma(pre0d[e], to_d2(kx), p.w_acc);
        p.y[gd0 + e] = yn;
        if (MIXED) static_cast<TX *>(p.y32)[gx0 + x] = from_d2<TX>(yn);
        if (row >= 0 && e < E) p.traj[row * E + e] = yn;
        if (flags) fl_put(r, yn);
      }
    }
    if (s == 3 && n0 == 0 && p.traj) {
      __syncthreads();
      if (tid == 0) {
        Rk4Ctl *rc = p.rk4;
        if (row >= 0) rc->nout = rc->nout + 1;
        rc->step = rc->step + 1;
      }
    }
  } else if (p.stage < 5) {
    // RKF45 stages 0-4: k_s and X_{s+1} = y + sum b k, in the storage type's
    // arithmetic (a complex64 stage input combined in FP32 differs from an
    // FP64 combine rounded to it by an ulp of complex64).  pre = {y, k_0 ..
    // k_{s-1}} (stage 0: y is the input); y is staged as y32 (mixed), staged
    // in complex128, or read from global memory (0 bytes).
    const int s = p.stage;
    TX *out = static_cast<TX *>(p.out) + gx0, *ks = static_cast<TX *>(p.k[s]) + gx0;
    const R *cf = MIXED ? reinterpret_cast<const R *>(coef + 24) : reinterpret_cast<const R *>(coef);
    cf += s * (s + 1) / 2;
    TX xv[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int x = m.xo[r];
      if (s == 0) {
        xv[r] = in.Xs[x];
      } else if (MIXED || p.pre_bytes[0] != 0) {
        xv[r] = pre0x[x];
      } else {
        xv[r] = m.on(r, in.nt_here) ? from_d2<TX>(__ldcg(p.ybuf[ycur] + gd0 + x)) : mk<TX>(0.0, 0.0);
      }
    }
    const TX *kb = reinterpret_cast<const TX *>(Pre + off1);
#pragma unroll 1
    for (int b = 0; b < s; ++b) {
      const R cb = cf[b];
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        const TX kr = kb[m.xo[r]];
        xv[r].x = fma(kr.x, cb, xv[r].x);
        xv[r].y = fma(kr.y, cb, xv[r].y);
      }
      kb = reinterpret_cast<const TX *>(reinterpret_cast<const unsigned char *>(kb) + offs);
    }
    const R cs = cf[s];
#pragma unroll
    for (int r = 0; r < RR; ++r)
      if (m.on(r, in.nt_here)) {
        const int x = m.xo[r];
        st_stream(ks + x, dx[r]);
        out[x] = mk<TX>(fma(dx[r].x, cs, xv[r].x), fma(dx[r].y, cs, xv[r].y));
      }
  } else {
    // RKF45 stage 5: pre = {y (or read from global), k0, k2, k3, k4}.
    const double *cf = coef;
    const TX *kb = reinterpret_cast<const TX *>(Pre + off1);
    const uint32_t ksz = offs / sizeof(TX);
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      if (!m.on(r, in.nt_here)) continue;
      const int x = m.xo[r], e = m.eo(r);
      const double2 kv = to_d2(dx[r]);
      const double2 ys = p.pre_bytes[0] == 0 ? __ldcg(p.ybuf[ycur] + gd0 + e) : pre0d[e];
      const double2 k0 = to_d2(kb[x]), k2 = to_d2(kb[ksz + x]);
      const double2 k3 = to_d2(kb[2 * ksz + x]), k4 = to_d2(kb[3 * ksz + x]);
      double2 y4 = cfma(ys, k0, cf[15]);
      y4 = cfma(y4, k2, cf[16]);
      y4 = cfma(y4, k3, cf[17]);
      y4 = cfma(y4, k4, cf[18]);
      double2 y5 = cfma(ys, k0, cf[19]);
      y5 = cfma(y5, k2, cf[20]);
      y5 = cfma(y5, k3, cf[21]);
      y5 = cfma(y5, k4, cf[22]);
      y5 = cfma(y5, kv, cf[23]);
      st_stream(p.ybuf[ycur ^ 1] + gd0 + e, y5);
      if (MIXED) st_stream(static_cast<TX *>(p.y32buf[ycur ^ 1]) + gx0 + x, from_d2<TX>(y5));
      if (flags) fl_put(r, y5);
      const double ex = y4.x - y5.x, ey = y4.y - y5.y;
      if (MIXED) {
        // max of |y4 - y5|^2; one square root per thread below
        const double e2 = fma(ex, ex, ey * ey);
        emax = (e2 > emax || e2 != e2) ? e2 : emax;
      } else {
        // |z| as PHI computes it (std::abs of the complex difference)
        const double err = hypot(ex, ey);
        emax = (err > emax || err != err) ? err : emax;
      }
    }
  }
}

// The RKF45 stage-5 error of a CTA: the maximum over its threads' emax, one
// atomicMax on the bit pattern of the control block's error word.
template <bool MIXED, int BT>
__device__ __forceinline__ void tile_error_max(const TileParams &p, double emax, unsigned long long *wmax) {
  const int tid = threadIdx.x;
  if (MIXED) emax = sqrt(emax);
  unsigned long long bits = (unsigned long long)__double_as_longlong(emax);
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, bits, off);
    bits = o > bits ? o : bits;
  }
  // One atomic per CTA: a single error word takes every CTA's maximum,
  // so per-warp atomics would serialise tens of thousands of updates.
  if ((tid & 31) == 0) wmax[tid >> 5] = bits;
  __syncthreads();
  if (tid == 0) {
    unsigned long long m = wmax[0];
#pragma unroll
    for (int w = 1; w < (BT / 32); ++w) m = wmax[w] > m ? wmax[w] : m;
    if (m) atomicMax(&p.ctl->err_bits, m);
  }
}

// An apply's inner product: the sum over the CTA's threads into its slot, in
// warp order; CTA 0 zeroes the slots past the grid.
template <int BT>
__device__ __forceinline__ void tile_dot_sum(const TileParams &p, double dsum, unsigned long long *wmax) {
  const int tid = threadIdx.x;
  for (int off = 16; off > 0; off >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, off);
  double *wsum = reinterpret_cast<double *>(wmax);
  if ((tid & 31) == 0) wsum[tid >> 5] = dsum;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < BT / 32; ++w) t += wsum[w];
    p.dot_part[blockIdx.x] = t;
  }
  if (blockIdx.x == 0)
    for (int q = (int)gridDim.x + tid; q < p.dot_slots; q += BT) p.dot_part[q] = 0.0;
}

// New filter flags of a tile's nodes after the stage that writes the new
// state (RK4 stage 3, RKF45 stage 5).
template <int N, int KT, bool MIXED, int BT, int ST>
__device__ __forceinline__ void tile_flags(const TileParams &p, const typename TileArith<MIXED>::TX *Us, long long n0,
                                           int nt_here, int ycur) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using TX = typename TileArith<MIXED>::TX;
  const HeomConsts &c = p.c;
  constexpr bool RKF = ST == kTileRkf45;
  if (!(c.filtered && p.stage == (RKF ? 5 : 3) && (RKF || p.mode == kModeRk4))) return;
  // Below the tolerance -> inactive, above -> active, equal -> unchanged
  // (hierarchy_integrator.cc:2827-2850, :2359-2384).
  __syncthreads();
  const int ap = RKF ? ycur : p.act_par;
  tile_filter_flags(reinterpret_cast<const unsigned char *>(Us), (int)sizeof(TX), N, S::NP, S::EU, nt_here,
                    p.act[ap] + n0, p.act[ap ^ 1] + n0, c.filter_tol, BT / 32);
}


// KT = terms per site (K + 1) under PHI's identity site map.
// One tile (NT consecutive nodes of one hierarchy) of one stage.  The caller
// has initialised the two mbarriers at the start of shared memory and passes
// the phase parity each is at.  Returns 1 when the tile was skipped before
// any copy was issued, 0 when both barriers completed a
// phase (barrier 1 with 0 bytes when p.npre == 0), -1 after a bounded wait gave up
// (err_flag set; the caller must stop).
template <int N, int KT, bool MIXED, int BT = kTileThreads>
__device__ __forceinline__ int tile_body(const TileParams &p, long long tile, unsigned char *smem_raw,
                                         uint32_t par0, uint32_t par1) {
  constexpr int ST = kTileBatch;  // apply and RK4 stages
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using Lay = TileLayout<N, MIXED, KT, BT, ST>;
  using TX = typename std::conditional<MIXED, float2, double2>::type;
  using R = typename std::conditional<MIXED, float, double>::type;
  constexpr int E = S::E, NT = S::NT, ES = Lay::ES;
  using In = TileIn<N, KT, MIXED, BT, ST>;
  const HeomConsts &c = p.c;
  constexpr int T = N * KT;  // PHI's identity site map: K+1 terms per site
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + Lay::kBars);
  TX *Xs = reinterpret_cast<TX *>(smem_raw + Lay::kX);   // NT*ES
  TX *Us = reinterpret_cast<TX *>(smem_raw + Lay::kU);   // NT*EU (column stride NP)
  unsigned char *PreBase = smem_raw + Lay::kPre;
  const size_t tail = Lay::kPre + (p.npre > 0 ? tile_pre_off<N, KT, MIXED, BT, ST>(p, p.npre) : 0);
  TX *Hs = reinterpret_cast<TX *>(smem_raw + tail);                 // E
  double *deph = reinterpret_cast<double *>(Hs + E + (E & 1));       // NT (16-aligned)
  typename In::C *cfs = reinterpret_cast<typename In::C *>(deph + NT + (NT & 1));  // NT*T neighbour coefficients
  R *mats = reinterpret_cast<R *>(cfs + NT * T);                    // E    Matsubara factor per element
  int2 *ids = reinterpret_cast<int2 *>(mats + E + (E & 1));         // NT*T element offsets (next, prev)

  const int tid = threadIdx.x;
  const long long n0 = tile * NT;
  if (n0 >= c.M) return 1;
  const int nt_here = (int)((c.M - n0) < NT ? (c.M - n0) : NT);
  const TX *xin = static_cast<const TX *>(p.x);

  // ---- t = 0: bulk prefetch of the tile's contiguous ranges ----
  if (tid == 0) {
    const uint32_t xbytes = (uint32_t)(nt_here * ES * Lay::XB);
    mbar_expect_tx(&bars[0], xbytes);
    bulk_g2s(Xs, xin + n0 * ES, xbytes, &bars[0]);
    uint32_t pbytes = 0;
#pragma unroll
    for (int b = 0; b < kMaxPre; ++b)
      if (b < p.npre) pbytes += (uint32_t)(nt_here * (p.pre_bytes[b] == 16 ? E : ES) * p.pre_bytes[b]);
    // Arrives on barrier 1 in every tile (with 0 bytes when nothing is
    // prefetched), so its phase advances once per tile like barrier 0's.
    mbar_expect_tx(&bars[1], pbytes);
#pragma unroll
    for (int b = 0; b < kMaxPre; ++b) {
      if (b >= p.npre) break;
      const unsigned char *src = static_cast<const unsigned char *>(p.pre[b]);
      const int stride = p.pre_bytes[b] == 16 ? E : ES;
      const uint32_t bytes = (uint32_t)(nt_here * stride * p.pre_bytes[b]);
      bulk_g2s(PreBase + tile_pre_off<N, KT, MIXED, BT, ST>(p, b), src + (size_t)n0 * stride * p.pre_bytes[b], bytes, &bars[1]);
    }
  }
  // A real Hamiltonian (every in-scope workload) is kept as E reals in the
  // same buffer, halving the products of A = H X.
  const bool hreal = c.h_real;
  R *Hr = reinterpret_cast<R *>(Hs);
  if (hreal) {
    for (int i = tid; i < E; i += BT) Hr[i] = (R)__ldg(c.H + i).x;
  } else {
    for (int i = tid; i < E; i += BT) Hs[i] = from_d2<TX>(__ldg(c.H + i));
  }
  for (int i = tid; i < E; i += BT) mats[i] = (R)__ldg(c.mats_elem + i);
  const int W = c.L + 2;
  const int tile_terms = nt_here * T;
  // Per (node, term): neighbour ids scaled to element offsets of the stage
  // input (-1 when absent), occupation, and the prefactor magnitudes for that
  // occupation, so the pair loop reads shared memory only.
  const uint8_t *act_in = c.filtered ? p.act[p.act_par] : nullptr;
  for (int q = tid; q < tile_terms; q += BT) {
    const int t = q % T;
    const int nx = __ldg(c.next + n0 * T + q), pv = __ldg(c.prev + n0 * T + q);
    const int nt = __ldg(c.mi + n0 * T + q);
    // An inactive neighbour contributes nothing (the DoNext / DoPrevious
    // overrides of IndependentBathAdaptiveTruncation, hierarchy_updater.cc:256-303).
    const bool nx_on = nx >= 0 && (!act_in || __ldg(act_in + nx));
    const bool pv_on = pv >= 0 && (!act_in || __ldg(act_in + pv));
    ids[q] = make_int2(nx_on ? nx * ES : -1, pv_on ? pv * ES : -1);
    cfs[q] = tile_coef<typename In::C, R>((R)__ldg(c.sq_next + t * W + nt), (R)__ldg(c.sq_prev + t * W + nt),
                                          __ldg(c.corr + t));
  }
  if (tid < nt_here) deph[tid] = __ldg(c.deph_node + n0 + tid);
  const long long polls0 = c.first_wait_polls == 0 ? kMaxPolls : (c.first_wait_polls < 0 ? 0 : c.first_wait_polls);
  bool ok = mbar_wait_bounded(&bars[0], par0, polls0);
  if (!__syncthreads_and(ok)) {  // metadata visible as well
    if (tid == 0) atomicOr(c.err_flag, 1);
    // Drain this tile's own copies with the built-in limit, so no copy is
    // still writing into shared memory when the CTA stops.
    mbar_wait_bounded(&bars[0], par0);
    if (p.npre > 0) mbar_wait_bounded(&bars[1], par1);
    return -1;
  }

  const TileMap<N, KT, MIXED, BT, ST> m(c);
  const In in{Xs, Us, Hs, mats, ids, cfs, nullptr, deph, c.mi + n0 * T, xin, nt_here, nullptr};
  TX dx[S::RR];
  tile_derivative<N, KT, MIXED, BT, ST>(c, m, in, dx);
  ok = p.npre == 0 || mbar_wait_bounded(&bars[1], par1);
  if (!__syncthreads_and(ok)) {
    if (tid == 0) atomicOr(c.err_flag, 1);
    return -1;
  }
  double emax = 0.0;
  tile_epilogue<N, KT, MIXED, BT, ST>(p, m, in, PreBase, nullptr, n0, 0, emax, dx);
  tile_flags<N, KT, MIXED, BT, ST>(p, Us, n0, nt_here, 0);
  return 0;
}

// Shared memory of a batched tile.
template <int N, int KT, bool MIXED, int BT = kTileThreads, int ST = kTileBatch>
inline size_t tile_smem(int T, int npre, const int *pre_bytes) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using Lay = TileLayout<N, MIXED, KT, BT, ST>;
  size_t b = Lay::kPre;
  for (int i = 0; i < npre; ++i) b += tile_pre_size<N, KT, MIXED, BT, ST>(pre_bytes[i]);
  b += (size_t)(S::E + (S::E & 1)) * Lay::XB;
  b += (size_t)(S::NT + (S::NT & 1)) * sizeof(double);  // deph
  b += (size_t)S::NT * T * sizeof(typename TileIn<N, KT, MIXED, BT, ST>::C);
  b += (size_t)(S::E + (S::E & 1)) * Lay::XB / 2;                     // mats
  b += (size_t)S::NT * T * sizeof(int2);                              // ids
  b += 16;
  return b;
}

// Threads per CTA of the single-instance kernel: 320 for the 24-site mixed
// kernel (20,475 nodes: RKF45 step 0.88 ms against 1.00 with 256, RK4 step 0.58
// against 0.65), 256 otherwise (320 everywhere was slower on the 7-site and the
// batched workloads).  The batched kernel always runs 256, so its tile counts
// (tile_count) use that.
template <int N, bool MIXED>
struct TileBlock {
  static constexpr int threads = (MIXED && N == 24) ? 320 : kTileThreads;
  // The autotuner's alternative block size (heom_tile.cu, tile_autotune).
  static constexpr int alt = threads == kTileThreads ? 320 : kTileThreads;
};

// The tile parameters of one stage launch (host; heom_tile.cu).
TileParams tile_params_for(const StageLaunch &L);

// Launches of the single-instance kernel (heom_tile_*_*.cu); *per_sm
// (optional) receives the resident CTAs per SM before the schedule's cap.
cudaError_t launch_tile_fp64_rk4(const TileParams &p, cudaStream_t stream, int *per_sm);
cudaError_t launch_tile_fp64_rkf45(const TileParams &p, cudaStream_t stream, int *per_sm);
cudaError_t launch_tile_mixed_rk4(const TileParams &p, cudaStream_t stream, int *per_sm);
cudaError_t launch_tile_mixed_rkf45(const TileParams &p, cudaStream_t stream, int *per_sm);
// The same for time-local runs of the shapes with kernels of their own.
cudaError_t launch_tile_fp64_rk4_tl(const TileParams &p, cudaStream_t stream, int *per_sm);
cudaError_t launch_tile_fp64_rkf45_tl(const TileParams &p, cudaStream_t stream, int *per_sm);
cudaError_t launch_tile_mixed_rk4_tl(const TileParams &p, cudaStream_t stream, int *per_sm);
cudaError_t launch_tile_mixed_rkf45_tl(const TileParams &p, cudaStream_t stream, int *per_sm);

}  // namespace tile_detail
}  // namespace phi
