// heom_tile_pipe.cuh -- the persistent tile kernel of one IndependentBath
// hierarchy and its launch.  Each including file instantiates it for one
// arithmetic and one kind of stage (RKF: RKF45; otherwise apply and RK4), for
// time-local runs or in general, so the sets compile side by side.  Internal
// header.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "heom_tile_body.cuh"

namespace phi {

using namespace tile_detail;

namespace {

// ---- persistent pipelined kernel ----
//
// A CTA stays resident and walks the tiles blockIdx.x, blockIdx.x +
// gridDim.x, ...  While tile i computes, the stage input X and the neighbour
// records (next / prev ids and occupations, contiguous per tile) of tile i+1
// arrive in the other of two shared-memory slots by cp.async.bulk; the
// epilogue operands of tile i (y, accumulator, k_r) are issued when tile i
// starts and land while its derivative runs; tile i+1's neighbour offsets and
// coefficients are prepared at the end of tile i, so one barrier ends a tile
// and starts the next.  H, the Matsubara factors, c_t and the prefactor tables
// are staged once per CTA: while the first tile's copies run, or, in a
// dependent launch, before the wait on the previous stage's kernel.
// mbarriers: one per slot (phase parity (i >> 1) & 1 for the CTA's i-th
// tile) and one for the epilogue operands (parity i & 1).
//
// The products A = H X stay on the CUDA cores at every N.  A split-TF32
// tcgen05.mma of the 24-site mixed tile (rows (node, column, re / im), A
// re-laid out and split per tile, accumulators read back from TMEM into the
// exchange tile) took longer, because the operands' shared memory and two
// barriers cost more than the 28 k FMAs of a node: 24-site RKF45 step 1.20 ms
// against 0.87, and rho_0 after 47 steps 1.0e-6 off against 1.8e-7.
template <int N, int KT, bool MIXED, int BT, int ST>
struct PipeLayout {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  static constexpr int T = N * KT;
  static constexpr int ES = S::ES;
  using C = typename TileIn<N, KT, MIXED, BT, ST>::C;
  static constexpr int XB = MIXED ? 8 : 16;
  static constexpr int RB = MIXED ? 4 : 8;  // bytes of the arithmetic type
  static constexpr size_t r16(size_t b) { return (b + 15) / 16 * 16; }
  static constexpr size_t r128(size_t b) { return (b + 127) / 128 * 128; }
  // One slot: the tile's X, then its next ids, prev ids (int32),
  // occupations (uint8) and dephasing rates (double), each copied from the
  // 16-byte aligned window around the tile's records (up to 3 ids, 15
  // bytes or 1 rate of slack on either side).
  static constexpr size_t kSlotX = r128((size_t)S::NT * ES * XB);
  static constexpr size_t kSlotIds = r16(((size_t)S::NT * T + 8) * 4);
  static constexpr size_t kSlotMi = r16((size_t)S::NT * T + 32);
  static constexpr size_t kSlotDeph = r16(((size_t)S::NT + 2) * 8);  // per-node dephasing rates
  static constexpr size_t kSlot = r128(kSlotX + 2 * kSlotIds + kSlotMi + kSlotDeph);
  static constexpr size_t kSlots = 128;                       // after the mbarriers
  static constexpr size_t kUs = kSlots + 2 * kSlot;           // exchange tile
  static constexpr size_t kPre = kUs + r128((size_t)S::NT * S::EU * XB);
};

template <int N, int KT, bool MIXED, int BT, int ST>
size_t pipe_smem(int T, int L, int npre, const int *pre_bytes) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using Lay = PipeLayout<N, KT, MIXED, BT, ST>;
  size_t b = Lay::kPre;
  for (int i = 0; i < npre; ++i) b += tile_pre_size<N, KT, MIXED, BT, ST>(pre_bytes[i]);
  const int W = L + 2, TW = T * W + ((T * W) & 1), E2 = S::E + (S::E & 1);
  b += (size_t)E2 * Lay::XB;                                          // H
  b += (size_t)(36 + tile_warp_slots(BT)) * sizeof(double);           // coef (FP64, FP32), warp maxima
  b += (size_t)2 * S::NT * T * sizeof(typename Lay::C);               // neighbour coefficients of two tiles
  b += (size_t)T * sizeof(double2);                                   // c_t
  b += (size_t)(E2 + 2 * TW) * Lay::RB;                               // mats, prefactor tables
  b += (size_t)2 * S::NT * T * sizeof(int2);                          // neighbour offsets of two tiles
  b += 16;
  return b;
}

template <int N, int KT, bool MIXED, int BT, int ST, bool TL>
__global__ void __launch_bounds__(BT, TileMinBlocks<N, KT, MIXED, BT, TileShape<N, MIXED, KT, BT, ST>::kPairs>::value) heom_tile_pipe_kernel(TileParams p) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  using Lay = PipeLayout<N, KT, MIXED, BT, ST>;
  using TX = typename TileArith<MIXED>::TX;
  using R = typename TileArith<MIXED>::R;
  using C = typename Lay::C;
  constexpr bool RKF = ST == kTileRkf45;
  constexpr int E = S::E, E2 = E + (E & 1), NT = S::NT, ES = Lay::ES, T = N * KT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const HeomConsts &c = p.c;
  const int tid = threadIdx.x;

  uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw);
  TX *Us = reinterpret_cast<TX *>(smem_raw + Lay::kUs);
  unsigned char *PreBase = smem_raw + Lay::kPre;
  const size_t tail = Lay::kPre + (p.npre > 0 ? tile_pre_off<N, KT, MIXED, BT, ST>(p, p.npre) : 0);
  const int W = c.L + 2, TW = T * W + ((T * W) & 1);
  TX *Hs = reinterpret_cast<TX *>(smem_raw + tail);                           // E
  double *coef = reinterpret_cast<double *>(Hs + E2);                         // 24, then 24 floats
  unsigned long long *wmax = reinterpret_cast<unsigned long long *>(coef + 36);  // per-warp maxima
  C *cfs = reinterpret_cast<C *>(wmax + tile_warp_slots(BT));                 // 2 * NT*T
  double2 *ccs = reinterpret_cast<double2 *>(cfs + 2 * NT * T);               // T    c_t
  R *mats = reinterpret_cast<R *>(ccs + T);                                   // E
  R *sqn = mats + E2;                                                         // T*W
  R *sqp = sqn + TW;                                                          // T*W
  int2 *ids = reinterpret_cast<int2 *>(sqp + TW);                             // 2 * NT*T (next, prev)

  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_init(&bars[2], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const long long ntiles = (c.M + NT - 1) / NT;
  long long tile = blockIdx.x;
  int ycur = 0;
  const TX *xin = static_cast<const TX *>(p.x);

  // Thread 0: the X and neighbour records of `tile` into slot s.
  auto issue_slot = [&](long long tile, int s) {
    const long long n0 = tile * NT;
    const int nt = (int)((c.M - n0) < NT ? (c.M - n0) : NT);
    unsigned char *b = smem_raw + Lay::kSlots + (size_t)s * Lay::kSlot;
    const long long q0 = n0 * T, q1 = q0 + (long long)nt * T;
    const long long a4 = q0 & ~3ll, e4 = (q1 + 3) & ~3ll, a16 = q0 & ~15ll, e16 = (q1 + 15) & ~15ll;
    const long long a2 = n0 & ~1ll, e2 = (n0 + nt + 1) & ~1ll;
    const uint32_t xbytes = (uint32_t)(nt * ES * Lay::XB), idbytes = (uint32_t)((e4 - a4) * 4),
                   mibytes = (uint32_t)(e16 - a16), dbytes = (uint32_t)((e2 - a2) * 8);
    mbar_expect_tx(&bars[s], xbytes + 2 * idbytes + mibytes + dbytes);
    bulk_g2s(b, xin + n0 * ES, xbytes, &bars[s]);
    bulk_g2s(b + Lay::kSlotX, c.next + a4, idbytes, &bars[s]);
    bulk_g2s(b + Lay::kSlotX + Lay::kSlotIds, c.prev + a4, idbytes, &bars[s]);
    bulk_g2s(b + Lay::kSlotX + 2 * Lay::kSlotIds, c.mi + a16, mibytes, &bars[s]);
    bulk_g2s(b + Lay::kSlotX + 2 * Lay::kSlotIds + Lay::kSlotMi, c.deph_node + a2, dbytes, &bars[s]);
  };
  // What needs the previous kernel's results: false once the RKF45 run is done
  // (uniform across the grid), else the first tile's copies.
  auto begin = [&]() {
    if (RKF) {
      if (*(volatile int *)&p.ctl->done) return false;
      ycur = *(volatile int *)&p.ctl->ycur;
      if (p.stage == 0)
        xin = MIXED ? static_cast<const TX *>(p.y32buf[ycur]) : reinterpret_cast<const TX *>(p.ybuf[ycur]);
    }
    if (tid == 0 && tile < ntiles) issue_slot(tile, 0);
    return true;
  };
  if (p.dependent) {
    if (RKF) pdl_launch_dependents();
    if (c.h_dynamic) pdl_wait();  // H is read below
  } else if (!begin()) {
    return;
  }
  const bool hreal = c.h_real;
  R *Hr = reinterpret_cast<R *>(Hs);
  if (hreal) {
    for (int i = tid; i < E; i += BT) Hr[i] = (R)__ldcg(c.H + i).x;
  } else {
    for (int i = tid; i < E; i += BT) Hs[i] = from_d2<TX>(__ldcg(c.H + i));
  }
  for (int i = tid; i < E; i += BT) mats[i] = (R)__ldg(c.mats_elem + i);
  for (int t = tid; t < T; t += BT) ccs[t] = __ldg(c.corr + t);
  for (int q = tid; q < T * W; q += BT) {
    sqn[q] = (R)__ldg(c.sq_next + q);
    sqp[q] = (R)__ldg(c.sq_prev + q);
  }
  if (p.dependent) {
    pdl_wait();
    if (!begin()) return;
  }
  // Filtering: an inactive neighbour contributes nothing (the DoNext /
  // DoPrevious overrides of IndependentBathAdaptiveTruncation,
  // hierarchy_updater.cc:256-303).
  const uint8_t *act_in = c.filtered ? p.act[RKF ? ycur : p.act_par] : nullptr;
  const long long polls0 = c.first_wait_polls == 0 ? kMaxPolls : (c.first_wait_polls < 0 ? 0 : c.first_wait_polls);

  if (RKF && tid < 24) {
    const double v = __ldcg(&p.ctl->coef[tid]);
    coef[tid] = v;
    reinterpret_cast<float *>(coef + 24)[tid] = (float)v;
  }
  __syncthreads();  // barriers initialised, constants visible

  // Thread 0: the epilogue operands of `tile`.
  auto issue_pre = [&](long long tile) {
    const long long n0 = tile * NT;
    const int nt = (int)((c.M - n0) < NT ? (c.M - n0) : NT);
    uint32_t pbytes = 0;
#pragma unroll
    for (int b = 0; b < kMaxPre; ++b)
      if (b < p.npre) pbytes += (uint32_t)(nt * (p.pre_bytes[b] == 16 ? E : ES) * p.pre_bytes[b]);
    mbar_expect_tx(&bars[2], pbytes);
#pragma unroll
    for (int b = 0; b < kMaxPre; ++b) {
      if (b >= p.npre) break;
      if (p.pre_bytes[b] == 0) {
        // Read from global memory in the epilogue (the RKF45 state y): an
        // L2 prefetch of the tile's contiguous range now, so the epilogue's
        // loads do not wait for DRAM.
        if (RKF && b == 0)
          bulk_prefetch_l2(p.ybuf[ycur] + (size_t)n0 * E, (uint32_t)((size_t)nt * E * sizeof(double2)));
        continue;
      }
      const unsigned char *src = static_cast<const unsigned char *>(p.pre[b]);
      if (RKF && b == 0)
        src = static_cast<const unsigned char *>(p.pre_bytes[0] == 8 ? p.y32buf[ycur] : (const void *)p.ybuf[ycur]);
      const int stride = p.pre_bytes[b] == 16 ? E : ES;
      bulk_g2s(PreBase + tile_pre_off<N, KT, MIXED, BT, ST>(p, b), src + (size_t)n0 * stride * p.pre_bytes[b],
               (uint32_t)(nt * stride * p.pre_bytes[b]), &bars[2]);
    }
  };

  // Slot s holds a tile's records from (n0 * T) & 15 on (ids from & 3).
  auto slot = [&](int s) { return smem_raw + Lay::kSlots + (size_t)s * Lay::kSlot; };
  auto slot_mi = [&](int s, long long n0) {
    return reinterpret_cast<const uint8_t *>(slot(s) + Lay::kSlotX + 2 * Lay::kSlotIds) + ((n0 * T) & 15);
  };
  auto slot_next = [&](int s, long long n0) {
    return reinterpret_cast<const int *>(slot(s) + Lay::kSlotX) + ((n0 * T) & 3);
  };
  // Per (node, term) of the tile in slot s: neighbour element offsets (-1 when
  // absent or inactive) and coefficients.
  auto records = [&](long long tile, int s) {
    const long long n0 = tile * NT;
    const int nt = (int)((c.M - n0) < NT ? (c.M - n0) : NT);
    const unsigned char *sb = slot(s);
    const int *nx_s = slot_next(s, n0);
    const int *pv_s = reinterpret_cast<const int *>(sb + Lay::kSlotX + Lay::kSlotIds) + ((n0 * T) & 3);
    const uint8_t *mi_s = slot_mi(s, n0);
    for (int q = tid; q < nt * T; q += BT) {
      const int t = q % T;
      const int nx = nx_s[q], pv = pv_s[q], occ = mi_s[q];
      const bool nx_on = nx >= 0 && (!act_in || __ldcg(act_in + nx));
      const bool pv_on = pv >= 0 && (!act_in || __ldcg(act_in + pv));
      ids[s * NT * T + q] = make_int2(nx_on ? nx * ES : -1, pv_on ? pv * ES : -1);
      cfs[s * NT * T + q] = tile_coef<C, R>(sqn[t * W + occ], sqp[t * W + occ], ccs[t]);
    }
  };

  const TileMap<N, KT, MIXED, BT, ST> m(c);
  double emax = 0.0;
  int i = 0;
  // ok: this thread's waits so far; checked by the whole CTA at the barrier
  // that ends a tile.  That barrier also frees the tile's slot, operands and
  // exchange tile and publishes the next tile's records.
  bool ok = true, failed = false, next_issued = false;
  if (tile < ntiles) {
    ok = mbar_wait_bounded(&bars[0], 0, polls0);
    if (ok) records(tile, 0);
    if (!__syncthreads_and(ok)) {
      if (tid == 0) atomicOr(c.err_flag, 1);
      mbar_wait_bounded(&bars[0], 0);
      return;
    }
  }
  for (; tile < ntiles; ++i, tile += gridDim.x) {
    const int s = i & 1;
    const long long n0 = tile * NT;
    const int nt_here = (int)((c.M - n0) < NT ? (c.M - n0) : NT);
    next_issued = tile + gridDim.x < ntiles;
    // The next kernel may start from each CTA's last tile on: released at
    // the start, its CTAs took the places that freed up first and a chain of
    // waiting kernels built up (16-site FP64 RK4 3.02 ms for 32 steps, 2.53
    // so; 3-site 1.01 and 0.83 ms).  RKF45 stages, which are dependents only
    // with one tile per CTA, are 1-2 % faster released at the start.
    if (!RKF && p.dependent && !next_issued) pdl_launch_dependents();
    if (tid == 0) {
      if (next_issued) issue_slot(tile + gridDim.x, s ^ 1);
      if (p.npre > 0) issue_pre(tile);
    }
    const unsigned char *sb = slot(s);
    const TX *Xs = reinterpret_cast<const TX *>(sb);
    const double *deph =
        reinterpret_cast<const double *>(sb + Lay::kSlotX + 2 * Lay::kSlotIds + Lay::kSlotMi) + (n0 & 1);
    const TileIn<N, KT, MIXED, BT, ST> in{Xs,   Us,   Hs, mats, ids + s * NT * T, cfs + s * NT * T,
                                      ccs, deph, slot_mi(s, n0), xin, nt_here, slot_next(s, n0)};
    TX dx[S::RR];
    tile_derivative<N, KT, MIXED, BT, ST, TL>(c, m, in, dx);
    // The operands have had the derivative's time to land.  A wait that gave
    // up skips the stores; the tile's last barrier then ends the CTA.
    ok = p.npre == 0 || mbar_wait_bounded(&bars[2], (uint32_t)i & 1u);
    if (!RKF || c.filtered) {
      // These epilogues may hold CTA barriers of their own.
      if (!__syncthreads_and(ok)) {
        failed = true;
        break;
      }
    }
    if (ok) tile_epilogue<N, KT, MIXED, BT, ST>(p, m, in, PreBase, coef, n0, ycur, emax, dx);
    tile_flags<N, KT, MIXED, BT, ST>(p, Us, n0, nt_here, ycur);
    if (next_issued) {
      const bool got = mbar_wait_bounded(&bars[s ^ 1], (uint32_t)((i + 1) >> 1) & 1u, polls0);
      if (got) records(tile + gridDim.x, s ^ 1);
      ok = ok && got;
    }
    if (!__syncthreads_and(ok)) {
      failed = true;
      break;
    }
  }
  if (failed) {
    // Record the failure and drain this CTA's copies in flight with the
    // built-in limit, so none is still writing into shared memory at exit
    // (this tile's X arrived before its derivative).
    if (tid == 0) atomicOr(c.err_flag, 1);
    const int s = i & 1;
    if (next_issued) mbar_wait_bounded(&bars[s ^ 1], (uint32_t)((i + 1) >> 1) & 1u);
    if (p.npre > 0) mbar_wait_bounded(&bars[2], (uint32_t)i & 1u);
    return;
  }
  if (RKF && p.stage == 5) tile_error_max<MIXED, BT>(p, emax, wmax);
  if (!RKF && !MIXED && p.dot_w) tile_dot_sum<BT>(p, emax, wmax);
}

// Resident CTAs per SM of a kernel at a dynamic shared-memory size and the
// SM count of the current device, cached per (kernel, size, device).
struct OccEntry {
  const void *fn;
  size_t smem;
  int dev;
  int grid;
};

int persistent_grid(const void *fn, int threads, size_t smem) {
  static thread_local OccEntry cache[64];
  static thread_local int used = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  for (int k = 0; k < used; ++k)
    if (cache[k].fn == fn && cache[k].smem == smem && cache[k].dev == dev) return cache[k].grid;
  int sms = 0, blocks = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, threads, smem) != cudaSuccess) return 0;
  const int grid = sms * (blocks > 0 ? blocks : 1);
  if (used < 64) cache[used++] = OccEntry{fn, smem, dev, grid};
  return grid;
}

// Launch of one block-size variant.  The grid is the resident-CTA count of
// this launch's shared-memory size (capped at tile_cps CTAs per SM when the
// schedule sets it) and never more than the tiles.  *per_sm (optional)
// receives the resident CTAs per SM before the cap.
template <int N, int KT, bool MIXED, int BT, int ST, bool TL>
cudaError_t launch_tile_bt(const TileParams &p, cudaStream_t stream, int *per_sm = nullptr) {
  using S = TileShape<N, MIXED, KT, BT, ST>;
  const long long tiles = (p.c.M + S::NT - 1) / S::NT;
  auto kern = heom_tile_pipe_kernel<N, KT, MIXED, BT, ST, TL>;
  static thread_local int raised[kSmemLimitDevices] = {};
  const size_t smem = pipe_smem<N, KT, MIXED, BT, ST>(p.c.T, p.c.L, p.npre, p.pre_bytes);
  cudaError_t e = raise_smem_limit(kern, smem, raised);
  if (e != cudaSuccess) return e;
  int cap = persistent_grid((const void *)kern, BT, smem);
  if (cap <= 0) return cudaErrorInvalidConfiguration;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return cudaErrorInvalidDevice;
  if (per_sm) *per_sm = cap / sms;
  if (p.c.tile_cps > 0 && p.c.tile_cps * sms < cap) cap = p.c.tile_cps * sms;
  if (p.dot_w && p.dot_slots < cap) cap = p.dot_slots;
  const long long grid = tiles < cap ? tiles : cap;
  // Dependent launch (the preamble overlaps the previous kernel) for the RK4
  // stages, the apply, and RKF45 stages of one tile per CTA: 8-site mixed RK4
  // stage 6.5 -> 5.5 us, 84-node trimer 4.0 -> 3.0 us, 4-site apply 37.2 -> 34.5
  // us, 7-site FP64 RK4 3.44 -> 3.22 ms (64 steps), 24-site 1.42 -> 1.31.  RKF45
  // stages of several tiles per CTA gain nothing (7-site mixed 9.61 -> 9.57
  // ms, FP64 8.67 -> 8.91) and keep the plain launch.
  TileParams d = p;
  d.dependent = ST == kTileRk4 || tiles <= cap;
  return launch_dependent(d.dependent, kern, dim3((unsigned)grid), dim3(BT), smem, stream, d);
}

template <int N, int KT, bool MIXED, int ST, bool TL>
cudaError_t launch_tile_nk(const TileParams &p, cudaStream_t stream, int *per_sm = nullptr) {
  if (p.c.tile_variant == 1)
    return launch_tile_bt<N, KT, MIXED, TileBlock<N, MIXED>::alt, ST, TL>(p, stream, per_sm);
  return launch_tile_bt<N, KT, MIXED, TileBlock<N, MIXED>::threads, ST, TL>(p, stream, per_sm);
}

template <int N, bool MIXED, int ST, bool TL>
cudaError_t launch_tile_n(const TileParams &p, cudaStream_t stream, int *per_sm) {
  if constexpr (TL && !tile_tl_kernels(N, ST == kTileRkf45)) return cudaErrorInvalidValue;
  else switch (p.c.K1) {
    case 1: return launch_tile_nk<N, 1, MIXED, ST, TL>(p, stream, per_sm);
    case 2: return launch_tile_nk<N, 2, MIXED, ST, TL>(p, stream, per_sm);
    case 3: return launch_tile_nk<N, 3, MIXED, ST, TL>(p, stream, per_sm);
    default: return cudaErrorInvalidValue;
  }
}

template <bool MIXED, int ST, bool TL>
cudaError_t launch_tile_dispatch(const TileParams &p, cudaStream_t stream, int *per_sm = nullptr) {
  switch (p.c.N) {
    case 2: return launch_tile_n<2, MIXED, ST, TL>(p, stream, per_sm);
    case 3: return launch_tile_n<3, MIXED, ST, TL>(p, stream, per_sm);
    case 4: return launch_tile_n<4, MIXED, ST, TL>(p, stream, per_sm);
    case 5: return launch_tile_n<5, MIXED, ST, TL>(p, stream, per_sm);
    case 6: return launch_tile_n<6, MIXED, ST, TL>(p, stream, per_sm);
    case 7: return launch_tile_n<7, MIXED, ST, TL>(p, stream, per_sm);
    case 8: return launch_tile_n<8, MIXED, ST, TL>(p, stream, per_sm);
    case 10: return launch_tile_n<10, MIXED, ST, TL>(p, stream, per_sm);
    case 12: return launch_tile_n<12, MIXED, ST, TL>(p, stream, per_sm);
    case 16: return launch_tile_n<16, MIXED, ST, TL>(p, stream, per_sm);
    case 24: return launch_tile_n<24, MIXED, ST, TL>(p, stream, per_sm);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace
}  // namespace phi
