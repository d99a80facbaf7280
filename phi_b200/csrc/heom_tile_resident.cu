// heom_tile_resident.cu -- the whole RK4 run of a small IndependentBath
// hierarchy in one thread-block cluster.
//
// A hierarchy of a few hundred nodes (a trimer at depth 3 has 84) is a few
// tiles: a launch per stage costs about 3 us whatever the tile does.
// Here a cluster of up to 16 CTAs keeps the hierarchy resident for the run:
// each CTA owns a tile, with its node records, coefficients and stage input in
// shared memory and the state and the RK4 accumulator in registers, and loops
// over the steps on the device.  A stage is the derivative of the tile
// (tile_derivative, so every bit equals the launch-per-stage path), the
// combine, and one cluster barrier; only the stage inputs pass through global
// memory (L2), where the linked ADOs of other tiles are gathered from.  What
// bounds a stage is that round trip, the exchange barrier and the cluster
// barrier: 84-node trimer 2.9 us per stage as launches, 1.5 us here.
#include <cuda_runtime.h>

#include <cstdint>

#include "heom_tile_body.cuh"

namespace phi {

using namespace tile_detail;

namespace {

constexpr int kMaxCluster = 16;

struct ResidentParams {
  HeomConsts c;
  double2 *y;      // state
  void *y32;       // MIXED: its complex64 copy
  void *xbuf[2];   // stage inputs
  double a[3], w[4];  // stage weights: X_{s+1} = y + a_s k_s, accumulator w_s
  long long steps;
  int nodes;       // nodes per CTA
  Rk4Ctl *rk4;
  double2 *traj;
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int N, int KT, bool MIXED, int ST>
struct ResidentLayout {
  using S = TileShape<N, MIXED, KT, kTileThreads, ST>;
  using In = TileIn<N, KT, MIXED, kTileThreads, ST>;
  static constexpr int T = N * KT, XB = MIXED ? 8 : 16, E2 = S::E + (S::E & 1);
  static constexpr size_t r16(size_t b) { return (b + 15) / 16 * 16; }
  static constexpr size_t kX = 0;  // two stage inputs
  static constexpr size_t kXBytes = r16((size_t)S::NT * S::ES * XB);
  static constexpr size_t kU = kX + 2 * kXBytes;
  static constexpr size_t kH = kU + r16((size_t)S::NT * S::EU * XB);
  static constexpr size_t kCf = kH + (size_t)E2 * XB;
  static constexpr size_t kMats = kCf + (size_t)S::NT * T * sizeof(typename In::C);
  static constexpr size_t kIds = kMats + r16((size_t)E2 * XB / 2);
  static constexpr size_t kDeph = kIds + r16((size_t)S::NT * T * sizeof(int2));
  static constexpr size_t kBytes = kDeph + (size_t)S::NT * sizeof(double);
};

template <int N, int KT, bool MIXED, int ST>
__global__ void __launch_bounds__(kTileThreads, 1) heom_tile_resident_kernel(const __grid_constant__ ResidentParams p) {
  using Lay = ResidentLayout<N, KT, MIXED, ST>;
  using S = typename Lay::S;
  using In = typename Lay::In;
  using TX = typename TileArith<MIXED>::TX;
  using R = typename TileArith<MIXED>::R;
  constexpr int E = S::E, ES = S::ES, RR = S::RR, T = Lay::T, BT = kTileThreads;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const HeomConsts &c = p.c;
  const int tid = threadIdx.x;
  TX *Xs[2] = {reinterpret_cast<TX *>(smem_raw + Lay::kX), reinterpret_cast<TX *>(smem_raw + Lay::kX + Lay::kXBytes)};
  TX *Us = reinterpret_cast<TX *>(smem_raw + Lay::kU);
  TX *Hs = reinterpret_cast<TX *>(smem_raw + Lay::kH);
  typename In::C *cfs = reinterpret_cast<typename In::C *>(smem_raw + Lay::kCf);
  R *mats = reinterpret_cast<R *>(smem_raw + Lay::kMats);
  int2 *ids = reinterpret_cast<int2 *>(smem_raw + Lay::kIds);
  double *deph = reinterpret_cast<double *>(smem_raw + Lay::kDeph);

  const long long n0 = (long long)blockIdx.x * p.nodes;
  const long long left = c.M - n0;
  const int nt = (int)(left < 0 ? 0 : (left < p.nodes ? left : p.nodes));  // CTAs past the hierarchy only keep step
  if (c.h_real) {
    R *Hr = reinterpret_cast<R *>(Hs);
    for (int i = tid; i < E; i += BT) Hr[i] = (R)__ldg(c.H + i).x;
  } else {
    for (int i = tid; i < E; i += BT) Hs[i] = from_d2<TX>(__ldg(c.H + i));
  }
  for (int i = tid; i < E; i += BT) mats[i] = (R)__ldg(c.mats_elem + i);
  const int W = c.L + 2;
  for (int q = tid; q < nt * T; q += BT) {
    const int t = q % T;
    const int nx = __ldg(c.next + n0 * T + q), pv = __ldg(c.prev + n0 * T + q), occ = __ldg(c.mi + n0 * T + q);
    ids[q] = make_int2(nx >= 0 ? nx * ES : -1, pv >= 0 ? pv * ES : -1);
    cfs[q] = tile_coef<typename In::C, R>((R)__ldg(c.sq_next + t * W + occ), (R)__ldg(c.sq_prev + t * W + occ),
                                          __ldg(c.corr + t));
  }
  for (int q = tid; q < nt; q += BT) deph[q] = __ldg(c.deph_node + n0 + q);
  const TileMap<N, KT, MIXED, BT, ST> m(c);
  double2 y[RR], acc[RR];
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    y[r] = acc[r] = make_double2(0.0, 0.0);
    if (m.on(r, nt)) {
      y[r] = p.y[n0 * E + m.eo(r)];
      Xs[0][m.xo[r]] = from_d2<TX>(y[r]);
    }
  }
  __syncthreads();

  Rk4Ctl *rc = p.rk4;
  long long step = rc->step, nout = rc->nout;
  const long long out_factor = rc->out_factor, capacity = rc->capacity;
  TX *ybuf = MIXED ? static_cast<TX *>(p.y32) : reinterpret_cast<TX *>(p.y);
  for (long long it = 0; it < p.steps; ++it) {
    const bool row = out_factor > 0 && step % out_factor == 0 && p.traj && nout < capacity;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      // Stage inputs: y, X_a, X_b, X_a; the tile's own in Xs[s & 1].
      const TX *xin = s == 0 ? ybuf : static_cast<const TX *>(p.xbuf[s == 2]);
      TX *out = (s == 3 ? ybuf : static_cast<TX *>(p.xbuf[s == 1])) + n0 * ES;
      const In in{Xs[s & 1], Us, Hs, mats, ids, cfs, nullptr, deph, nullptr, xin, nt, nullptr};
      TX dx[RR];
      tile_derivative<N, KT, MIXED, BT, ST>(c, m, in, dx);
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        if (!m.on(r, nt)) continue;
        const int x = m.xo[r];
        TX nx;
        if (s < 3) {
          if constexpr (MIXED) {
            const float af = (float)p.a[s];
            const TX ys = from_d2<TX>(y[r]);
            nx = mk<TX>(fmaf(dx[r].x, af, ys.x), fmaf(dx[r].y, af, ys.y));
          } else {
            nx = cfma(y[r], dx[r], p.a[s]);
          }
          acc[r] = cfma(s == 0 ? y[r] : acc[r], to_d2(dx[r]), p.w[s]);
        } else {
          y[r] = cfma(acc[r], to_d2(dx[r]), p.w[3]);
          nx = from_d2<TX>(y[r]);
          if (MIXED) p.y[n0 * E + m.eo(r)] = y[r];
          if (row && n0 == 0 && m.eo(r) < E) p.traj[nout * E + m.eo(r)] = y[r];
        }
        out[x] = nx;
        Xs[(s & 1) ^ 1][x] = nx;
      }
      // The next stage's inputs are complete, in this CTA and in L2, and the
      // exchange tile is free.
      cluster_barrier();
    }
    if (row) ++nout;
    ++step;
  }
  if (blockIdx.x == 0 && tid == 0) {
    rc->step = step;
    rc->nout = nout;
  }
}

template <int N, int KT, bool MIXED, int ST>
cudaError_t launch_shape(const ResidentParams &p0, cudaStream_t stream) {
  // The smallest power of two of CTAs that holds the hierarchy.
  int size = 1;
  while (size < kMaxCluster && (p0.c.M + size - 1) / size > ResidentLayout<N, KT, MIXED, ST>::S::NT) size *= 2;
  if ((p0.c.M + size - 1) / size > ResidentLayout<N, KT, MIXED, ST>::S::NT) return cudaErrorNotSupported;
  auto kern = heom_tile_resident_kernel<N, KT, MIXED, ST>;
  constexpr size_t smem = ResidentLayout<N, KT, MIXED, ST>::kBytes;
  static thread_local int raised[kSmemLimitDevices] = {};
  cudaError_t e = raise_smem_limit(kern, smem, raised);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  ResidentParams p = p0;
  p.nodes = (int)((p.c.M + size - 1) / size);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = size;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(kTileThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
  if (e != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return cudaErrorNotSupported;
  }
  return cudaLaunchKernelEx(&cfg, kern, p);
}

// One element per thread (the shortest stage) where 16 CTAs hold it so, several
// otherwise: 84-node trimer 1.5 us per stage with one, 1.7 with two.
template <int N, int KT, bool MIXED>
cudaError_t launch_nk(const ResidentParams &p, cudaStream_t stream) {
  const cudaError_t e = launch_shape<N, KT, MIXED, kTileResident>(p, stream);
  return e == cudaErrorNotSupported ? launch_shape<N, KT, MIXED, kTileResidentWide>(p, stream) : e;
}

template <bool MIXED, int N>
cudaError_t launch_n(const ResidentParams &p, cudaStream_t stream) {
  switch (p.c.K1) {
    case 1: return launch_nk<N, 1, MIXED>(p, stream);
    case 2: return launch_nk<N, 2, MIXED>(p, stream);
    case 3: return launch_nk<N, 3, MIXED>(p, stream);
    default: return cudaErrorNotSupported;
  }
}

template <bool MIXED>
cudaError_t launch_any(const ResidentParams &p, cudaStream_t stream) {
  switch (p.c.N) {
    case 2: return launch_n<MIXED, 2>(p, stream);
    case 3: return launch_n<MIXED, 3>(p, stream);
    case 4: return launch_n<MIXED, 4>(p, stream);
    case 5: return launch_n<MIXED, 5>(p, stream);
    case 6: return launch_n<MIXED, 6>(p, stream);
    case 7: return launch_n<MIXED, 7>(p, stream);
    case 8: return launch_n<MIXED, 8>(p, stream);
    case 10: return launch_n<MIXED, 10>(p, stream);
    case 12: return launch_n<MIXED, 12>(p, stream);
    case 16: return launch_n<MIXED, 16>(p, stream);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace

cudaError_t launch_tile_resident_rk4(const StageLaunch &L, double dt, long long steps, cudaStream_t stream) {
  const HeomConsts &c = L.c;
  // The run's features that change between stages, and the test of the tile
  // kernel's bounded waits, stay on the launch-per-stage path.
  if (!tile_kernel_available(c) || c.filtered || c.time_local || c.h_dynamic || c.first_wait_polls != 0 || steps <= 0)
    return cudaErrorNotSupported;
  ResidentParams p{};
  p.c = c;
  p.y = L.y;
  p.y32 = L.y32;
  p.xbuf[0] = const_cast<void *>(L.xv);
  p.xbuf[1] = L.outv;
  const double a[3] = {dt / 2, dt / 2, dt}, w[4] = {dt / 6, dt / 3, dt / 3, dt / 6};
  for (int s = 0; s < 3; ++s) p.a[s] = a[s];
  for (int s = 0; s < 4; ++s) p.w[s] = w[s];
  p.steps = steps;
  p.rk4 = L.rk4;
  p.traj = L.traj;
  return L.mixed ? launch_any<true>(p, stream) : launch_any<false>(p, stream);
}

}  // namespace phi
