// heom_tile.cu -- tiled Liouvillian-apply / RK-stage kernel for one
// IndependentBath hierarchy: the choice of kernel and
// schedule (the kernel itself: heom_tile_pipe.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "heom_tile_body.cuh"

namespace phi {

using namespace tile_detail;

namespace {
cudaError_t launch_tile(const TileParams &p, bool mixed, cudaStream_t stream, int *per_sm = nullptr) {
  if (p.c.time_local && tile_tl_kernels(p.c.N, p.mode == kModeRkf45)) {
    if (p.mode == kModeRkf45)
      return mixed ? launch_tile_mixed_rkf45_tl(p, stream, per_sm) : launch_tile_fp64_rkf45_tl(p, stream, per_sm);
    return mixed ? launch_tile_mixed_rk4_tl(p, stream, per_sm) : launch_tile_fp64_rk4_tl(p, stream, per_sm);
  }
  if (p.mode == kModeRkf45)
    return mixed ? launch_tile_mixed_rkf45(p, stream, per_sm) : launch_tile_fp64_rkf45(p, stream, per_sm);
  return mixed ? launch_tile_mixed_rk4(p, stream, per_sm) : launch_tile_fp64_rk4(p, stream, per_sm);
}
}  // namespace

bool tile_kernel_available(const HeomConsts &c) {
  // IndependentBath with PHI's identity site map and K + 1 <= 3.
  if (c.kind != kIndependent || !c.identity_sites || c.K1 < 1 || c.K1 > 3 || c.nb != c.N) return false;
  // neighbour offsets are 32-bit element indices of the stage input
  if ((long long)c.M * (c.N * c.N + 1) >= (1ll << 31)) return false;
  switch (c.N) {
    case 2: case 3: case 4: case 5: case 6: case 7: case 8:
    case 10: case 12: case 16: case 24:
      return true;
    default:
      return false;
  }
}

int mixed_node_stride(int N) { return N * N + ((N * N) & 1); }

namespace tile_detail {
TileParams tile_params_for(const StageLaunch &L) {
  TileParams p;
  p.c = L.c;
  if (L.mode == kModeRkf45) {
    p.c.tile_variant = L.c.tile_variant_rkf;
    p.c.tile_cps = L.c.tile_cps_rkf;
  }
  p.mode = L.mode;
  p.stage = L.stage;
  p.x = L.xv;
  p.out = L.outv;
  p.y = L.y;
  p.acc = L.acc;
  p.y32 = L.y32;
  p.a_next = L.a_next;
  p.w_acc = L.w_acc;
  p.rk4 = L.rk4;
  p.traj = L.traj;
  for (int i = 0; i < 5; ++i) p.k[i] = L.kv[i];
  p.ybuf[0] = L.ybuf[0];
  p.ybuf[1] = L.ybuf[1];
  p.y32buf[0] = L.y32buf[0];
  p.y32buf[1] = L.y32buf[1];
  p.ctl = L.ctl;
  p.act[0] = L.act[0];
  p.act[1] = L.act[1];
  p.act_par = L.act_par;
  p.dot_w = (L.mode == kModeApply && !L.mixed) ? L.dot_w : nullptr;
  p.dot_part = p.dot_w ? L.dot_part : nullptr;
  p.dot_slots = p.dot_w ? L.dot_slots : 0;
  const bool mixed = L.mixed;
  const int xb = mixed ? 8 : 16;
  // Epilogue operands of this (mode, stage), in the order the epilogue reads them.
  p.dependent = 0;  // set by the launch
  p.npre = 0;
  for (int b = 0; b < kMaxPre; ++b) {
    p.pre[b] = nullptr;
    p.pre_bytes[b] = 16;
  }
  if (p.dot_w) {
    p.pre[0] = p.dot_w;
    p.npre = 1;
  }
  if (L.mode == kModeRk4) {
    if (L.stage == 0 && mixed) {
      p.pre[0] = L.y;
      p.npre = 1;
    } else if (L.stage == 1 || L.stage == 2) {
      // mixed: the complex64 copy y32 feeds the complex64 stage input
      p.pre[0] = mixed ? (const void *)L.y32 : (const void *)L.y;
      p.pre_bytes[0] = mixed ? 8 : 16;
      p.pre[1] = L.acc;
      p.npre = 2;
    } else if (L.stage == 3) {
      p.pre[0] = L.acc;
      p.npre = 1;
    }
  } else if (L.mode == kModeRkf45) {
    if (L.stage == 0) {
      p.npre = 0;              // y (or y32) is the stage input itself
    } else if (L.stage <= 4) {
      p.npre = 1 + L.stage;    // y, k_0 .. k_{s-1}
      for (int r = 0; r < L.stage; ++r) {
        p.pre[1 + r] = L.kv[r];
        p.pre_bytes[1 + r] = xb;
      }
    } else {
      p.npre = 5;              // y, k0, k2, k3, k4
      const int ks[4] = {0, 2, 3, 4};
      for (int r = 0; r < 4; ++r) {
        p.pre[1 + r] = L.kv[ks[r]];
        p.pre_bytes[1 + r] = xb;
      }
    }
    // Slot 0 (y, chosen on the device): complex64 y32 for the mixed stage
    // inputs of stages 1-4; read from global memory in mixed stage 5 and in
    // the 24-site FP64 stages 3-5 (see tile_epilogue).
    if (mixed && L.stage >= 1 && L.stage <= 4) p.pre_bytes[0] = 8;
    if ((mixed && L.stage == 5) || (!mixed && L.c.N == 24 && L.stage >= 3)) p.pre_bytes[0] = 0;
  }
  return p;
}
}  // namespace tile_detail

cudaError_t launch_tile_stage(const StageLaunch &L, cudaStream_t stream) {
  const TileParams p = tile_params_for(L);
  return launch_tile(p, L.mixed, stream);
}

namespace {
template <bool MIXED>
int block_threads_n(int N, int variant) {
  switch (N) {
#define PHI_TB(n) \
  case n: return variant == 1 ? TileBlock<n, MIXED>::alt : TileBlock<n, MIXED>::threads;
    PHI_TB(2) PHI_TB(3) PHI_TB(4) PHI_TB(5) PHI_TB(6) PHI_TB(7) PHI_TB(8) PHI_TB(10) PHI_TB(12) PHI_TB(16) PHI_TB(24)
#undef PHI_TB
    default: return 0;
  }
}
}  // namespace

int tile_block_threads(const HeomConsts &c, bool mixed, int variant) {
  return mixed ? block_threads_n<true>(c.N, variant) : block_threads_n<false>(c.N, variant);
}

cudaError_t tile_autotune(const StageLaunch &L0, cudaStream_t stream, TileSchedule *out) {
  StageLaunch L = L0;
  L.dot_w = nullptr;
  L.dot_part = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  TileSchedule best{};
  best.ms = 1e30f;
  float ms_default = 0.f;
  constexpr int kReps = 3;
  for (int variant = 0; variant < 2 && e == cudaSuccess; ++variant) {
    int per_sm = 0;
    TileParams p = tile_params_for(L);
    p.c.tile_variant = variant;
    p.c.tile_cps = 0;
    // warm-up launch (module load, smem attribute) and the occupancy
    e = launch_tile(p, L.mixed, stream, &per_sm);
    for (int cps = per_sm; cps >= 1 && e == cudaSuccess; --cps) {
      p.c.tile_cps = cps == per_sm ? 0 : cps;
      e = cudaEventRecord(e0, stream);
      for (int r = 0; r < kReps && e == cudaSuccess; ++r)
        e = launch_tile(p, L.mixed, stream);
      if (e == cudaSuccess) e = cudaEventRecord(e1, stream);
      if (e == cudaSuccess) e = cudaEventSynchronize(e1);
      float ms = 0.f;
      if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
      if (e != cudaSuccess) break;
      ms /= kReps;
      if (variant == 0 && cps == per_sm) ms_default = ms;
      if (ms < best.ms) {
        best.ms = ms;
        best.variant = variant;
        best.cps = p.c.tile_cps;
      }
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (e != cudaSuccess) return e;
  best.ms_default = ms_default;
  best.threads = tile_block_threads(L.c, L.mixed, best.variant);
  *out = best;
  return cudaSuccess;
}

namespace {
template <int N, int KT>
long long tiles_of_k(long long M, bool mixed) {
  const long long nt = mixed ? TileShape<N, true, KT, kTileThreads, kTileBatch>::NT
                             : TileShape<N, false, KT, kTileThreads, kTileBatch>::NT;
  return (M + nt - 1) / nt;
}
template <int N>
long long tiles_of(long long M, bool mixed, int K1) {
  switch (K1) {
    case 1: return tiles_of_k<N, 1>(M, mixed);
    case 2: return tiles_of_k<N, 2>(M, mixed);
    case 3: return tiles_of_k<N, 3>(M, mixed);
    default: return -1;
  }
}
template <int N>
size_t stage_smem_n(const TileParams &p, bool mixed) {
  switch (p.c.K1) {
    case 1: return mixed ? tile_smem<N, 1, true>(p.c.T, p.npre, p.pre_bytes) : tile_smem<N, 1, false>(p.c.T, p.npre, p.pre_bytes);
    case 2: return mixed ? tile_smem<N, 2, true>(p.c.T, p.npre, p.pre_bytes) : tile_smem<N, 2, false>(p.c.T, p.npre, p.pre_bytes);
    case 3: return mixed ? tile_smem<N, 3, true>(p.c.T, p.npre, p.pre_bytes) : tile_smem<N, 3, false>(p.c.T, p.npre, p.pre_bytes);
    default: return 0;
  }
}
}  // namespace

long long tile_count(const HeomConsts &c, bool mixed) {
  switch (c.N) {
    case 2: return tiles_of<2>(c.M, mixed, c.K1);
    case 3: return tiles_of<3>(c.M, mixed, c.K1);
    case 4: return tiles_of<4>(c.M, mixed, c.K1);
    case 5: return tiles_of<5>(c.M, mixed, c.K1);
    case 6: return tiles_of<6>(c.M, mixed, c.K1);
    case 7: return tiles_of<7>(c.M, mixed, c.K1);
    case 8: return tiles_of<8>(c.M, mixed, c.K1);
    case 10: return tiles_of<10>(c.M, mixed, c.K1);
    case 12: return tiles_of<12>(c.M, mixed, c.K1);
    case 16: return tiles_of<16>(c.M, mixed, c.K1);
    case 24: return tiles_of<24>(c.M, mixed, c.K1);
    default: return -1;
  }
}

size_t tile_stage_smem(const StageLaunch &L) {
  const TileParams p = tile_params_for(L);
  switch (L.c.N) {
    case 2: return stage_smem_n<2>(p, L.mixed);
    case 3: return stage_smem_n<3>(p, L.mixed);
    case 4: return stage_smem_n<4>(p, L.mixed);
    case 5: return stage_smem_n<5>(p, L.mixed);
    case 6: return stage_smem_n<6>(p, L.mixed);
    case 7: return stage_smem_n<7>(p, L.mixed);
    case 8: return stage_smem_n<8>(p, L.mixed);
    case 10: return stage_smem_n<10>(p, L.mixed);
    case 12: return stage_smem_n<12>(p, L.mixed);
    case 16: return stage_smem_n<16>(p, L.mixed);
    case 24: return stage_smem_n<24>(p, L.mixed);
    default: return 0;
  }
}

size_t tile_params_bytes() { return sizeof(TileParams); }

void tile_params_host(const StageLaunch &L, void *out) {
  const TileParams p = tile_params_for(L);
  std::memcpy(out, &p, sizeof(p));
}


}  // namespace phi
