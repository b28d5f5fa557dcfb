// The grouped GEMM of the expert MLP: rows sorted by expert in runs of whole 128-row tiles, every tile multiplied with the weights
// of its expert (tile_expert, see GemmArgs).
//
// One CTA takes up to two consecutive tiles of one expert, 256 rows x BN columns: each stage holds both tiles' rows of A beside the
// expert's weights, and the MMA warp issues for the two accumulators in turn.  The experts' weights are what this product reads
// (67 MB at 720p, 8 experts), so they cross into shared memory once per expert instead of once per tile, and a run that spills over
// 128 rows by a few tokens costs no CTA of its own: with a CTA per tile 512 tokens of 8 experts (top 2) made 192 CTAs of 256
// columns, two rounds over the 148 SMs.  Roles as in gemm.cu: warp 0 TMA, warp 1 MMA, warps 2-9 epilogue.
#include <atomic>

#include "gemm_common.cuh"

namespace qb {

template <int BN>
struct GroupedSmem {
  static constexpr int kABytes = kBM * kRowBytes;
  static constexpr int kStageBytes = 2 * kABytes + BN * kRowBytes;
  static constexpr int kFit = 200 * 1024 / kStageBytes;
  static constexpr int kStages = kFit > 5 ? 5 : kFit;
  static constexpr int kBarOffset = kStages * kStageBytes;
  static constexpr int kColOffset = kBarOffset + 128;
  static constexpr int kTotal = kColOffset + 3 * BN * 4 + 1024;
  static_assert(kStages >= 3 && (2 * kStages + 1) * 8 + 16 <= 128 && kTotal <= 227 * 1024, "shared memory of one CTA");
};

template <int BN, bool FP8>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_grouped_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g) {
  using L = GroupedSmem<BN>;
  constexpr int kStages = L::kStages;
  constexpr int kKElems = FP8 ? 128 : 64;
  constexpr uint32_t kTmemCols = 2 * BN;
  constexpr uint32_t kIdesc = FP8 ? umma_idesc(0, 0, kBM, BN) : umma_idesc(1, 1, kBM, BN);

  grid_dep_wait();  // the table is written by the routing kernel just before
  grid_dep_launch();
  const int* table = after_wait(g.tile_expert);
  const int tile = blockIdx.y, expert = table[tile];
  if (expert < 0) return;  // a padding tile
  int run = 0;  // tiles of this expert before this one
  while (run < tile && table[tile - 1 - run] == expert) ++run;
  if (run & 1) return;  // the CTA of the tile before takes this one too
  const int tiles = tile + 1 < static_cast<int>(gridDim.y) && table[tile + 1] == expert ? 2 : 1;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* acc_bar = empty_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* drain_flag = abort_flag + 1;  // never set: lets the drain waits below run their own limit
  float* col = reinterpret_cast<float*>(smem + L::kColOffset);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = tile * kBM, n0 = blockIdx.x * BN, b_row0 = expert * g.N + n0;
  const int n_iter = g.kb_total;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(acc_bar), 1);
    *abort_flag = 0;
    *drain_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      const uint32_t stage_tx = tiles * L::kABytes + BN * kRowBytes;
      int s = 0, issued = 0;
      uint32_t ph = 0;
      for (int it = 0; it < n_iter; ++it) {
        if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) break;
        const uint32_t fb = smem_u32(&full_bar[s]);
        const uint32_t st = smem_u32(smem + s * L::kStageBytes);
        mbar_arrive_expect_tx(fb, stage_tx);
        tma_load_2d(st + 2 * L::kABytes, &tmB, fb, it * kKElems, b_row0);
        tma_load_2d(st, &tmA, fb, it * kKElems, m0);
        if (tiles == 2) tma_load_2d(st + L::kABytes, &tmA, fb, it * kKElems, m0 + kBM);
        issued = it + 1;
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
      if (*abort_flag) {
        // Giving up: let the copies already in flight land before this CTA's memory goes away.
        for (int it = max(0, issued - kStages); it < issued; ++it)
          mbar_wait(smem_u32(&full_bar[it % kStages]), (it / kStages) & 1, drain_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM);
      } else {
        // Tail: see the last stage releases land before the CTA can exit.
        for (int it = max(0, n_iter - kStages); it < n_iter; ++it)
          if (!mbar_wait(smem_u32(&empty_bar[it % kStages]), (it / kStages) & 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) break;
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = 0; it < n_iter; ++it) {
        ok = mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM);
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = smem_u32(smem + s * L::kStageBytes);
        const uint64_t b_desc = umma_desc_k_sw128(st + 2 * L::kABytes);
        for (int r = 0; r < tiles; ++r) {
          const uint64_t a_desc = umma_desc_k_sw128(st + r * L::kABytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // 4 x 32 bytes of K per stage row
            const uint32_t accumulate = (it > 0 || k > 0) ? 1u : 0u;
            if (FP8) umma_f8(tmem_base + r * BN, a_desc + 2 * k, b_desc + 2 * k, kIdesc, accumulate);
            else umma_f16(tmem_base + r * BN, a_desc + 2 * k, b_desc + 2 * k, kIdesc, accumulate);
          }
        }
        umma_commit(smem_u32(&empty_bar[s]));
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
      if (ok && late(blockIdx.x == gridDim.x - 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) ok = false;
      if (ok) umma_commit(smem_u32(acc_bar));  // else the epilogue gives up as well
    }
  } else {
    // epilogue: two warps share each TMEM lane quarter and split the row's columns
    const int lane_grp = warp & 3, half = (warp - 2) >> 2, et = threadIdx.x - 64;
    const float sa = g.a_scale ? *after_wait(g.a_scale) : 1.0f;
    for (int j = et; j < BN; j += 256) col[j] = sa;
    asm volatile("bar.sync 2, 256;" ::: "memory");
    const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(acc_bar), 0, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM));
    tc_fence_after();
    const bool wide = g.N % 32 == 0 && (reinterpret_cast<uintptr_t>(g.C) & 31u) == 0;
    for (int r = 0; ok && r < tiles; ++r) {
      const int m = m0 + r * kBM + lane_grp * 32 + lane;
      const uint32_t taddr = tmem_base + r * BN + (static_cast<uint32_t>(lane_grp * 32) << 16);
      uint8_t* c_row = row_of_c(g, m);
#pragma unroll 1
      for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 16) {
        if (n0 + c >= g.N) break;
        uint32_t x[16];
        tmem_ld16(taddr + c, x);
        tmem_wait_ld_into(x);
        epilogue16<BN>(g, x, m, n0 + c, col + c, nullptr, true, c_row, wide, true);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int BN, bool FP8>
static int32_t launch_grouped(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& g, cudaStream_t st) {
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  int dev = 0;
  QB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 64 || (configured.load(std::memory_order_relaxed) >> dev & 1) == 0) {
    QB_CUDA_OK(cudaFuncSetAttribute(gemm_grouped_kernel<BN, FP8>, cudaFuncAttributeMaxDynamicSharedMemorySize, GroupedSmem<BN>::kTotal));
    if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  return launch_dep("gemm kernel (grouped)", gemm_grouped_kernel<BN, FP8>, dim3((g.N + BN - 1) / BN, g.M / kBM), dim3(kGemmThreads),
                    GroupedSmem<BN>::kTotal, st, tmA, tmB, g);
}

int32_t launch_gemm_grouped(int bn, const void* A, const void* B, int n_experts, const GemmArgs& g, bool fp8, cudaStream_t st) {
  CUtensorMap tmA, tmB;
  const int es = fp8 ? 1 : 2;
  int32_t rc = make_tmap_2d_sw(&tmA, A, es, g.M, g.K, kBM, kRowBytes / es, 128);
  if (rc != QB_OK) return rc;
  // (a box that runs past the expert's last row only feeds columns >= N, which nothing stores)
  rc = make_tmap_2d_sw(&tmB, B, es, static_cast<uint64_t>(g.N) * n_experts, g.K, bn, kRowBytes / es, 128);
  if (rc != QB_OK) return rc;
  if (fp8) return bn == 256 ? launch_grouped<256, true>(tmA, tmB, g, st) : bn == 128 ? launch_grouped<128, true>(tmA, tmB, g, st) : launch_grouped<64, true>(tmA, tmB, g, st);
  return bn == 256 ? launch_grouped<256, false>(tmA, tmB, g, st) : bn == 128 ? launch_grouped<128, false>(tmA, tmB, g, st) : launch_grouped<64, false>(tmA, tmB, g, st);
}

}  // namespace qb
