// The GEMM of gemm.cu on tiles of a pair of CTAs (tcgen05 cta_group::2), persistent over the tiles: for products large enough to
// keep the tensor cores busy.
//
// The two CTAs of a pair work on one 256 x BN tile: each stages its 128 rows of A and BN / 2 rows of B, the even CTA's MMA thread
// issues for both, and each CTA's TMEM receives its own 128 rows.  An SM then takes (128 + BN / 2) instead of (128 + BN) rows of
// operands per 128 bytes of K, and a 256 x 256 tile is bound by the tensor cores (512 clocks per 128 bytes of K) and no longer by
// the way into shared memory.  Two TMEM accumulators: the epilogue warps read one while the next tile fills the other, so of all
// epilogues only the last is seen.  8192^3 e4m3: 550 us in one-CTA tiles of one wave after the other, 413 - 424 us here (2.6 PFLOP/s,
// at the power limit).  Small products stay with gemm.cu: a pair's barriers cost 1 us more per launch.
//
// K slices (tiles of 128 columns, for products with few tiles and a long K) are summed inside the cluster as in gemm.cu.
#include <atomic>

#include "gemm_common.cuh"

namespace qb {

constexpr int kMaxStages = 9;

// The shared memory is laid out as scratch area, barriers, column vectors, stages; the scratch area takes the partial sums that
// other CTAs of the cluster push (a tile of f32), and what it leaves goes to the stages.
template <int BN>
struct PairSmem {
  static constexpr int kBRows = BN / 2;  // rows of B staged by one CTA
  static constexpr int kStageBytes = (kBM + kBRows) * kRowBytes;
  static constexpr int kBarBytes = 256;
  static constexpr int kColBytes = 3 * BN * 4;  // per-column scale, bias, gate of this tile as f32
  __host__ __device__ static constexpr int before_stages(int scratch) { return (scratch + kBarBytes + kColBytes + 1023) / 1024 * 1024; }
  static constexpr int stages(int scratch) {
    const int n = (227 * 1024 - 1024 - before_stages(scratch)) / kStageBytes;
    return n < kMaxStages ? n : kMaxStages;
  }
  static constexpr int scratch(bool slices) { return slices ? kBM * BN * 4 : 0; }
  static_assert((2 * kMaxStages + 4) * 8 + 16 <= kBarBytes && stages(0) >= 4, "shared memory of one CTA");
};

// Tile `t` of the walk: groups of `group_m` row tiles, row index fastest inside a group, so that the CTAs that run at the same
// time share both row tiles of A and column tiles of B in L2.
__device__ __forceinline__ void tile_at(const GemmArgs& g, int t, int& mt, int& nt) {
  if (g.tiles_m <= g.group_m) {
    nt = t / g.tiles_m;
    mt = t - nt * g.tiles_m;
    return;
  }
  const int tiles_n = g.n_tiles / g.tiles_m;
  const int per_group = g.group_m * tiles_n;
  const int first = t / per_group * g.group_m;
  const int gm = min(g.tiles_m - first, g.group_m);
  const int i = t % per_group;
  mt = first + i % gm;
  nt = i / gm;
}

template <int BN, bool FP8, bool kSlices>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g) {
  using L = PairSmem<BN>;
  constexpr int kKElems = FP8 ? 128 : 64;  // elements of K per stage
  constexpr uint32_t kTmemCols = 2 * BN;   // two accumulators: one is filled while the other is read
  constexpr uint32_t kIdesc = FP8 ? umma_idesc(0, 0, 2 * kBM, BN) : umma_idesc(1, 1, 2 * kBM, BN);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* scratch = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int stages = g.stages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(scratch + g.scratch);
  float* col = reinterpret_cast<float*>(scratch + g.scratch + L::kBarBytes);
  uint8_t* smem = scratch + L::before_stages(g.scratch);  // the stages
  uint64_t* full_bar = bars;                    // [stage] A and B have landed (of both CTAs of a pair: the even CTA's barrier)
  uint64_t* empty_bar = bars + kMaxStages;      // [stage] the MMAs that read the stage are done
  uint64_t* acc_full = bars + 2 * kMaxStages;   // [2] the accumulator is complete
  uint64_t* acc_empty = acc_full + 2;           // [2] the epilogue warps (of both CTAs of a pair) have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* lost_flag = abort_flag + 1;  // set by a CTA of the cluster whose slice is missing

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x & 1);  // of this CTA in its pair (the cluster is 2 wide in x)
  const int split = blockIdx.z;
  const int rank0 = 2 * split;  // rank in the cluster of this slice's even CTA (the slices of a tile are the cluster's z)
  const int first_tile = blockIdx.x / 2, tile_step = gridDim.x / 2;
  const int kb0 = split * g.kb_per_split;
  const int n_iter = min(kb0 + g.kb_per_split, g.kb_total) - kb0;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), 16);
    }
    *abort_flag = 0;
    *lost_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync();  // the other CTAs signal barriers and push partial sums into this one's memory
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();  // set-up is done: the next kernel in the stream may begin its own

  // first row of A, first column of C and first row of B of tile t
  auto locate = [&](int t, int& m0, int& n0, int& b_row0) {
    int mt, nt;
    tile_at(g, t, mt, nt);
    m0 = (2 * mt + rank) * kBM;
    n0 = nt * BN;
    b_row0 = n0 + rank * L::kBRows;
  };

  if (warp == 0) {
    // ---------------- TMA producer
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      bool alive = true, waited = false;
      const uint32_t full0 = map_to_cta(smem_u32(full_bar), rank0);
      const uint32_t stage0 = smem_u32(smem);
      auto expect = [&](int st) {
        if (rank == 0) mbar_arrive_expect_tx(smem_u32(&full_bar[st]), 2 * L::kStageBytes);
      };
      auto load_a = [&](int st, int it, int row) {
        tma_load_2d_pair(stage0 + st * L::kStageBytes, &tmA, full0 + st * 8, (kb0 + it) * kKElems, row);
      };
      auto load_b = [&](int st, int it, int row) {
        tma_load_2d_pair(stage0 + st * L::kStageBytes + kBM * kRowBytes, &tmB, full0 + st * 8, (kb0 + it) * kKElems, row);
      };
      for (int t = first_tile; t < g.n_tiles && alive; t += tile_step) {
        int m0, n0, b_row0;
        locate(t, m0, n0, b_row0);
        int it = 0;
        if (!waited) {
          // The weight tiles of the first stages do not depend on the kernels before this one, so they are
          // already on their way while those kernels finish; A follows once they have.
          const int ahead = g.b_const ? min(stages, n_iter) : 0;
          for (int i = 0; i < ahead; ++i) {
            expect(i);
            load_b(i, i, b_row0);
          }
          grid_dep_wait();
          for (int i = 0; i < ahead; ++i) load_a(i, i, m0);
          waited = true;
          it = ahead;
          s = ahead == stages ? 0 : ahead;
          ph = ahead == stages ? 1 : 0;
        }
        for (; it < n_iter; ++it) {
          alive = mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM);
          if (!alive) break;
          expect(s);
          load_a(s, it, m0);
          load_b(s, it, b_row0);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
      if (alive && *abort_flag == 0) {
        // Tail: the last stage releases arrive on barriers in this CTA's shared memory; see them land before it can exit
        // (a stage that was never used passes at once).
        for (int i = 0; i < stages; ++i) {
          if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) break;
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      } else {
        // Giving up: leave the copies already in flight time to land before this CTA's memory goes away.
        const long long t0 = clock64();
        while (clock64() - t0 < (1ll << 22)) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the even CTA's, for both
    if (rank == 0 && elect_one()) {
      const uint16_t pair_mask = static_cast<uint16_t>(3u << rank0);
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        return mbar_wait_cluster(smem_u32(bar), parity, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM);
      };
      auto commit = [&](uint64_t* bar) {
        umma_commit_pair(smem_u32(bar), pair_mask);
      };
      const uint64_t desc0 = umma_desc_k_sw128(smem_u32(smem));
      int s = 0, done = 0;  // tiles finished: accumulator done & 1
      uint32_t ph = 0;
      bool ok = true;
      for (int t = first_tile; t < g.n_tiles && ok; t += tile_step) {
        int m0, n0, b_row0;
        locate(t, m0, n0, b_row0);
        const int acc = done & 1;
        if (done >= 2) ok = wait(&acc_empty[acc], ((done >> 1) - 1) & 1);
        tc_fence_after();
        const uint32_t d = tmem_base + acc * BN;
        for (int it = 0; it < n_iter && ok; ++it) {
          ok = wait(&full_bar[s], ph);
          if (!ok) break;
          tc_fence_after();
          const uint64_t a_desc = desc0 + static_cast<uint64_t>(s * (L::kStageBytes >> 4));
          const uint64_t b_desc = a_desc + (kBM * kRowBytes >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // 4 x 32 bytes of K per stage row
            const uint32_t accumulate = (it > 0 || k > 0) ? 1u : 0u;
            if (FP8) umma_f8_pair(d, a_desc + 2 * k, b_desc + 2 * k, kIdesc, accumulate);
            else umma_f16_pair(d, a_desc + 2 * k, b_desc + 2 * k, kIdesc, accumulate);
          }
          commit(&empty_bar[s]);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (ok && late(blockIdx.x / 2 == gridDim.x / 2 - 1 && blockIdx.z == gridDim.z - 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) ok = false;
        if (ok) commit(&acc_full[acc]);  // else both CTAs' epilogues give up as well
        ++done;
      }
    }
  } else {
    // ---------------- epilogue: warp w may touch TMEM lanes 32 * (w % 4) .. + 31.  Two warps share each lane quarter (w and
    // w + 4 see the same 32 rows) and split the row's columns.
    const int lane_grp = warp & 3, half = (warp - 2) >> 2;
    const int row = lane_grp * 32 + lane;
    const int et = threadIdx.x - 64;  // 0 .. 255
    const uint32_t lane_addr = static_cast<uint32_t>(lane_grp * 32) << 16;
    grid_dep_wait();  // bias / gate / residual are read and C is written only after the earlier kernels are done
    const uint32_t empty0 = map_to_cta(smem_u32(acc_empty), rank0);
    int acc = 0;
    uint32_t aph = 0;
    bool first = true, ok = true;
    for (int t = first_tile; t < g.n_tiles; t += tile_step) {  // after a wait that ran out the barriers are still met
      int m0, n0, b_row0;
      locate(t, m0, n0, b_row0);
      const int m = m0 + row;
      const int m_last = min(m0 + kBM, g.M) - 1;
      const bool one_gate = g.gate == nullptr || m0 >= g.M || m0 / g.rows_per_gate == m_last / g.rows_per_gate;
      const int slice_rows = kBM / (kSlices ? g.splits : 1), slice_row0 = split * slice_rows;  // rows this CTA finishes
      uint4 pre[kSlices ? BN / 32 : 1][2];  // slices: [..][0] the residuals of the 8-column groups that this thread will finish
      if (!first) asm volatile("bar.sync 2, 256;" ::: "memory");  // the last tile's readers of `col` and the scratch area are done
      first = false;
      // while the main loop runs: per-column vectors of this tile and its residual to shared memory (or, by the thread that will
      // use them, to registers), so that no global load sits between the accumulator and the stores
      const float sa = g.a_scale ? *g.a_scale : 1.0f;
      const size_t grow = g.gate && m0 < g.M ? static_cast<size_t>(m0 / g.rows_per_gate) * g.N : 0;
      for (int j = et; j < BN; j += 256) {
        const int n = n0 + j;
        const bool in = n < g.N;
        col[j] = (in && g.w_scale) ? sa * __ldg(g.w_scale + n) : sa;
        col[BN + j] = (in && g.bias) ? bf16_bits_to_f32(g.bias[n]) : 0.f;
        col[2 * BN + j] = (in && g.gate) ? bf16_bits_to_f32(g.gate[grow + n]) : 0.f;
      }
      if constexpr (kSlices) {
        constexpr int kVecs = BN / 8;  // 16-byte vectors of a row
        if (g.gate != nullptr) {
#pragma unroll
          for (int k = 0; k < BN / 32; ++k) {
            const int r = et / kVecs + 256 / kVecs * k, mm = m0 + slice_row0 + r, n = n0 + et % kVecs * 8;
            pre[k][0] = make_uint4(0u, 0u, 0u, 0u);
            if (r < slice_rows && mm < g.M && n < g.N) pre[k][0] = *reinterpret_cast<const uint4*>(g.residual + static_cast<size_t>(mm) * g.N + n);
          }
        }
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
      const uint32_t taddr = tmem_base + acc * BN + lane_addr;
      auto wait_acc = [&]() {
        ok = __all_sync(0xffffffffu, ok && mbar_wait(smem_u32(&acc_full[acc]), aph, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM));
        if (kSlices) ok = all_of_epilogue(ok);  // the paths below meet at barriers: the 256 threads take the same one
        tc_fence_after();
      };
      if constexpr (!kSlices) {
        // Half an accumulator row per thread, 16 columns at a time.  The loop's first turn for the first tile comes before the
        // accumulator is complete, on zeros and without a store: the instructions are in the SM's cache when they are wanted.
        uint8_t* c_row = m < g.M ? row_of_c(g, m) : nullptr;
        const bool wide = g.N % 32 == 0 && (reinterpret_cast<uintptr_t>(g.C) & 31u) == 0;
        const uint4* res_row = reinterpret_cast<const uint4*>(g.residual + static_cast<size_t>(m) * g.N + n0);
        const int c0 = half * (BN / 2);
        uint4 next[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};  // residual of the next turn
        auto fetch = [&](int c) {
          if (g.gate != nullptr && c < c0 + BN / 2 && m < g.M && n0 + c < g.N) {
            next[0] = res_row[c / 8];
            if (n0 + c + 8 < g.N) next[1] = res_row[c / 8 + 1];
          }
        };
        fetch(c0);
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = 0u;
#pragma unroll 1
        for (int c = t == first_tile ? c0 - 16 : c0; c < c0 + BN / 2; c += 16) {
          const bool live = c >= c0;
          uint4 res[2] = {next[0], next[1]};
          if (live) {
            if (c == c0) {
              wait_acc();
              if (!ok) break;
            }
            if (n0 + c >= g.N) break;
            tmem_ld16(taddr + c, r);
            fetch(c + 16);
            tmem_wait_ld_into(r);
          }
          const int cc = live ? c : c0;
          if (m < g.M && n0 + cc < g.N) epilogue16<BN>(g, r, m, n0 + cc, col + cc, res, one_gate, c_row, wide, live);
        }
      } else {
        wait_acc();
        if (ok) push_slices<2, BN>(scratch, taddr, split, rank, row, half, g.splits);
        else if (threadIdx.x == 64) tell_lost<2>(lost_flag, rank, g.splits);
        cluster_sync();  // every slice's share of this CTA's rows has arrived after this barrier (warps 0 and 1 join it below)
        if (ok && *lost_flag == 0) finish_slices<BN>(g, reinterpret_cast<const float4*>(scratch), col, m0, n0, slice_row0, slice_rows, one_gate, pre);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive_cluster(empty0 + acc * 8);
      }
      if (++acc == 2) { acc = 0; aph ^= 1; }
    }
  }

  tc_fence_before();
  __syncwarp();
  if (kSlices && warp < 2) cluster_sync();  // the barrier after which the epilogue warps read what was pushed to them
  cluster_sync();  // nobody leaves while another CTA may still signal a barrier in this one's memory, or use its TMEM or operands
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

template <int BN, bool FP8, bool kSlices>
static int32_t launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmArgs g, cudaStream_t st) {
  using L = PairSmem<BN>;
  g.scratch = L::scratch(kSlices);
  g.stages = L::stages(g.scratch);
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  int dev = 0;
  QB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 64 || (configured.load(std::memory_order_relaxed) >> dev & 1) == 0) {
    QB_CUDA_OK(cudaFuncSetAttribute(gemm_pair_kernel<BN, FP8, kSlices>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  const int pairs = num_sms() / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (kSlices || g.n_tiles < pairs ? g.n_tiles : pairs), 1, g.splits);  // slices: one tile per cluster
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = 1024 + L::before_stages(g.scratch) + g.stages * L::kStageBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(g.splits);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_dependent_launch ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_pair_kernel<BN, FP8, kSlices>, tmA, tmB, static_cast<const GemmArgs&>(g));
  ++g_launch_count;
  if (e != cudaSuccess) return fail(QB_ERR_LAUNCH, "gemm kernel (pairs, %d columns, %d slices): %s", BN, g.splits, cudaGetErrorString(e));
  return QB_OK;
}

template <bool FP8>
static int32_t launch_pair(int bn, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& g, cudaStream_t st) {
  if (g.splits > 1) return launch_pair<128, FP8, true>(tmA, tmB, g, st);
  return bn == 256 ? launch_pair<256, FP8, false>(tmA, tmB, g, st) : launch_pair<128, FP8, false>(tmA, tmB, g, st);
}

int32_t launch_gemm_pair(const GemmPlan& pl, const void* A, const void* B, const GemmArgs& args, bool fp8, cudaStream_t st) {
  GemmArgs g = args;
  g.tiles_m = (g.M + 2 * kBM - 1) / (2 * kBM);
  g.n_tiles = g.tiles_m * ((g.N + pl.bn - 1) / pl.bn);
  g.group_m = 8;  // 2048 rows: the operands of the tiles in flight stay in L2
  CUtensorMap tmA, tmB;
  const int es = fp8 ? 1 : 2;
  int32_t rc = make_tmap_2d_sw(&tmA, A, es, g.M, g.K, kBM, kRowBytes / es, 128);
  if (rc != QB_OK) return rc;
  rc = make_tmap_2d_sw(&tmB, B, es, g.N, g.K, pl.bn / 2, kRowBytes / es, 128);
  if (rc != QB_OK) return rc;
  return fp8 ? launch_pair<true>(pl.bn, tmA, tmB, g, st) : launch_pair<false>(pl.bn, tmA, tmB, g, st);
}

}  // namespace qb
