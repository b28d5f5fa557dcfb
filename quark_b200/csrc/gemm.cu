// C[M,N] = epilogue(A[M,K] . B[N,K]^T) on the sm_100a tensor cores: tiles of one CTA (gemm_pair.cu has the tiles of a pair of
// CTAs that large products use), and the host side of both.
//
// One CTA computes one 128 x BN output tile over one K slice.  Warp 0 feeds a ring of
// shared-memory stages with TMA (128-byte swizzle), one thread of warp 1 issues
// tcgen05.mma into a TMEM accumulator, warps 2-9 read the accumulator back (one row per thread, two
// warps per TMEM lane quarter sharing each row's columns) and run the epilogue: 320 threads per CTA.  bf16 operands use
// kind::f16 (K = 16 per instruction), e4m3 operands kind::f8f6f4 (K = 32); both move 128 bytes of K per stage row, so the two
// paths share every address computation.
//
// K can be split over `splits` CTAs per tile.  As the CTAs of one thread-block cluster (64-column tiles) they push the rows that other CTAs will
// finish into those CTAs' shared memory; after one cluster barrier each CTA sums its 128 / splits rows in slice order and runs
// the epilogue on them.  Through the workspace (any number of slices) each CTA writes its partial tile and takes a ticket, and
// the CTA that draws the last ticket adds the partials in slice order.  Either way the sum does not depend on which CTA came
// last, and no CTA waits for another outside its cluster.
#include <atomic>

#include "gemm_common.cuh"

namespace qb {

constexpr int kSmemBudget = 200 * 1024;

#ifdef QB_GEMM_TRACE
__device__ long long g_gemm_trace[148 * 4][8];  // [CTA][point]: globaltimer ns
__device__ __forceinline__ long long gtime() { long long t; asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); return t; }
#define QB_GT(pt) do { const int cta_ = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x; if (cta_ < 148 * 4) g_gemm_trace[cta_][pt] = gtime(); } while (0)
#else
#define QB_GT(pt) do { } while (0)
#endif

template <int BN>
struct GemmSmem {
  static constexpr int kStageBytes = kBM * kRowBytes + BN * kRowBytes;
  static constexpr int kStages = (kSmemBudget / kStageBytes) > 8 ? 8 : (kSmemBudget / kStageBytes);
  // partial sums that the other K slices of the cluster push, and this CTA's own: 128 / splits rows of f32 from each.  They need
  // memory of their own, since a slower CTA's stages are in use while its peers push: 64-column tiles only.
  static constexpr int kSliceBytes = BN == 64 ? kBM * BN * 4 : 0;
  static constexpr int kSliceOffset = kStages * kStageBytes;
  static constexpr int kBarOffset = kSliceOffset + kSliceBytes;
  static constexpr int kColOffset = kBarOffset + 256;            // per-column scale, bias, gate of this tile as f32
  static constexpr int kTotal = kColOffset + 3 * BN * 4 + 1024;  // + alignment slack
  static_assert(kTotal <= 227 * 1024, "shared memory of one CTA");
};

template <int BN, bool FP8, bool QKV>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g) {
  using L = GemmSmem<BN>;
  constexpr int kStages = L::kStages;
  constexpr int kKElems = FP8 ? 128 : 64;  // elements of K per stage
  constexpr uint32_t kTmemCols = BN < 32 ? 32 : BN;
  constexpr uint32_t kIdesc = FP8 ? umma_idesc(0, 0, kBM, BN) : umma_idesc(1, 1, kBM, BN);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  uint64_t* acc_bar = bars + 2 * kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* last_flag = abort_flag + 1;
  volatile int* drain_flag = abort_flag + 2;  // never set: lets the drain waits below run their own limit
  volatile int* lost_flag = abort_flag + 3;   // set by a CTA of the cluster whose slice is missing

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) QB_GT(0);
  const int n0 = blockIdx.x * BN;
  const int m0 = blockIdx.y * kBM;
  const int split = blockIdx.z;
  const int kb0 = split * g.kb_per_split;
  const int kb1 = min(kb0 + g.kb_per_split, g.kb_total);
  const int n_iter = kb1 - kb0;
  const uint32_t stage_tx = g.a_rows * kRowBytes + BN * kRowBytes;
  const bool clustered = L::kSliceBytes > 0 && g.cluster != 0;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(acc_bar), 1);
    *abort_flag = 0;
    *last_flag = 0;
    *drain_flag = 0;
    *lost_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  if (clustered) cluster_sync();  // every CTA of the cluster is there before anyone pushes to it
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();  // set-up is done: the next kernel in the stream may begin its own
  if (threadIdx.x == 0) QB_GT(1);

  if (warp == 0) {
    // ---------------- TMA producer
    if (elect_one()) {
      // The weight tiles of the first stages do not depend on the kernels before this one, so they are
      // already on their way while those kernels finish; A follows once they have.
      const int ahead = g.b_const ? min(kStages, n_iter) : 0;
      for (int it = 0; it < ahead; ++it) {
        const uint32_t fb = smem_u32(&full_bar[it]);
        mbar_arrive_expect_tx(fb, stage_tx);
        tma_load_2d(smem_u32(smem + it * L::kStageBytes + kBM * kRowBytes), &tmB, fb, (kb0 + it) * kKElems, n0);
      }
      grid_dep_wait();
      QB_GT(2);
      for (int it = 0; it < ahead; ++it)
        tma_load_2d(smem_u32(smem + it * L::kStageBytes), &tmA, smem_u32(&full_bar[it]), (kb0 + it) * kKElems, m0);
      int issued = ahead;
      for (int it = ahead; it < n_iter; ++it) {
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1;
        if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) break;
        const uint32_t fb = smem_u32(&full_bar[s]);
        mbar_arrive_expect_tx(fb, stage_tx);
        uint8_t* a_s = smem + s * L::kStageBytes;
        tma_load_2d(smem_u32(a_s), &tmA, fb, (kb0 + it) * kKElems, m0);
        tma_load_2d(smem_u32(a_s + kBM * kRowBytes), &tmB, fb, (kb0 + it) * kKElems, n0);
        issued = it + 1;
      }
      if (*abort_flag) {
        // Giving up: let the copies already in flight land before this CTA's memory goes away.
        for (int it = max(0, issued - kStages); it < issued; ++it)
          mbar_wait(smem_u32(&full_bar[it % kStages]), (it / kStages) & 1, drain_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM);
      } else {
        // Tail: the MMA warp's last stage releases arrive on barriers in this CTA's shared memory;
        // see them land before the CTA can exit.
        for (int it = max(0, n_iter - kStages); it < n_iter; ++it)
          if (!mbar_wait(smem_u32(&empty_bar[it % kStages]), (it / kStages) & 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) break;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer
    if (elect_one()) {
      bool ok = true;
      for (int it = 0; it < n_iter && ok; ++it) {
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1;
        ok = mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM);
        if (!ok) break;
        if (it == 0) QB_GT(3);
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + s * L::kStageBytes);
        const uint64_t a_desc = umma_desc_k_sw128(a_addr);
        const uint64_t b_desc = umma_desc_k_sw128(a_addr + kBM * kRowBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // 4 x 32 bytes of K per stage row
          const uint32_t acc = (it > 0 || k > 0) ? 1u : 0u;
          if (FP8)
            umma_f8(tmem_base, a_desc + 2 * k, b_desc + 2 * k, kIdesc, acc);
          else
            umma_f16(tmem_base, a_desc + 2 * k, b_desc + 2 * k, kIdesc, acc);
        }
        umma_commit(smem_u32(&empty_bar[s]));
      }
      if (ok && late(blockIdx.x == gridDim.x - 1 && blockIdx.z == gridDim.z - 1, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM)) ok = false;
      if (ok) umma_commit(smem_u32(acc_bar));  // else the epilogue gives up as well
      QB_GT(4);
    }
  } else {
    // ---------------- epilogue, part 1: warp w may touch TMEM lanes 32 * (w % 4) .. + 31
    const int lane_grp = warp & 3;
    const int row = lane_grp * 32 + lane;
    const int m = m0 + row;
    grid_dep_wait();  // bias / gate / residual are read and C is written only after the earlier kernels are done
    // The fast epilogue needs whole 32-column chunks inside N, 32-byte aligned rows of C, and one gate row
    // for the whole tile; anything else takes the general path below.
    const int m_last = min(m0 + kBM, g.M) - 1;
    const bool fast = !QKV && g.splits == 1 && g.N % 32 == 0 && (reinterpret_cast<uintptr_t>(g.C) & 31u) == 0 &&
                      (g.gate == nullptr || m0 / g.rows_per_gate == m_last / g.rows_per_gate);
    // Two warps share each TMEM lane quarter (w and w + 4 see the same 32 rows): in the fast epilogue the
    // first takes the even 32-column chunks of the row, the second the odd ones.  All eight warps run the other
    // paths too, but for K slices through the workspace, which the first four sum alone.
    const int half = (warp - 2) >> 2;
    constexpr int kMyChunks = BN / 64;  // 32-column chunks per warp
    constexpr int kResInRegs = BN <= 128 ? 1 : 0;
    uint32_t res[kResInRegs ? kMyChunks * 16 : 1];
    const int slice_rows = kBM / (clustered ? g.splits : 1), slice_row0 = clustered ? split * slice_rows : 0;  // rows this CTA finishes
    const bool one_gate = g.gate == nullptr || m0 / g.rows_per_gate == m_last / g.rows_per_gate;
    uint4 pre[QKV || BN == 64 ? 2 : 1][2];  // QKV: see qkv_fetch; slices: the residuals of the 8-column groups this thread finishes
    QkvFrame fr{};  // QKV
    if (QKV || (clustered && one_gate)) {
      float* col = reinterpret_cast<float*>(smem + L::kColOffset);
      const int et = threadIdx.x - 64;
      const float sa = g.a_scale ? *g.a_scale : 1.0f;
      const size_t grow = g.gate ? static_cast<size_t>(m0 / g.rows_per_gate) * g.N : 0;
      for (int j = et; j < BN; j += 256) {
        const int n = n0 + j;
        const bool in = n < g.N;
        col[j] = (in && g.w_scale) ? sa * __ldg(g.w_scale + n) : sa;
        if (!QKV) {
          col[BN + j] = (in && g.bias) ? bf16_bits_to_f32(g.bias[n]) : 0.f;
          col[2 * BN + j] = (in && g.gate) ? bf16_bits_to_f32(g.gate[grow + n]) : 0.f;
        }
      }
      if constexpr (QKV) {
        fr = qkv_frame(g.qkv);
        qkv_share<BN>(g.qkv, fr, et, n0, reinterpret_cast<QkvShared*>(col + BN));
        if (blockIdx.x == 0 && blockIdx.y == 0 && split == 0 && et == 32) qkv_segments(g.qkv, fr);
        qkv_fetch<BN>(g, et, slice_row0, slice_rows, m0, n0, 0, pre[0]);
        qkv_fetch<BN>(g, et, slice_row0, slice_rows, m0, n0, 1, pre[1]);
      } else if constexpr (BN == 64) {
        if (g.gate != nullptr) {
#pragma unroll
          for (int k = 0; k < BN / 32; ++k) {
            const int r = et / (BN / 8) + 256 / (BN / 8) * k, mm = m0 + slice_row0 + r, n = n0 + et % (BN / 8) * 8;
            pre[k][0] = make_uint4(0u, 0u, 0u, 0u);
            if (r < slice_rows && mm < g.M && n < g.N) pre[k][0] = *reinterpret_cast<const uint4*>(g.residual + static_cast<size_t>(mm) * g.N + n);
          }
        }
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
    }
    if (!QKV && g.splits == 1) {
      // while the main loop runs: per-column vectors of this tile to shared memory, this row's residual to registers
      float* col = reinterpret_cast<float*>(smem + L::kColOffset);
      const int et = threadIdx.x - 64;  // 0 .. 255
      const float sa = g.a_scale ? *g.a_scale : 1.0f;
      const size_t grow = g.gate ? static_cast<size_t>(m0 / g.rows_per_gate) * g.N : 0;
      for (int j = et; j < BN; j += 256) {
        const int n = n0 + j;
        const bool in = n < g.N;
        col[j] = (in && g.w_scale) ? sa * __ldg(g.w_scale + n) : sa;
        col[BN + j] = (in && g.bias) ? bf16_bits_to_f32(g.bias[n]) : 0.f;
        col[2 * BN + j] = (in && g.gate) ? bf16_bits_to_f32(g.gate[grow + n]) : 0.f;
      }
      if (kResInRegs && fast && g.gate != nullptr && m < g.M) {
#pragma unroll
        for (int q = 0; q < kMyChunks * 4; ++q) {
          const int n = n0 + (2 * (q >> 2) + half) * 32 + (q & 3) * 8;  // chunk 2 * (q / 4) + half, 8 columns at a time
          uint4 x = make_uint4(0u, 0u, 0u, 0u);
          if (n < g.N) x = *reinterpret_cast<const uint4*>(g.residual + static_cast<size_t>(m) * g.N + n);
          res[(kResInRegs ? q : 0) * 4 + 0] = x.x;
          res[(kResInRegs ? q : 0) * 4 + 1] = x.y;
          res[(kResInRegs ? q : 0) * 4 + 2] = x.z;
          res[(kResInRegs ? q : 0) * 4 + 3] = x.w;
        }
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
    }
    bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(acc_bar), 0, abort_flag, g.status, QB_DEV_WAIT_TIMEOUT_GEMM));
    if (!fast) ok = all_of_epilogue(ok);  // the paths below meet at barriers: the 256 threads take the same one
    if (threadIdx.x == 64) QB_GT(5);
    tc_fence_after();
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(lane_grp * 32) << 16);
    if (ok && fast) {
      // One accumulator row per thread, 32 columns at a time.  Per-column vectors come from shared
      // memory and the residual row from registers, both fetched during the main loop, so no global
      // load sits between the accumulator and the stores; every store writes whole 32-byte sectors.
      const float* col = reinterpret_cast<const float*>(smem + L::kColOffset);
      const bool has_gate = g.gate != nullptr;
      const bool has_scale = g.a_scale != nullptr || g.w_scale != nullptr;
      const bool has_bias = g.bias != nullptr;
      // One or two chunks to a warp: unrolled, the next one on its way from TMEM while the current one is processed.  The four of a
      // 256-column tile: a loop, since its instructions, run once per launch, cost more to fetch than the loads from TMEM to wait for
      // (512 x 8192 x 2048 e4m3 SiLU 9.27 -> 8.79 us, 512 x 4096 x 512 5.77 -> 5.60 e4m3, 8.72 -> 8.62 bf16).  Two as a loop: SiLU 6.04 ->
      // 5.91 us (512 x 4096 x 2048, 128-column tiles), but with gate and residual, whose registers then move, 6.53 -> 6.60.
      constexpr bool kRolled = kMyChunks > 2;
      constexpr int kUnroll = kRolled ? 1 : kMyChunks;
      uint32_t rbuf[kRolled ? 1 : 2][32];
      if (!kRolled) tmem_ld32(taddr + half * 32, rbuf[0]);
#pragma unroll kUnroll
      for (int lc = 0; lc < kMyChunks; ++lc) {
        const int c = 2 * lc + half;
        uint32_t(&r)[32] = rbuf[kRolled ? 0 : lc & 1];
        if (kRolled) tmem_ld32(taddr + c * 32, r);
        tmem_wait_ld_into(r);
        if (!kRolled && lc + 1 < kMyChunks) tmem_ld32(taddr + (c + 2) * 32, rbuf[kRolled ? 0 : (lc + 1) & 1]);
        const int n = n0 + c * 32;
        if (m < g.M && n < g.N) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          if (has_scale) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= col[c * 32 + j];
          }
          if (has_bias) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] += col[BN + c * 32 + j];
          }
          if (g.activation == 1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = silu_fast(v[j]);
          }
          if (has_gate) {
            uint32_t rw[16];
            if (kResInRegs) {
#pragma unroll
              for (int j = 0; j < 16; ++j) rw[j] = res[kResInRegs ? lc * 16 + j : 0];
            } else {  // 256-column tiles: the row does not fit in registers beside the accumulator chunk
              const uint4* rp = reinterpret_cast<const uint4*>(g.residual + static_cast<size_t>(m) * g.N + n);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 x = rp[q];
                rw[4 * q] = x.x; rw[4 * q + 1] = x.y; rw[4 * q + 2] = x.z; rw[4 * q + 3] = x.w;
              }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              v[2 * j] = __fadd_rn(bf16lo(rw[j]), __fmul_rn(col[2 * BN + c * 32 + 2 * j], v[2 * j]));
              v[2 * j + 1] = __fadd_rn(bf16hi(rw[j]), __fmul_rn(col[2 * BN + c * 32 + 2 * j + 1], v[2 * j + 1]));
            }
          }
          const size_t off = static_cast<size_t>(m) * g.N + n;
          if (g.c_dtype == QB_BF16) {
            uint16_t* dst = static_cast<uint16_t*>(g.C) + off;
            if (g.tp_world != 0) {
              const int owner = m / g.tp_rpo;
              dst = g.tp_dst[owner] + static_cast<size_t>(m - owner * g.tp_rpo) * g.N + n;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t w[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) w[j] = pack_bf16x2(v[16 * h + 2 * j], v[16 * h + 2 * j + 1]);
              st_global_v8(dst + 16 * h, w);
            }
          } else if (g.c_dtype == QB_E4M3) {
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) w[j] = pack_e4m3x4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            st_global_v8(static_cast<uint8_t*>(g.C) + off, w);
          } else {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              uint32_t w[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) w[j] = __float_as_uint(v[8 * h + j]);
              st_global_v8(static_cast<float*>(g.C) + off + 8 * h, w);
            }
          }
        }
      }
    } else if (QKV) {
      if constexpr (QKV) {
        float* col = reinterpret_cast<float*>(smem + L::kColOffset);
        uint16_t* vt = reinterpret_cast<uint16_t*>(smem);  // over the stage memory (this CTA's MMAs are done)
        if (clustered) {
          if (ok) push_slices<1, BN>(smem + L::kSliceOffset, taddr, split, 0, row, half, g.splits);
          else if (threadIdx.x == 64) tell_lost<1>(lost_flag, 0, g.splits);
          cluster_sync();  // warps 0 and 1 join it below
          ok = ok && *lost_flag == 0;
        } else if (ok) {  // scaled (acc * (a_scale * w_scale[n])) and rounded to bf16, as the plain epilogue would store it
          const bool has_scale = g.a_scale != nullptr || g.w_scale != nullptr;
#pragma unroll 1
          for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
            uint32_t r[32];
            tmem_ld32(taddr + c * 32, r);
            tmem_wait_ld_into(r);
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float a = __uint_as_float(r[2 * j]), b = __uint_as_float(r[2 * j + 1]);
              if (has_scale) {
                a *= col[c * 32 + 2 * j];
                b *= col[c * 32 + 2 * j + 1];
              }
              w[j] = pack_bf16x2(a, b);
            }
            uint4* dst = reinterpret_cast<uint4*>(vt + row * (BN + 8) + c * 32);
#pragma unroll
            for (int v = 0; v < 4; ++v) dst[v] = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
          }
          asm volatile("bar.sync 2, 256;" ::: "memory");
        }
        if (ok) {
          const float4* parts = reinterpret_cast<const float4*>(smem + L::kSliceOffset);
          if (g.qkv.kv_fp8) qkv_finish<BN, true>(g, parts, vt, col, reinterpret_cast<const QkvShared*>(col + BN), fr, clustered ? g.splits : 1, slice_row0, slice_rows, m0, n0, pre);
          else qkv_finish<BN, false>(g, parts, vt, col, reinterpret_cast<const QkvShared*>(col + BN), fr, clustered ? g.splits : 1, slice_row0, slice_rows, m0, n0, pre);
        }
      }
    } else if (clustered) {
      if constexpr (BN == 64 && !QKV) {
        if (ok) push_slices<1, BN>(smem + L::kSliceOffset, taddr, split, 0, row, half, g.splits);
        else if (threadIdx.x == 64) tell_lost<1>(lost_flag, 0, g.splits);
        cluster_sync();  // every slice's share of this CTA's rows has arrived after this barrier (warps 0 and 1 join it below)
        if (ok && *lost_flag == 0) finish_slices<BN>(g, reinterpret_cast<const float4*>(smem + L::kSliceOffset), reinterpret_cast<const float*>(smem + L::kColOffset), m0, n0,
                                  slice_row0, slice_rows, one_gate, pre);
      }
    } else if (g.splits == 1) {
      // columns that are no multiple of 32, or a tile that spans several gate rows: half a row per thread, 16 columns at a time
      // (four warps with 8 columns at a time measured 9.0 against 7.5 us at 777 x 1096 x 1296 bf16, bias + SiLU)
      if (ok) {
        const float* col = reinterpret_cast<const float*>(smem + L::kColOffset);
        uint8_t* c_row = m < g.M ? row_of_c(g, m) : nullptr;
        const uint16_t* res_row = g.residual + static_cast<size_t>(m) * g.N + n0;
        const bool wide = g.N % 32 == 0 && (reinterpret_cast<uintptr_t>(g.C) & 31u) == 0;
#pragma unroll 1
        for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 16) {
          if (n0 + c >= g.N) break;
          uint32_t r[16];
          tmem_ld16(taddr + c, r);
          tmem_wait_ld_into(r);
          if (m < g.M) epilogue16<BN>(g, r, m, n0 + c, col + c, reinterpret_cast<const uint4*>(res_row + c), one_gate, c_row, wide, true);
        }
      }
    } else if (half == 1) {
      // K slices through the workspace are summed by the first four epilogue warps
    } else {
      // K slices through the global workspace: partial tile out, ticket, last CTA adds the slices in order
      float* part = g.partials + static_cast<size_t>(split) * g.M * g.N;
#pragma unroll 1
      for (int c = 0; ok && c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(taddr + c * 32, r);
        tmem_wait_ld_into(r);
        if (m < g.M) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int n = n0 + c * 32 + q * 4;
            if (n < g.N)
              __stcg(reinterpret_cast<float4*>(part + static_cast<size_t>(m) * g.N + n),
                     make_float4(__uint_as_float(r[q * 4]), __uint_as_float(r[q * 4 + 1]), __uint_as_float(r[q * 4 + 2]),
                                 __uint_as_float(r[q * 4 + 3])));
          }
        }
      }
      __threadfence();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      int* counter = g.counters + blockIdx.y * gridDim.x + blockIdx.x;
      if (threadIdx.x == 64) {
        const int ticket = atomicAdd(counter, ok ? 1 : kLostTicket + 1);
        const bool last = (ticket & (kLostTicket - 1)) == g.splits - 1;
        if (last) *counter = 0;  // ready for the next launch
        *last_flag = last && ok && ticket < kLostTicket;
        __threadfence();
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (*last_flag) {
        const int et = threadIdx.x - 64;  // 0..127
#pragma unroll 1
        for (int i8 = et; i8 < kBM * (BN / 8); i8 += 128) {
          const int mm = m0 + i8 / (BN / 8);
          const int n = n0 + (i8 % (BN / 8)) * 8;
          if (mm >= g.M || n >= g.N) continue;
          float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          for (int s = 0; s < g.splits; ++s) {
            const float4* src = reinterpret_cast<const float4*>(g.partials + (static_cast<size_t>(s) * g.M + mm) * g.N + n);
            const float4 x = __ldcg(src), y = __ldcg(src + 1);
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
            v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
          }
          epilogue_store8(g, v, mm, n);
        }
      }
    }
  }

  tc_fence_before();
  if (clustered && warp < 2) {
    __syncwarp();
    cluster_sync();  // the barrier after which the epilogue warps read what was pushed to them
  }
  __syncthreads();
  if (threadIdx.x == 0) QB_GT(6);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*ReplaceAddressFn)(CUtensorMap*, void*);

static void* driver_entry(const char* name) {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  return cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? p : nullptr;
}

// Tensor map of a contiguous row-major tensor [rows, cols] of 1- or 2-byte elements with a box of
// [box_rows, box_cols] elements; box_cols * elem_bytes must equal the swizzle span (64 or 128).
// Out-of-range parts of a box are filled with zeros.
//
// The driver's encoder takes longer than the rest of a small call's host side, so each thread keeps the maps of the last geometries
// and puts a call's own address into a copy: the layers of a model have a dozen geometries among hundreds of tensors.
int32_t make_tmap_2d_sw(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint32_t box_rows,
                        uint32_t box_cols, int swizzle_bytes) {
  struct Made {
    CUtensorMap map;
    uint64_t rows, cols;  // 0: empty
    uint32_t box_rows, box_cols;
    int elem_bytes, swizzle_bytes;
  };
  constexpr int kMade = 64;
  static thread_local Made made[kMade];
  static const auto encode = reinterpret_cast<EncodeTiledFn>(driver_entry("cuTensorMapEncodeTiled"));
  static const auto replace = reinterpret_cast<ReplaceAddressFn>(driver_entry("cuTensorMapReplaceAddress"));
  QB_REQUIRE(encode != nullptr && replace != nullptr, QB_ERR_CUDA, "the driver has no tensor maps");
  QB_REQUIRE(base != nullptr && aligned16(base), QB_ERR_ALIGN, "tensor map: address not 16-byte aligned");
  QB_REQUIRE((cols * elem_bytes) % 16 == 0, QB_ERR_ALIGN, "tensor map: row pitch of %llu bytes is not a multiple of 16",
             static_cast<unsigned long long>(cols * elem_bytes));
  const uint64_t h = ((rows * 31 + cols) * 31 + box_rows) * 0x9E3779B97F4A7C15ull;
  Made& m = made[(h >> 32) % kMade];
  if (m.rows == rows && m.cols == cols && m.box_rows == box_rows && m.box_cols == box_cols && m.elem_bytes == elem_bytes && m.swizzle_bytes == swizzle_bytes) {
    *tm = m.map;
    const CUresult r = replace(tm, const_cast<void*>(base));
    QB_REQUIRE(r == CUDA_SUCCESS, QB_ERR_CUDA, "cuTensorMapReplaceAddress failed with CUresult %d", static_cast<int>(r));
    return QB_OK;
  }
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * elem_bytes};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  const CUtensorMapSwizzle sw = swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
  const CUresult r = encode(tm, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  QB_REQUIRE(r == CUDA_SUCCESS, QB_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
  m = Made{*tm, rows, cols, box_rows, box_cols, elem_bytes, swizzle_bytes};
  return QB_OK;
}

static int32_t make_tmap_2d(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  return make_tmap_2d_sw(tm, base, elem_bytes, rows, cols, box_rows, static_cast<uint32_t>(kRowBytes / elem_bytes), 128);
}

// Tile counters of the workspace K slices live in a fixed area at the start of the workspace, so that calls of
// different shapes that share one workspace agree on where the counters end and the data begins (a
// shape-dependent area would let one call's e4m3 copy of A or partial sums land on counters that a later
// call with more tiles expects to find zero).
constexpr size_t kCounterBytes = 64u << 10;  // 16384 tiles

int num_sms() {
  static const int n = [] {
    int v = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    return v;
  }();
  return n;
}

// Whether `s` K slices of a tile can be summed inside a cluster (of at most 8 CTAs): the widths whose partial sums have room.
static bool cluster_slices(int cg, int bn, int s) { return cg == 1 ? bn == 64 && (s == 2 || s == 4 || s == 8) : bn == 128 && s == 2; }

// Picks the CTAs per tile, the tile width and the number of K slices from a small cost model in ns, so that every call with the
// same shape makes the same choice.
static GemmPlan make_plan(const qb_gemm_params& p, int max_cg, double* cost_out) {
  const bool fp8 = p.compute_dtype == QB_E4M3;
  const int k_elems = fp8 ? 128 : 64;
  GemmPlan best{};
  double best_cost = 1e30;
  const int sms = num_sms();
  const int kb_total = (p.K + k_elems - 1) / k_elems;
  const int bns[3] = {256, 128, 64};
  const int ss[10] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16};
  for (int cg = 1; cg <= max_cg; ++cg) {
    if (cg == 2 && (p.M <= kBM || (p.reserved & 1) != 0)) continue;
    for (int bn : bns) {
      if (p.tile_n != 0 && p.tile_n != bn) continue;
      if (cg == 2 && bn == 64) continue;
      if (p.tile_n == 0 && bn > 64 && bn / 2 >= p.N) continue;  // tile mostly empty
      const int tiles = ((p.M + cg * kBM - 1) / (cg * kBM)) * ((p.N + bn - 1) / bn);
      for (int s : ss) {
        if (p.split_k != 0 && p.split_k != s) continue;
        if (s > kb_total) continue;
        const int kbps = (kb_total + s - 1) / s;
        if ((kb_total + kbps - 1) / kbps != s) continue;
        const bool cl = s > 1 && (p.reserved & 1) == 0 && cluster_slices(cg, bn, s);
        if (s > 1 && p.split_k == 0 && kbps < 4) continue;  // too little K to share
        if (s > 1 && !cl && (cg == 2 || static_cast<size_t>(tiles) * sizeof(int) > kCounterBytes)) continue;  // more tiles than counters
        // Against every forced width and number of slices (60 shapes, M and N and K over the whole range, back to back with the
        // operands in L2) the choice is the fastest or within 2.5 % of it for nine in ten, at worst 9.5 % (7954 x 144 x 80 e4m3).
        // Measured with 128 CTAs, e4m3 and bf16 alike: ns per 128 bytes of K, and the rest of a launch that waits for the one
        // before it.  Tiles run in rounds over the SMs; a pair's CTAs stay for all rounds and hide all epilogues but the last.
        // Slices add their exchange: through the cluster it grows with the CTAs that push at once (16 CTAs 0.4 us, 128 CTAs
        // 1.3 - 2.5 us), the trip through the workspace is far slower.
        const double per_kb = cg == 1 ? (bn == 64 ? 143.0 : bn == 128 ? 190.0 : 390.0) : (bn == 128 ? 155.0 : 290.0);
        const double fixed = cg == 1 ? (bn == 64 ? 3150.0 : bn == 128 ? 3600.0 : 3400.0) : (bn == 128 ? 5200.0 : 5500.0);
        const double tail = cg == 1 ? 2200.0 + 7.0 * bn : bn == 128 ? 3200.0 : 4500.0;
        const long units = static_cast<long>(tiles) * (cl ? 1 : s);
        const long slots = cl && s == 4 ? 33 : cl && s == 8 ? 15 : sms / (cg * (cl ? s : 1));  // clusters that run at once
        const long rounds = (units + slots - 1) / slots;
        const double body = kbps * per_kb;
        double cost = fixed + body + (rounds - 1) * (cg == 1 ? body + tail : body > tail ? body : tail);
        if (s > 1) cost += cg == 2 ? 4000.0 : cl ? 300.0 + 12.0 * tiles * s : 9000.0;
        if (cost < best_cost) {
          best_cost = cost;
          best.cg = cg;
          best.bn = bn;
          best.splits = s;
          best.kb_total = kb_total;
          best.kb_per_split = kbps;
          best.cluster = cl ? 1 : 0;
        }
      }
    }
  }
  if (best.bn == 0) {  // forced values that fit nothing: fall back to the plain configuration
    best.cg = 1;
    best.bn = p.tile_n ? p.tile_n : 128;
    best.splits = 1;
    best.kb_total = kb_total;
    best.kb_per_split = kb_total;
  }
  *cost_out = best_cost;
  best.counters_bytes = kCounterBytes;
  best.aq_bytes = (fp8 && p.a_dtype == QB_BF16) ? round_up(static_cast<size_t>(p.M) * p.K, 1024) : 0;
  best.partial_bytes = (best.splits > 1 && !best.cluster) ? static_cast<size_t>(best.splits) * p.M * p.N * sizeof(float) : 0;
  return best;
}

// The plan of a shape that this thread planned a moment ago is read back: a call plans twice (its workspace, then its launch), and
// the model above takes about as long as a launch.
static GemmPlan plan_gemm(const qb_gemm_params& p, int max_cg = 2, double* cost_out = nullptr) {
  struct Key {
    int32_t M, N, K, a_dtype, compute_dtype, split_k, tile_n, no_cluster, max_cg;
    bool operator==(const Key& o) const {
      return M == o.M && N == o.N && K == o.K && a_dtype == o.a_dtype && compute_dtype == o.compute_dtype && split_k == o.split_k && tile_n == o.tile_n &&
             no_cluster == o.no_cluster && max_cg == o.max_cg;
    }
  };
  struct Made {
    Key key;  // M 0: empty
    GemmPlan plan;
    double cost;
  };
  constexpr int kMade = 16;
  static thread_local Made made[kMade];
  const Key key{p.M, p.N, p.K, p.a_dtype, p.compute_dtype, p.split_k, p.tile_n, p.reserved & 1, max_cg};
  const uint32_t h = (static_cast<uint32_t>(p.M) * 31u + static_cast<uint32_t>(p.N)) * 31u + static_cast<uint32_t>(p.K) + static_cast<uint32_t>(p.split_k) * 5u +
                     static_cast<uint32_t>(p.tile_n >> 6);
  Made& m = made[(h * 0x9E3779B1u >> 16) % kMade];
  if (!(m.key == key)) {
    m.plan = make_plan(p, max_cg, &m.cost);
    m.key = key;
  }
  if (cost_out != nullptr) *cost_out = m.cost;
  return m.plan;
}

static int32_t validate_gemm(const qb_gemm_params* p) {
  QB_REQUIRE(p != nullptr, QB_ERR_INVALID_ARG, "gemm params are NULL");
  QB_REQUIRE(p->M > 0 && p->N > 0 && p->K > 0, QB_ERR_INVALID_ARG, "gemm: M, N, K must be positive (got %d, %d, %d)", p->M, p->N, p->K);
  QB_REQUIRE(p->compute_dtype == QB_BF16 || p->compute_dtype == QB_E4M3, QB_ERR_INVALID_ARG, "gemm: compute_dtype %d", p->compute_dtype);
  if (p->compute_dtype == QB_BF16) {
    QB_REQUIRE(p->a_dtype == QB_BF16 && p->b_dtype == QB_BF16, QB_ERR_INVALID_ARG, "gemm: bf16 compute needs bf16 A and B");
  } else {
    QB_REQUIRE(p->b_dtype == QB_E4M3, QB_ERR_INVALID_ARG, "gemm: e4m3 compute needs an e4m3 B (weights are quantised ahead of time)");
    QB_REQUIRE(p->a_dtype == QB_E4M3 || p->a_dtype == QB_BF16, QB_ERR_INVALID_ARG, "gemm: A must be bf16 or e4m3");
  }
  QB_REQUIRE(p->c_dtype == QB_BF16 || p->c_dtype == QB_F32 || p->c_dtype == QB_E4M3, QB_ERR_INVALID_ARG, "gemm: c_dtype %d", p->c_dtype);
  QB_REQUIRE(p->K % 16 == 0, QB_ERR_ALIGN, "gemm: K = %d must be a multiple of 16", p->K);
  QB_REQUIRE(p->N % 8 == 0, QB_ERR_ALIGN, "gemm: N = %d must be a multiple of 8", p->N);
  QB_REQUIRE(p->activation == 0 || p->activation == 1, QB_ERR_INVALID_ARG, "gemm: activation %d", p->activation);
  QB_REQUIRE(p->tile_n == 0 || p->tile_n == 64 || p->tile_n == 128 || p->tile_n == 256, QB_ERR_INVALID_ARG, "gemm: tile_n %d", p->tile_n);
  QB_REQUIRE(p->split_k >= 0 && p->split_k <= 16, QB_ERR_INVALID_ARG, "gemm: split_k %d", p->split_k);
  QB_REQUIRE(p->reserved >= 0 && p->reserved <= 7, QB_ERR_INVALID_ARG, "gemm: flags %d", p->reserved);
  return QB_OK;
}

template <int BN, bool FP8, bool QKV>
static int32_t launch_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& args, dim3 grid, cudaStream_t st) {
  using L = GemmSmem<BN>;
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  int dev = 0;
  QB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 64 || (configured.load(std::memory_order_relaxed) >> dev & 1) == 0) {
    QB_CUDA_OK(cudaFuncSetAttribute(gemm_kernel<BN, FP8, QKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
    if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  if (args.cluster) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = L::kTotal;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = static_cast<unsigned>(args.splits);
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_dependent_launch ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_kernel<BN, FP8, QKV>, tmA, tmB, args);
    ++g_launch_count;
    if (e != cudaSuccess) return fail(QB_ERR_LAUNCH, "gemm kernel (cluster of %d): %s", args.splits, cudaGetErrorString(e));
    return QB_OK;
  }
  return launch_dep("gemm kernel", gemm_kernel<BN, FP8, QKV>, grid, dim3(kGemmThreads), L::kTotal, st, tmA, tmB, args);
}

template <bool FP8>
static int32_t launch_gemm(int bn, bool qkv, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& g, dim3 grid, cudaStream_t st) {
  if (qkv) return bn == 128 ? launch_gemm<128, FP8, true>(tmA, tmB, g, grid, st) : launch_gemm<64, FP8, true>(tmA, tmB, g, grid, st);
  if (bn == 256) return launch_gemm<256, FP8, false>(tmA, tmB, g, grid, st);
  if (bn == 128) return launch_gemm<128, FP8, false>(tmA, tmB, g, grid, st);
  return launch_gemm<64, FP8, false>(tmA, tmB, g, grid, st);
}

int32_t quantize_e4m3_launch(const void* X, void* out, size_t n, int32_t src_dtype, cudaStream_t st);

}  // namespace qb

using namespace qb;

#ifdef QB_GEMM_TRACE
extern "C" int32_t qb_debug_gemm_trace(void* host_out) {
  return cudaMemcpyFromSymbol(host_out, qb::g_gemm_trace, sizeof(qb::g_gemm_trace)) == cudaSuccess ? 0 : -1;
}
#endif

extern "C" size_t qb_gemm_workspace_bytes(const qb_gemm_params* p) {
  if (validate_gemm(p) != QB_OK) return 0;
  const GemmPlan pl = plan_gemm(*p);
  if (pl.aq_bytes == 0 && pl.partial_bytes == 0) return 0;  // no scratch memory is touched
  return pl.counters_bytes + pl.aq_bytes + pl.partial_bytes;
}

// clear_counters: the workspace may hold anything (the built-in scratch array keeps the last call's contents), so the
// tile counters are zeroed on the stream first, after every check has passed and only if this plan reads them.
struct TpDest {
  int world, rpo;
  uint16_t* dst[8];
};

// The QKV projection with its fused epilogue: tiles of one or two heads of one CTA, and the K slices that the plain projection
// would have with 64-column tiles, as long as whole 16-byte vectors of cached V tokens lie in the 128 / S rows that a CTA finishes.
static GemmPlan plan_qkv(const qb_gemm_params& p, const QkvTail& t) {
  qb_gemm_params q = p;
  GemmPlan best{};
  double best_cost = 1e30;
  for (int bn = 64; bn <= 128; bn += 64) {
    for (int s = 1; s <= (bn == 64 ? 4 : 1); s *= 2) {
      if (s > 1 && (kBM / s % t.quilt != 0 || kBM / s / t.quilt < (t.kv_fp8 ? 16 : 8))) continue;
      q.tile_n = bn;
      q.split_k = s;
      double cost = 0;
      const GemmPlan pl = plan_gemm(q, 1, &cost);
      if (pl.splits == s && pl.cluster == (s > 1) && cost < best_cost) {
        best_cost = cost;
        best = pl;
      }
    }
  }
  return best;
}

// Column width of the grouped GEMM's tiles: the one whose CTAs (256 rows of an expert each) take the fewest rounds over the SMs, by
// the rows that its slots leave once every expert's run is padded to 128.
static int plan_grouped(const qb_gemm_params& p, int n_experts) {
  if (p.tile_n != 0) return p.tile_n;
  const int kb = (p.K + (p.compute_dtype == QB_E4M3 ? 127 : 63)) / (p.compute_dtype == QB_E4M3 ? 128 : 64);
  int rows = p.M - kBM * n_experts;
  if (rows < p.M / 2) rows = p.M / 2;
  const int per_expert = rows / n_experts + 1;
  const bool two = per_expert > 96;  // about every second run then spills into a second tile of 128 rows
  int best = 64;
  double best_cost = 1e30;
  for (int bn = 64; bn <= 256; bn *= 2) {
    if (bn > 64 && bn / 2 >= p.N) continue;
    const int ctas = n_experts * ((per_expert + 255) / 256) * ((p.N + bn - 1) / bn);
    const double per_kb = two ? (bn == 64 ? 240.0 : bn == 128 ? 300.0 : 540.0) : (bn == 64 ? 150.0 : bn == 128 ? 220.0 : 420.0);
    const double cost = ((ctas + num_sms() - 1) / num_sms()) * (kb * per_kb + 3500.0 + bn * 6.0);
    if (cost < best_cost) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

static int32_t gemm_run(const void* A, const void* B, void* C, const void* bias, const void* gate, const void* residual,
                        const qb_gemm_params* p, void* workspace, size_t workspace_bytes, void* stream, const QkvTail* tail,
                        bool clear_counters = false, const TpDest* tp = nullptr, const int* tile_expert = nullptr, int n_experts = 1) {
  int32_t rc = validate_gemm(p);
  if (rc != QB_OK) return rc;
  QB_REQUIRE(A && B && C, QB_ERR_INVALID_ARG, "gemm: A, B and C must not be NULL");
  QB_REQUIRE((gate == nullptr) == (residual == nullptr), QB_ERR_INVALID_ARG, "gemm: gate and residual come together");
  QB_REQUIRE(aligned16(A) && aligned16(B) && aligned16(C) && aligned16(bias) && aligned16(gate) && aligned16(residual), QB_ERR_ALIGN,
             "gemm: every pointer must be 16-byte aligned");
  int rows_per_gate = p->M;
  if (gate != nullptr) {
    QB_REQUIRE(p->gate_groups >= 1 && p->M % p->gate_groups == 0, QB_ERR_INVALID_ARG, "gemm: gate_groups %d does not divide M = %d",
               p->gate_groups, p->M);
    rows_per_gate = p->M / p->gate_groups;
  }
  GemmPlan pl = plan_gemm(*p, tp != nullptr ? 1 : 2);
  if (tail != nullptr) pl = plan_qkv(*p, *tail);
  const size_t need = pl.counters_bytes + pl.aq_bytes + pl.partial_bytes;
  const bool uses_ws = pl.aq_bytes > 0 || pl.partial_bytes > 0;
  if (uses_ws) {
    QB_REQUIRE(workspace != nullptr && workspace_bytes >= need, QB_ERR_WORKSPACE, "gemm: workspace of %zu bytes needed, %zu given", need,
               workspace_bytes);
    QB_REQUIRE(aligned16(workspace), QB_ERR_ALIGN, "gemm: workspace must be 16-byte aligned");
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool fp8 = p->compute_dtype == QB_E4M3;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  unsigned int* status = status_word();
  QB_REQUIRE(status != nullptr, QB_ERR_CUDA, "gemm: device status word unavailable");
  if (clear_counters && pl.partial_bytes > 0) QB_CUDA_OK(cudaMemsetAsync(ws, 0, pl.counters_bytes, st));
  const void* a_ptr = A;
  if (pl.aq_bytes > 0) {
    uint8_t* aq = ws + pl.counters_bytes;
    rc = quantize_e4m3_launch(A, aq, static_cast<size_t>(p->M) * p->K, QB_BF16, st);
    if (rc != QB_OK) return rc;
    a_ptr = aq;
  }
  GemmArgs g{};
  g.M = p->M; g.N = p->N; g.K = p->K;
  g.a_rows = p->M < kBM ? (p->M + 7) / 8 * 8 : kBM;
  g.kb_total = pl.kb_total; g.kb_per_split = pl.kb_per_split; g.splits = pl.splits;
  g.cluster = pl.cluster;
  g.b_const = (p->reserved & 2) != 0;
  g.through_bf16 = (p->reserved & 4) != 0;
  QB_REQUIRE(!g.through_bf16 || tile_expert != nullptr, QB_ERR_UNSUPPORTED, "gemm: flag bit 2 belongs to the grouped GEMM");
  g.c_dtype = p->c_dtype; g.activation = p->activation; g.rows_per_gate = rows_per_gate;
  g.a_scale = p->a_scale; g.w_scale = p->w_scale;
  g.bias = static_cast<const uint16_t*>(bias);
  g.gate = static_cast<const uint16_t*>(gate);
  g.residual = static_cast<const uint16_t*>(residual);
  g.C = C;
  g.counters = reinterpret_cast<int*>(ws);
  g.partials = pl.partial_bytes ? reinterpret_cast<float*>(ws + pl.counters_bytes + pl.aq_bytes) : nullptr;
  g.status = status;
  if (tp != nullptr) {
    // the per-row destinations exist in the one-slice fast epilogue only: whole 32-column chunks, bf16, no gate
    QB_REQUIRE(pl.splits == 1 && p->N % 32 == 0 && p->c_dtype == QB_BF16 && gate == nullptr && tail == nullptr, QB_ERR_UNSUPPORTED,
               "gemm_tp: needs one K slice, N a multiple of 32, bf16 output, no gate");
    g.tp_world = tp->world;
    g.tp_rpo = tp->rpo;
    for (int r = 0; r < tp->world; ++r) g.tp_dst[r] = tp->dst[r];
  }
  if (tail != nullptr) {
    g.qkv = *tail;
  }
  if (tile_expert != nullptr) {
    QB_REQUIRE(p->M % kBM == 0, QB_ERR_UNSUPPORTED, "gemm_grouped: M = %d must be a multiple of 128", p->M);
    // per-column vectors would have to be per expert
    QB_REQUIRE(tail == nullptr && tp == nullptr && bias == nullptr && gate == nullptr && p->w_scale == nullptr,
               QB_ERR_UNSUPPORTED, "gemm_grouped: takes the plain or the SiLU epilogue only");
    g.tile_expert = tile_expert;
  }

  if (tile_expert != nullptr) return launch_gemm_grouped(plan_grouped(*p, n_experts), a_ptr, B, n_experts, g, fp8, st);
  if (pl.cg == 2) return launch_gemm_pair(pl, a_ptr, B, g, fp8, st);
  CUtensorMap tmA, tmB;
  const int es = fp8 ? 1 : 2;
  rc = make_tmap_2d(&tmA, a_ptr, es, p->M, p->K, g.a_rows);
  if (rc != QB_OK) return rc;
  rc = make_tmap_2d(&tmB, B, es, p->N, p->K, pl.bn);
  if (rc != QB_OK) return rc;

  dim3 grid((p->N + pl.bn - 1) / pl.bn, (p->M + kBM - 1) / kBM, pl.splits);
  return fp8 ? launch_gemm<true>(pl.bn, tail != nullptr, tmA, tmB, g, grid, st) : launch_gemm<false>(pl.bn, tail != nullptr, tmA, tmB, g, grid, st);
}

extern "C" int32_t qb_gemm(const void* A, const void* B, void* C, const void* bias, const void* gate, const void* residual,
                           const qb_gemm_params* p, void* workspace, size_t workspace_bytes, void* stream) {
  return gemm_run(A, B, C, bias, gate, residual, p, workspace, workspace_bytes, stream, nullptr);
}

extern "C" int32_t qb_gemm_qkv_post(const void* A, const void* B, void* qkv_out, const void* qkv_first, const float* lamb,
                                    const int32_t* frame_t, const int32_t* frozen, void* K_cache, void* Vt_cache, int32_t* segments,
                                    int32_t* n_segments, const float* rope_xy, const qb_gemm_params* gp, const qb_kv_params* kp, float eps,
                                    void* workspace, size_t workspace_bytes, void* stream) {
  QB_REQUIRE(gp != nullptr && kp != nullptr, QB_ERR_INVALID_ARG, "gemm_qkv_post: params are NULL");
  QB_REQUIRE(qkv_out && frame_t && frozen && K_cache && Vt_cache && segments && n_segments && rope_xy, QB_ERR_INVALID_ARG,
             "gemm_qkv_post: NULL pointer");
  QB_REQUIRE((qkv_first == nullptr) == (lamb == nullptr), QB_ERR_INVALID_ARG, "gemm_qkv_post: qkv_first and lamb come together");
  QB_REQUIRE(kp->packed_qkv == 1, QB_ERR_UNSUPPORTED, "gemm_qkv_post: the packed QKV layout only");
  // a 128-token tile must hold whole 16-byte vectors of cached V tokens (8 bf16 / 16 e4m3 per vector)
  QB_REQUIRE(kp->quilt_factor >= 1 && (kp->quilt_factor & (kp->quilt_factor - 1)) == 0 &&
                 kp->quilt_factor * (kp->kv_dtype == QB_E4M3 ? 16 : 8) <= 128,
             QB_ERR_UNSUPPORTED, "gemm_qkv_post: quilt_factor %d (a power of two, at most %d for this cache dtype)", kp->quilt_factor,
             kp->kv_dtype == QB_E4M3 ? 8 : 16);
  QB_REQUIRE(kp->quilt_offset >= 0 && kp->quilt_offset < kp->quilt_factor, QB_ERR_INVALID_ARG, "gemm_qkv_post: quilt_offset %d", kp->quilt_offset);
  QB_REQUIRE(kp->n_kv_heads > 0 && kp->n_q_heads > 0 && kp->n_q_heads % kp->n_kv_heads == 0, QB_ERR_INVALID_ARG,
             "gemm_qkv_post: %d Q heads over %d KV heads", kp->n_q_heads, kp->n_kv_heads);
  QB_REQUIRE(kp->H_spatial > 0 && kp->W_spatial > 0 && kp->num_buckets > 0 && kp->pinned_dilation > 0, QB_ERR_INVALID_ARG,
             "gemm_qkv_post: sizes must be positive");
  QB_REQUIRE(kp->kv_dtype == QB_BF16 || kp->kv_dtype == QB_E4M3, QB_ERR_INVALID_ARG, "gemm_qkv_post: kv_dtype %d", kp->kv_dtype);
  QB_REQUIRE(kp->max_segments >= 3, QB_ERR_INVALID_ARG, "gemm_qkv_post: max_segments %d < 3", kp->max_segments);
  const int tpf = kp->H_spatial * kp->W_spatial;
  QB_REQUIRE(gp->M == tpf && gp->N == (kp->n_q_heads + 2 * kp->n_kv_heads) * 64, QB_ERR_INVALID_ARG,
             "gemm_qkv_post: the projection is [%d, %d] but the geometry needs [%d, %d]", gp->M, gp->N, tpf,
             (kp->n_q_heads + 2 * kp->n_kv_heads) * 64);
  QB_REQUIRE((tpf / kp->quilt_factor) % 16 == 0 && tpf % kp->quilt_factor == 0, QB_ERR_UNSUPPORTED,
             "gemm_qkv_post: H*W / quilt_factor = %d / %d must be a multiple of 16", tpf, kp->quilt_factor);
  QB_REQUIRE(gp->c_dtype == QB_BF16 && gp->activation == 0, QB_ERR_INVALID_ARG, "gemm_qkv_post: bf16 output without activation");
  QB_REQUIRE((reinterpret_cast<uintptr_t>(qkv_out) & 31u) == 0 && (reinterpret_cast<uintptr_t>(K_cache) & 31u) == 0 && aligned16(Vt_cache) &&
                 aligned16(qkv_first) && aligned16(rope_xy),
             QB_ERR_ALIGN, "gemm_qkv_post: qkv_out and K_cache must be 32-byte aligned, the other pointers 16-byte aligned");
  qb_gemm_params p = *gp;
  p.tile_n = p.split_k = 0;
  QkvTail t{};
  t.qkv_first = static_cast<const uint16_t*>(qkv_first);
  t.lamb = lamb; t.frame_t = frame_t; t.frozen = frozen;
  t.K_cache = K_cache; t.Vt_cache = Vt_cache; t.segments = segments; t.n_segments = n_segments; t.rope_xy = rope_xy;
  t.n_q_heads = kp->n_q_heads; t.n_kv_heads = kp->n_kv_heads; t.tpf = tpf; t.nb = kp->num_buckets; t.pd = kp->pinned_dilation;
  t.max_segments = kp->max_segments; t.kv_fp8 = kp->kv_dtype == QB_E4M3; t.eps = eps;
  t.k_scale = kp->k_scale; t.v_scale = kp->v_scale;
  t.quilt = kp->quilt_factor; t.qoff = kp->quilt_offset;
  return gemm_run(A, B, qkv_out, nullptr, nullptr, nullptr, &p, workspace, workspace_bytes, stream, &t);
}

extern "C" int32_t qb_gemm_tp(const void* A, const void* B, const qb_gemm_params* p, const qb_tp_params* tp, void* workspace,
                              size_t workspace_bytes, void* stream) {
  QB_REQUIRE(p != nullptr && tp != nullptr, QB_ERR_INVALID_ARG, "gemm_tp: params are NULL");
  QB_REQUIRE(tp->world >= 1 && tp->world <= 8 && tp->rank >= 0 && tp->rank < tp->world, QB_ERR_INVALID_ARG, "gemm_tp: rank %d of %d", tp->rank,
             tp->world);
  QB_REQUIRE(tp->rows == p->M && tp->D == p->N && p->M % tp->world == 0, QB_ERR_INVALID_ARG,
             "gemm_tp: the partial is [%d, %d] but the arenas are laid out for [%d, %d] over %d ranks", p->M, p->N, tp->rows, tp->D, tp->world);
  qb_gemm_params q = *p;
  q.split_k = 1;  // the partial must leave the kernel in one piece
  TpDest d{};
  d.world = tp->world;
  d.rpo = p->M / tp->world;
  size_t off[6];
  int32_t rc = qb_tp_arena_offsets(tp->rows, tp->D, off);
  if (rc != QB_OK) return rc;
  for (int r = 0; r < tp->world; ++r) {
    QB_REQUIRE(tp->arena[r] != nullptr, QB_ERR_INVALID_ARG, "gemm_tp: arena %d is NULL", r);
    // rank r's staging area (its y slot 0) holds one block of rows per source rank: [source][rows / world][D]
    d.dst[r] = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(tp->arena[r]) + off[0]) + static_cast<size_t>(tp->rank) * d.rpo * p->N;
  }
  // C is unused (every row has a destination of its own); the rank's own staging block stands in for the pointer checks
  return gemm_run(A, B, d.dst[tp->rank], nullptr, nullptr, nullptr, &q, workspace, workspace_bytes, stream, nullptr, false, &d);
}

extern "C" size_t qb_gemm_grouped_workspace_bytes(const qb_gemm_params* p) {
  if (validate_gemm(p) != QB_OK) return 0;
  qb_gemm_params q = *p;
  q.split_k = 1;
  return qb_gemm_workspace_bytes(&q);
}

extern "C" int32_t qb_gemm_grouped(const void* A, const void* B, void* C, const int32_t* tile_expert, int32_t n_experts, const qb_gemm_params* p,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  QB_REQUIRE(p != nullptr && tile_expert != nullptr, QB_ERR_INVALID_ARG, "gemm_grouped: params or tile table are NULL");
  QB_REQUIRE(n_experts >= 1 && static_cast<long long>(n_experts) * p->N < (1ll << 31), QB_ERR_INVALID_ARG, "gemm_grouped: %d experts", n_experts);
  qb_gemm_params q = *p;
  q.split_k = 1;  // a padding tile leaves before any K slice could wait for it
  return gemm_run(A, B, C, nullptr, nullptr, nullptr, &q, workspace, workspace_bytes, stream, nullptr, false, nullptr, tile_expert, n_experts);
}

// ---------------------------------------------------------------- GEMM on built-in scratch memory
// Scratch for qb_gemm_static_scratch: lives in the library image, so every GPU that loads the library
// holds these 8 MiB until the process exits.  In host code the name below is only a handle for
// cudaGetSymbolAddress; the device address it yields is what the kernels receive.
namespace qb {
constexpr size_t kStaticScratchBytes = 8u << 20;
static __device__ __align__(256) unsigned char g_gemm_static_scratch[kStaticScratchBytes];

// Device address of the scratch array on the calling thread's current device (the device the stream must belong
// to), looked up once per device and published with a release store, so that two host threads that make their
// first calls at the same time both end up with the same, fully written entry.  cudaDeviceReset invalidates
// the entry of that device; a process that resets a device must not call this entry point on it afterwards.
static int32_t static_scratch_ptr(void** out) {
  static std::atomic<void*> cache[64];
  int dev = 0;
  QB_CUDA_OK(cudaGetDevice(&dev));
  QB_REQUIRE(dev >= 0 && dev < 64, QB_ERR_DEVICE, "gemm_static_scratch: device ordinal %d out of range", dev);
  void* p = cache[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    QB_CUDA_OK(cudaGetSymbolAddress(&p, g_gemm_static_scratch));
    QB_REQUIRE(p != nullptr, QB_ERR_CUDA, "gemm_static_scratch: cudaGetSymbolAddress returned a null address");
    cache[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return QB_OK;
}
}  // namespace qb

extern "C" size_t qb_gemm_static_scratch_capacity(void) { return qb::kStaticScratchBytes; }

extern "C" int32_t qb_gemm_static_scratch(const void* A, const void* B, void* C, const void* bias, const void* gate,
                                          const void* residual, const qb_gemm_params* p, void* stream) {
  int32_t rc = validate_gemm(p);
  if (rc != QB_OK) return rc;
  const GemmPlan pl = plan_gemm(*p);
  const size_t need = pl.counters_bytes + pl.aq_bytes + pl.partial_bytes;
  QB_REQUIRE(need <= kStaticScratchBytes, QB_ERR_WORKSPACE,
             "gemm_static_scratch: this GEMM needs %zu bytes of scratch but the built-in scratch holds %zu; "
             "use qb_gemm with a caller-provided workspace, or force a smaller split_k",
             need, static_cast<size_t>(kStaticScratchBytes));
  void* scratch = nullptr;
  rc = static_scratch_ptr(&scratch);
  if (rc != QB_OK) return rc;
  // The array keeps whatever the previous call left.  Only the tile counters must start at zero (the e4m3 copy of
  // A and the K-slice partials are fully written before they are read); gemm_run clears them on the stream once all
  // of its own checks have passed, and only when this plan sums K slices through the scratch memory.
  return gemm_run(A, B, C, bias, gate, residual, p, scratch, kStaticScratchBytes, stream, nullptr, true);
}
