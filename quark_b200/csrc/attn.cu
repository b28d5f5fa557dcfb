// owl_attn: segment-sparse GQA flash attention with inline ortho-RoPE on Q, head_dim 64.  This file: the host side, and the kernel for
// e4m3 caches and for key splits in either type; bf16 without key splits is in attn3.cu.
//
// One CTA owns 128 query tokens of one Q head and walks the valid keys in tiles of 128, enumerated from the (start, length)
// segment table, so a masked bucket is never loaded.  384 threads:
//   warp 0        TMA producer: a ring of K tiles [128 keys x 64] and one of V^T tiles [64 x 128 keys] (e4m3: + 16 rows of ones)
//   warps 1, 2    one thread each issues tcgen05.mma for softmax group 0 / 1: S = Q K^T and O += P V
//   warp 3        sines and cosines of the temporal angles
//   warps 4-7     softmax group 0: even key tiles        warps 8-11  softmax group 1: odd key tiles
// After set-up the control warps hand registers to the softmax warps (setmaxnreg), each of whose
// threads holds a whole score row of one query (128 values).
//
// Per group, TMEM holds one S tile (128 columns), the accumulator O and P (the A operand of O += P V).  A softmax
// thread copies its row of S(i) to registers (S(i + 1) may then be computed), takes the row maximum, makes P(i) = 2^(score - m) and
// stores it, packed, once PV(i - 1) has read the P before: long ago, since the exponentials of tile i come in between.
// m is the maximum the row was last rescaled to, not the running maximum: O (and the row sum) are multiplied by 2^(m - m') only when
// a tile's maximum exceeds m by more than kSlack, which is rare after the first tiles.
// The two groups' results (m, row sum, 64 outputs) are merged once at the end.
//
// The row sum is that of exactly the rounded P that is multiplied with V.  In e4m3 the tensor core makes it: 16 rows of ones follow the
// 64 V^T rows of every stage, so PV has 80 columns and column 64 is sum_k P[q, k].  bf16 path: kind::f16 MMAs, P rounded to bf16.  fp8
// path: Q (after RoPE), K, V and P are e4m3 (kind::f8f6f4); P is scaled by 2^kPShift so small probabilities keep mantissa bits (the
// factor cancels in the division by the row sum).  exp2 is ex2.approx.f32 (ex2.approx.f16x2 issues at half the rate of the f32 form: no
// gain per element), the chord of ex2_lin_from_biased for every second e4m3 probability, a polynomial for every fourth bf16 one.
//
// What bounds it (e4m3, 720p, 8320 keys): instruction issue of the softmax warps, two per scheduler.  A loop with the same softmax
// instructions and nothing else takes 726 cycles per tile, with one warp per scheduler 911; this kernel 1040, the waits, fences and
// arrivals of a tile being what the other warp covers in part only.  Before (47.8 us at 16 buckets, 318 at 128, 168 at 64), a stage of
// the one K / V ring was held from S to PV, so the MMA threads waited 850 to 1350 cycles per tile for K, and P went through shared
// memory with the groups taking turns on the exponentials; now 41.4, 272 and 143 us.  Tried and dropped: the turns kept (46.0); a third
// group of warps for the maxima (50.3: S, maximum, exponentials in a row take longer than the tile before covers); three groups over
// 64-key tiles (46.9: the fixed work of a tile twice); the chord's integer multiply-add held on the FMA pipe (42.9).
#include <atomic>

#include <cuda.h>

#include "attn_common.cuh"

namespace qb {

int num_sms();
int32_t launch_attn3(const CUtensorMap& tmK, const CUtensorMap& tmV, const AttnArgs& a, int Hq, bool helped, cudaStream_t st);
int32_t make_tmap_2d_sw(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint32_t box_rows,
                        uint32_t box_cols, int swizzle_bytes);

constexpr int kAttnThreads = 384;
// setmaxnreg moves registers inside the pool the CTA was given at launch (384 threads x 168 registers): an increase waits until
// other warps of the CTA have released enough, so the budget must close or the softmax warps would wait for ever.
constexpr int kLaunchRegs = 168;
constexpr int kCtrlRegs = 72;      // per thread, warps 0-3
constexpr int kSoftmaxRegs = 216;  // per thread, warps 4-11
static_assert(128 * kCtrlRegs + 256 * kSoftmaxRegs <= kAttnThreads * kLaunchRegs, "register budget of the CTA");

// Cluster splits: 2 groups x S CTAs leave 64 outputs, m, the row sum and whether they are to be used of each query row with the CTA that
// writes the row (128 / S rows each): 17 units of 16 bytes a row, [2 S][17][rows].  Neighbouring rows (the lanes of a pushing warp) are
// neighbours, and each unit's rows are rotated so that the units of a row (the lanes that read them) lie in different banks.
constexpr int kUnits = 17;
__host__ __device__ constexpr int merge_rows(int splits) { return (kQTile + splits - 1) / splits; }
__device__ __forceinline__ int merge_unit(int part, int u, int row, int rows) {
  const int turned = row + u * (1 + (rows & 1));
  return (part * kUnits + u) * rows + turned % rows;
}

template <bool kFp8, bool kCluster = false>
struct AttnSmem {
  static constexpr int kEs = kFp8 ? 1 : 2;
  // Of each ring.  A stage is given back when its MMAs are done, so the groups hold those of up to four tiles; with four stages the next
  // tiles were only asked for when they were needed (e4m3, 720p: 47.8 -> 42.5 us with eight).  Even: a stage then belongs to one
  // group's tiles.  (With three a group waited for a phase of a stage whose previous phase the other group watches: where that earlier
  // copy was still on its way, the parity wait returned at once.)
  static constexpr int kKStages = kFp8 ? (kCluster ? 6 : 8) : 4, kVStages = kFp8 ? (kCluster ? 6 : 8) : (kCluster ? 4 : 6);
  // e4m3: 16 rows of ones under the 64 V^T rows make the tensor core return the row sum of P in column 64 of O.  bf16 has no TMEM
  // columns left for that (S 128, O 64, P 64 a group): the softmax threads add up the rounded probabilities.
  static constexpr int kRows = kFp8 ? kVRows : 64;
  static constexpr int kQBytes = kQTile * 64 * kEs;          // 8 KB | 16 KB
  static constexpr int kKBytes = kKeyTile * 64 * kEs;        // 8 KB | 16 KB
  static constexpr int kVTile = kRows * 128;                 // 128 bytes of keys a row: 10 KB | 8 KB
  static constexpr int kVBytes = kVTile * kEs;               // bf16: two (keys 0-63, 64-127)
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kQOff + kQBytes;
  static constexpr int kVOff = kKOff + kKStages * kKBytes;
  static constexpr int kMergeBytes = 266 * kUnits * 16;        // 2 groups, S CTAs, 128 / S rows each (7 CTAs need most)
  static constexpr int kCombOff = kVOff + kVStages * kVBytes;  // where the groups meet | the CTAs of a cluster (memory of its own, since others push early)
  static constexpr int kBarOff = kCombOff + (kCluster ? kMergeBytes : 2 * 34 * kQTile * 4);
  static constexpr int kTotal = kBarOff + 640 + 1024;
  static_assert(kKStages % 2 == 0 && kVStages % 2 == 0 && kTotal <= 227 * 1024, "see kKStages; shared memory of one CTA");
};

// What follows the rings in shared memory.
struct AttnBars {
  uint64_t k_full[8], k_empty[8], v_full[8], v_empty[8];
  uint64_t s_full[2];       // [group] S(i) is in TMEM
  uint64_t s_free[2];       // [group] the group holds S(i) in registers
  uint64_t p_full[2];       // [group] P(i) is in TMEM
  uint64_t pv_done[2];      // [group] O += P(i) V(i) has finished
  uint64_t o_final[2];      // [group] every PV of a piece has finished
  uint64_t q_ready;
  uint32_t tmem_slot;
  int abort_flag, drain_flag, exchange;
  float tm[16];  // cosines and sines of the temporal angles
  int seg[6];    // the segment table, for tiles that need a mask: tile j of the CTA is tile j + tile_shift of the table
  int tiles, tile_shift;  // kHelped: tiles of an item
};
static_assert(sizeof(AttnBars) <= 640, "kBarOff + 640");

// Tiles j = 2 i + g, i = 0, 1, ..., below `end`: those of softmax group g.
__device__ __forceinline__ int group_tiles(int end, int g) { return (end - g + 1) >> 1; }

// 32 scores of one row -> packed probabilities 2^(score * sl2 + nshift); bf16: `sum` grows by the rounded ones.  e4m3 makes every second
// one by the chord of ex2_lin_from_biased (kLin), or none: the setting is there for ex2.approx throughout (720p: 57.0 us; every fourth by the
// polynomial took 50.9).  bf16 takes every fourth from the polynomial, since the special-function unit would be the bound (360p: 14.2 -> 13.5).
template <bool kFp8, bool kLin>
__device__ __forceinline__ void p_chunk(const uint32_t (&s)[32], uint64_t sl2, uint64_t nshift, uint32_t* w, uint64_t (&sum)[2]) {
  float e[32];
#pragma unroll
  for (int q = 0; q < 32; q += 2) {
    fma_f32x2(e[q], e[q + 1], s[q], s[q + 1], sl2, nshift);
    if (!kFp8 && (q & 7) == 6) {
      ex2_poly_f32x2(e[q], e[q + 1]);
      continue;
    }
    e[q] = ex2_approx(e[q]);
    e[q + 1] = kLin ? ex2_lin_from_biased(e[q + 1]) : ex2_approx(e[q + 1]);
  }
  if (kFp8) {
#pragma unroll
    for (int q = 0; q < 8; ++q) w[q] = merge_e4m3x4(e[4 * q], e[4 * q + 1], e[4 * q + 2], e[4 * q + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      w[q] = pack_bf16x2(e[2 * q], e[2 * q + 1]);
      add_f32x2(sum[q & 1], w[q] << 16, w[q] & 0xFFFF0000u);
    }
  }
}

// Group 0's threads bring both groups' results for their row together (`comb`: [66][128], shared memory nobody else uses by then).
__device__ __forceinline__ void merge_groups(float* comb, int g, int r, float& m, float& l, float (&o)[64]) {
  asm volatile("bar.sync 2, 256;" ::: "memory");
  if (g == 1) {
    comb[r] = m;
    comb[128 + r] = l;
#pragma unroll
    for (int d = 0; d < 64; ++d) comb[(2 + d) * 128 + r] = o[d];
  }
  asm volatile("bar.sync 2, 256;" ::: "memory");
  if (g == 0) {
    const float m1 = comb[r], top = fmaxf(m, m1);
    const float a0 = ex2_approx(m - top), a1 = ex2_approx(m1 - top);
    l = l * a0 + comb[128 + r] * a1;
    m = top;
#pragma unroll
    for (int d = 0; d < 64; ++d) o[d] = o[d] * a0 + comb[(2 + d) * 128 + r] * a1;
  }
}

// kHelped: the end of a piece, for the softmax warps.  Reads O, brings the groups' results together, asks for the next piece's
// query rows and hands the finished rows on.  A function of its own, because what it works with (addresses, the places of pieces)
// would otherwise be kept in registers, or spilled, through the loop over the tiles.
__device__ __noinline__ int end_piece(const AttnArgs& a, uint8_t* smem, uint32_t tmem_o, int piece, bool any, float m) {
  using L = AttnSmem<true>;
  AttnBars* b = reinterpret_cast<AttnBars*>(smem + L::kBarOff);
  volatile int* abort_flag = &b->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = (warp - 4) >> 2, r = (warp & 3) * 32 + lane;
  const KeyShares kr(a, *const_cast<volatile int*>(&b->tiles), kHelperCost);
  const int item = kr.first_item + piece;
  const Piece done = kr.at(item), next = kr.at(item + 1);
  int q0 = 0, qh = 0, kvh = 0;
  QueryTile q;
  if (next.n > 0) {
    next.place(a, q0, qh, kvh);
    q.request_angles(a, q0);
    q.request(a, q0, qh);
  }
  float o[64];
  float l = 0.f;
#pragma unroll
  for (int d = 0; d < 64; ++d) o[d] = 0.f;
  mbar_wait_warp(smem_u32(&b->o_final[g]), piece & 1, abort_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN);
  if (any) {
    tc_fence_after();
    read_o<true>(tmem_o, o, l);
  }
  // The next piece's K and V are on their way into the rings, so the groups meet in memory of their own.
  merge_groups(reinterpret_cast<float*>(smem + L::kCombOff), g, r, m, l, o);
  const bool good = *abort_flag == 0;
  if (g == 1 && r == 0) b->tile_shift = next.tile0 - (piece + 1) * done.n;  // (read again behind q_ready of the next piece)
  if (next.n > 0) q.stage<true>(smem + L::kQOff, b->tm, &b->q_ready);
  if (g == 0) kr.finish(a, done, r, good, m, l, o, &b->exchange);
  return next.n;
}

template <bool kFp8, int kSplit, bool kLin>
__global__ void __launch_bounds__(kAttnThreads, 1)
owl_attn_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ AttnArgs a) {
  using L = AttnSmem<kFp8, kSplit == kSplitCluster>;
  constexpr int kKS = L::kKStages, kVS = L::kVStages;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kIdescS = kFp8 ? umma_idesc(0, 0, 128, kKeyTile) : umma_idesc(1, 1, 128, kKeyTile);
  constexpr uint32_t kIdescPV = kFp8 ? umma_idesc(0, 0, 128, L::kRows) : umma_idesc(1, 1, 128, L::kRows);
  // P = 2^(kPShift + score - m) with m the maximum the row was last rescaled to; m is raised (and O
  // rescaled) only when a tile's maximum exceeds it by more than kSlack, so P <= 2^(kPShift + kSlack):
  // 256, inside the range of e4m3 and bf16.  (Not rounded to a whole number: the key that m came from, often the one that counts
  // most, then has a probability of exactly 2^kPShift.  A whole m doubled the e4m3 error of rows with few large scores.)
  constexpr float kPShift = kFp8 ? 5.0f : 0.0f;
  constexpr float kSlack = kFp8 ? 3.0f : 8.0f;
  constexpr uint32_t kGroupCols = 256;  // TMEM columns per softmax group: S at 0, O (80 | 64 columns) at 128, P (32 | 64) behind it
  constexpr uint32_t kOCol = 128, kPCol = kOCol + L::kRows;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  AttnBars* bars = reinterpret_cast<AttnBars*>(smem + L::kBarOff);
  volatile int* abort_flag = &bars->abort_flag;
  volatile int* drain_flag = &bars->drain_flag;
  // for single threads, which stop when a wait runs out
  auto wait = [&](uint64_t& bar, uint32_t parity) { return mbar_wait(smem_u32(&bar), parity, abort_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN); };
  // for whole warps, which go on: what they work out then is not written (abort_flag)
  auto wait_warp = [&](uint64_t& bar, uint32_t parity) { mbar_wait_warp(smem_u32(&bar), parity, abort_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN); };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int q0 = blockIdx.x * kQTile;
  int qh = blockIdx.y;
  int kvh = qh / a.gqa;

  if (warp == 0) {  // (a barrier per lane: one thread took 700 cycles for all of them)
    for (unsigned i = lane; i < offsetof(AttnBars, tmem_slot) / 8; i += 32)
      mbar_init(smem_u32(reinterpret_cast<uint64_t*>(bars) + i), i >= offsetof(AttnBars, s_free) / 8 && i < offsetof(AttnBars, pv_done) / 8 ? 4 : i == offsetof(AttnBars, q_ready) / 8 ? 8 : 1);
    if (lane == 0) {
      *abort_flag = 0;
      *drain_flag = 0;
    }
    fence_barrier_init();
  } else if (threadIdx.x == 96) {
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (kFp8) {  // rows of ones under every V^T tile (16 rows x 128 bytes each)
    for (int i = threadIdx.x; i < kVS * 128; i += kAttnThreads)  // 128 x 16 bytes per tile
      *reinterpret_cast<uint4*>(smem + L::kVOff + (i >> 7) * L::kVBytes + 64 * 128 + (i & 127) * 16) = make_uint4(0x38383838u, 0x38383838u, 0x38383838u, 0x38383838u);
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&bars->tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_slot;
  if (kSplit == kSplitCluster) cluster_arrive();  // this CTA is there (waited for before anyone pushes to it)

  // Everything above touched only this CTA's shared memory and TMEM, so it may run while the kernels before this one in the stream are
  // still at work; everything below reads what they wrote.
  grid_dep_launch();
  grid_dep_wait();

  // The table, the query rows with their angles and the frame counter are asked for at once, so that the first K tile is two trips to L2
  // away.
  QueryTile q;
  if (kSplit != kHelped && warp >= 4) {
    q.request(a, q0, qh);
    q.request_angles(a, q0);
  }
  int seg[6];
  const int nseg = request_table(a, seg);
  const int frame_t = *after_wait(a.frame_t);
  int n_tiles = load_table(a, nseg, seg);
  int tile0 = 0;
  KeyShares kr;
  Piece pc;
  if (kSplit == kHelped) {
    kr = KeyShares(a, n_tiles, kHelperCost);
    pc = kr.first();
    pc.place(a, q0, qh, kvh);
    tile0 = pc.tile0;
    n_tiles = kr.all_tiles();
    if (warp >= 4 && pc.n > 0) {
      q.request_angles(a, q0);
      q.request(a, q0, qh);
    }
  }
  // key splits: this CTA's share of the tiles
  const int n_splits = kSplit == kSplitWorkspace || kSplit == kSplitCluster ? static_cast<int>(gridDim.z) : 1;
  if (kSplit == kSplitWorkspace || kSplit == kSplitCluster) {
    tile0 = static_cast<int>(blockIdx.z) * n_tiles / n_splits;
    n_tiles = static_cast<int>(blockIdx.z + 1) * n_tiles / n_splits - tile0;
  }
  // every segment a multiple of the tile (720p: 512 keys a bucket): no tile needs a mask, so none is looked up
  const bool whole = ((seg[1] | seg[3] | seg[5]) & (kKeyTile - 1)) == 0;

  if (warp < 4) {
    setmaxnreg_dec<kCtrlRegs>();
    if (warp == 3) {
      if (lane < 8) temporal_cos_sin(frame_t, lane, bars->tm);
      if (lane == 8) {
#pragma unroll
        for (int i = 0; i < 6; ++i) bars->seg[i] = seg[i];
        bars->tiles = kr.tiles;
        bars->tile_shift = tile0;
      }
      __syncwarp();
      asm volatile("bar.arrive 4, 288;" ::: "memory");  // groups 0 and 1 wait for it
    } else if (warp == 0) {
      // ---------------- TMA producer: K(t), then V(t - 2), in the order in which they are used
      if (elect_one()) {
        int tile = tile0;  // within the item
        int row[3] = {0, 0, 0}, head[3] = {0, 0, 0};  // of tiles t, t - 1, t - 2
        int k_issued = 0, v_issued = 0;
        for (int t = 0; t < n_tiles + 2; ++t) {
          if (t < n_tiles) {
            if (kSplit == kHelped && tile == pc.tile0 + pc.n) {  // on to the next item
              kr.next(pc);
              tile = pc.tile0;
              pc.place(a, q0, qh, kvh);
            }
            int valid;
            locate_tile(seg, tile, row[0], valid);
            head[0] = kvh;
            ++tile;
            const int s = t % kKS;
            if (!wait(bars->k_empty[s], ((t / kKS) & 1) ^ 1)) break;
            const uint32_t fb = smem_u32(&bars->k_full[s]);
            mbar_arrive_expect_tx(fb, L::kKBytes);
            tma_load_2d(smem_u32(smem + L::kKOff + s * L::kKBytes), &tmK, fb, 0, kvh * a.capacity + row[0]);
            k_issued = t + 1;
          }
          if (t >= 2) {
            const int v = t - 2, s = v % kVS;
            if (!wait(bars->v_empty[s], ((v / kVS) & 1) ^ 1)) break;
            const uint32_t fb = smem_u32(&bars->v_full[s]);
            mbar_arrive_expect_tx(fb, L::kEs * 64 * 128);
            uint8_t* st = smem + L::kVOff + s * L::kVBytes;
            tma_load_2d(smem_u32(st), &tmV, fb, row[2], head[2] * 64);
            if (!kFp8) tma_load_2d(smem_u32(st + L::kVTile), &tmV, fb, row[2] + 64, head[2] * 64);
            v_issued = v + 1;
          }
          row[2] = row[1]; row[1] = row[0];
          head[2] = head[1]; head[1] = head[0];
        }
        if (*abort_flag) {
          // Giving up: let the copies already in flight land before this CTA's memory goes away.
          for (int j = max(0, k_issued - kKS); j < k_issued; ++j)
            mbar_wait(smem_u32(&bars->k_full[j % kKS]), (j / kKS) & 1, drain_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN);
          for (int j = max(0, v_issued - kVS); j < v_issued; ++j)
            mbar_wait(smem_u32(&bars->v_full[j % kVS]), (j / kVS) & 1, drain_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN);
        } else {
          // Tail: see the last stage releases land before the CTA can exit.
          for (int j = max(0, n_tiles - kKS); j < n_tiles; ++j)
            if (!wait(bars->k_empty[j % kKS], (j / kKS) & 1)) break;
          for (int j = max(0, n_tiles - kVS); j < n_tiles; ++j)
            if (!wait(bars->v_empty[j % kVS], (j / kVS) & 1)) break;
        }
      }
    } else {
      // ---------------- MMA issuers: warp 1 serves softmax group 0 (even tiles), warp 2 group 1 (odd tiles).
      // Per group: S(i + 1) goes to the group's S columns as soon as the group has copied S(i) into its registers; once the group has
      // written P(i), O += P(i) V(i) accumulates in the group's O columns.
      const int g = warp - 1;
      // A piece of work is a run of tiles of one item: all that this CTA has, or (kHelped) one after the other.  Tiles are counted
      // over the pieces, so stages and barrier phases run on; only O starts anew.
      if (elect_one()) {
        const uint32_t q_addr = smem_u32(smem + L::kQOff), k0_addr = smem_u32(smem + L::kKOff), v0_addr = smem_u32(smem + L::kVOff);
        const uint32_t tmem_sg = tmem_base + g * kGroupCols, tmem_og = tmem_sg + kOCol, tmem_pg = tmem_sg + kPCol;
        bool ok = true;
        auto issue_s = [&](int i) {
          const int j = 2 * i + g, s = j % kKS;
          if (!wait(bars->k_full[s], (j / kKS) & 1)) return false;
          if (i > 0 && !wait(bars->s_free[g], (i - 1) & 1)) return false;
          tc_fence_after();
          const uint32_t k_addr = k0_addr + s * L::kKBytes;
          if (kFp8) {
            const uint64_t qd = umma_desc_k_sw64(q_addr), kd = umma_desc_k_sw64(k_addr);
#pragma unroll
            for (int k = 0; k < 2; ++k) umma_f8(tmem_sg, qd + 2 * k, kd + 2 * k, kIdescS, k > 0);
          } else {
            const uint64_t qd = umma_desc_k_sw128(q_addr), kd = umma_desc_k_sw128(k_addr);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_f16(tmem_sg, qd + 2 * k, kd + 2 * k, kIdescS, k > 0);
          }
          umma_commit(smem_u32(&bars->s_full[g]));
          umma_commit(smem_u32(&bars->k_empty[s]));
          return true;
        };
        int i0 = 0, end = kSplit == kHelped ? pc.n : n_tiles, i1 = group_tiles(end, g);  // the group's tiles of the piece
        for (int piece = 0; ok && (kSplit == kHelped ? pc.n > 0 : piece == 0); ++piece) {
          if (kSplit == kHelped || i0 < i1) ok = wait(bars->q_ready, piece & 1);
          if (i0 < i1) ok = ok && issue_s(i0);
          for (int i = i0; i < i1 && ok; ++i) {
            if (i + 1 < i1) ok = issue_s(i + 1);
            const int j = 2 * i + g, s = j % kVS;
            ok = ok && wait(bars->v_full[s], (j / kVS) & 1) && wait(bars->p_full[g], i & 1);
            if (!ok) break;
            tc_fence_after();
            const uint64_t vd = umma_desc_k_sw128(v0_addr + s * L::kVBytes);
            if (kFp8) {
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f8_ts(tmem_og, tmem_pg + 8 * k, vd + 2 * k, kIdescPV, i > i0 || k > 0);
            } else {
              const uint64_t vd1 = umma_desc_k_sw128(v0_addr + s * L::kVBytes + L::kVTile);
#pragma unroll
              for (int k = 0; k < 8; ++k) umma_f16_ts(tmem_og, tmem_pg + 8 * k, (k < 4 ? vd : vd1) + 2 * (k & 3), kIdescPV, i > i0 || k > 0);
            }
            umma_commit(smem_u32(&bars->pv_done[g]));
            umma_commit(smem_u32(&bars->v_empty[s]));
          }
          if (ok && late(g == 0 && blockIdx.x == gridDim.x - 1 && blockIdx.z == gridDim.z - 1, abort_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN)) ok = false;
          // pv_done flips once per tile, so its parity cannot tell "all finished" from "two still in flight"; the end of the
          // accumulation has a barrier of its own
          if (ok && (kSplit == kHelped || i0 < i1)) umma_commit(smem_u32(&bars->o_final[g]));
          if (kSplit == kHelped) {
            kr.next(pc);
            i0 = i1;
            end += pc.n;
            i1 = group_tiles(end, g);
          }
        }
      }
    }
  } else {
    setmaxnreg_inc<kSoftmaxRegs>();
    // ---------------- softmax groups: one query row per thread, group g takes tiles j = 2 i + g
    const int g = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int t = q0 + r;
    const bool row_ok = t < a.tpf;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + g * kGroupCols + lane_addr;  // this thread's row of the group's S,
    const uint32_t tmem_o = tmem_s + kOCol, tmem_p = tmem_s + kPCol;  // ... of its O and of its P

    asm volatile("bar.sync 4, 288;" ::: "memory");  // the temporal angles
    if (kSplit != kHelped || pc.n > 0) q.stage<kFp8>(smem + L::kQOff, bars->tm, &bars->q_ready);  // (else nothing was requested)
    int i0 = 0, i1 = group_tiles(kSplit == kHelped ? pc.n : n_tiles, g);  // the group's tiles of the piece, as the MMA warp counts them
    // What the end of a piece needs is worked out there from its number, so that it takes no registers in the loop.
    int end = pc.n;
    bool more = kSplit != kHelped || pc.n > 0;

    for (int piece = 0; more; ++piece) {
      if (kSplit == kHelped && piece > 0) {
        const KeyShares again(a, *const_cast<volatile int*>(&bars->tiles), kHelperCost);
        again.at(again.first_item + piece).place(a, q0, qh, kvh);
      }
      const float ks = a.k_scale ? __ldg(a.k_scale + kvh) : 1.0f;
      const float sl2 = ks * 0.125f * 1.4426950408889634f;  // scores -> log2 domain, 1/sqrt(64) folded in
      const uint64_t sl2_2 = pack_f32x2(sl2, sl2);
      float m_run = -1.0e30f, l_run = 0.f;  // bf16: the row sum, of the rounded probabilities
      for (int i = i0; i < i1; ++i) {
        wait_warp(bars->s_full[g], i & 1);
        tc_fence_after();
        int row, valid = kKeyTile;
        if (!whole) locate_tile(bars->seg, 2 * i + g + bars->tile_shift, row, valid);  // (the table is there: Q was staged after it)
        // the whole score row into registers; the S columns are then free for the next tile
        uint32_t sc[kKeyTile / 32][32];
#pragma unroll
        for (int c = 0; c < kKeyTile / 32; ++c) tmem_ld32(tmem_s + c * 32, sc[c]);
        // the wait names the loaded registers, so that nothing the compiler does with them (a move, a spill)
        // can be placed between a load and the wait, where they do not hold the scores yet
        tmem_wait_ld_into(sc[0]);
#pragma unroll
        for (int c = 1; c < kKeyTile / 32; ++c) tmem_loaded(sc[c]);
        tc_fence_before();
        warp_arrive(smem_u32(&bars->s_free[g]), lane);
        if (valid != kKeyTile) {  // last tile of a segment whose length is not a multiple of the tile
#pragma unroll
          for (int c = 0; c < kKeyTile / 32; ++c) mask_chunk(sc[c], c, valid);
        }
        float mx[4] = {-1.0e30f, -1.0e30f, -1.0e30f, -1.0e30f};
#pragma unroll
        for (int q = 0; q < kKeyTile / 2; ++q) mx[q & 3] = max3f(mx[q & 3], __uint_as_float(sc[q >> 4][2 * (q & 15)]), __uint_as_float(sc[q >> 4][2 * (q & 15) + 1]));
        const float m_tile = fmaxf(max3f(mx[0], mx[1], mx[2]), mx[3]) * sl2;
        if (i == i0) {
          m_run = m_tile;
        } else if (const bool jump = m_tile > m_run + kSlack; __any_sync(0xffffffffu, jump)) {
          wait_warp(bars->pv_done[g], (i - 1) & 1);  // O may be rescaled only when PV(i - 1) has finished
          const float before = m_run;
          if (jump) m_run = m_tile;
          const float alpha = ex2_approx(before - m_run);
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t oo[16];
            tmem_ld16(tmem_o + c * 16, oo);
            tmem_wait_ld_into(oo);
#pragma unroll
            for (int q = 0; q < 16; ++q) oo[q] = __float_as_uint(__uint_as_float(oo[q]) * alpha);
            tmem_st16(tmem_o + c * 16, oo);
          }
          if (kFp8) {
            uint32_t lsum = tmem_ld1(tmem_o + 64);
            tmem_wait_ld();
            tmem_loaded(lsum);
            tmem_st1(tmem_o + 64, __float_as_uint(__uint_as_float(lsum) * alpha));
          } else {
            l_run *= alpha;
          }
          tmem_wait_st();
        }
        const float nshift = kPShift - m_run;
        const uint64_t nshift_2 = pack_f32x2(nshift, kLin ? nshift + kLinMagic : nshift);
        uint32_t pw[kFp8 ? 1 : 2][32];
        uint64_t sum[2] = {0, 0};
#pragma unroll
        for (int c = 0; c < kKeyTile / 32; ++c) p_chunk<kFp8, kLin>(sc[c], sl2_2, nshift_2, kFp8 ? pw[0] + c * 8 : pw[c >> 1] + (c & 1) * 16, sum);
        if (!kFp8) l_run += sum_f32x2(sum[0], sum[1]);
        if (i > 0) wait_warp(bars->pv_done[g], (i - 1) & 1);  // PV(i - 1) has read the P before: long ago, as a rule
        tmem_st32(tmem_p, pw[0]);
        if constexpr (!kFp8) tmem_st32(tmem_p + 32, pw[1]);
        tmem_wait_st();
        tc_fence_before();
        warp_arrive(smem_u32(&bars->p_full[g]), lane);
      }
      if constexpr (kSplit == kHelped) {
        const int n = end_piece(a, smem, tmem_o, piece, i0 < i1, m_run);
        end += n;
        i0 = i1;
        i1 = group_tiles(end, g);
        more = n > 0;
        continue;
      }
      more = false;

      float o[64];
#pragma unroll
      for (int d = 0; d < 64; ++d) o[d] = 0.f;
      if (i0 < i1) {
        wait_warp(bars->o_final[g], 0);
        tc_fence_after();
        read_o<kFp8>(tmem_o, o, l_run);
      }
      if constexpr (kSplit == kSplitCluster) {
        // Both groups of every CTA of the cluster hand their rows to the CTA that writes them.  (Pushed with a row's 272 bytes together and
        // between two cluster barriers, 32 rows an instruction, the end took 10600 of a launch's 23700 cycles at 360p; laid out per receiver
        // and copied in bulk 7900.)
        const int S = static_cast<int>(gridDim.z), rows = merge_rows(S), cta = static_cast<int>(blockIdx.z);
        const int me = static_cast<int>(threadIdx.x) - 128;
        const float4* parts = reinterpret_cast<const float4*>(smem + L::kCombOff);
        cluster_wait();  // (long since)
        {
          const uint32_t base = map_to_cta(smem_u32(parts), r / rows);
          auto push = [&](int u, float x, float y, float z, float w) {
            st_dsmem_v4(base + 16u * merge_unit(2 * cta + g, u, r % rows, rows), __float_as_uint(x), __float_as_uint(y), __float_as_uint(z), __float_as_uint(w));
          };
#pragma unroll
          for (int u = 0; u < 16; ++u) push(u, o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
          // where one of this CTA's waits ran out, the rows that its results belong to are not written by any CTA of the cluster
          push(16, m_run, l_run, *abort_flag != 0 ? 1.0f : 0.0f, 0.0f);
        }
        cluster_arrive();
        const float vs = a.v_scale ? __ldg(a.v_scale + kvh) : 1.0f;
        cluster_wait();
        for (int n = me; n < rows * 8; n += 256) {  // outputs d0 .. d0 + 3 and 32 more of a row per thread
          const int rl = n >> 3, u = n & 7, d0 = 4 * u, rr = cta * rows + rl;
          if (rr >= kQTile || q0 + rr >= a.tpf) continue;
          float4 head[16];  // m, row sum, lost
          float m = -1.0e30f, lost = 0.f;
#pragma unroll
          for (int q = 0; q < 16; ++q)
            if (q < 2 * S) head[q] = parts[merge_unit(q, 16, rl, rows)];
#pragma unroll
          for (int q = 0; q < 16; ++q)
            if (q < 2 * S) {
              m = fmaxf(m, head[q].x);
              lost += head[q].z;
            }
          if (lost != 0.f) continue;
          float l = 0.f, e[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int q = 0; q < 16; ++q)
            if (q < 2 * S) {
              const float w = ex2_approx(head[q].x - m);
              l = fmaf(w, head[q].y, l);
              const float4 x = parts[merge_unit(q, u, rl, rows)], y = parts[merge_unit(q, u + 8, rl, rows)];
              e[0] = fmaf(w, x.x, e[0]); e[1] = fmaf(w, x.y, e[1]); e[2] = fmaf(w, x.z, e[2]); e[3] = fmaf(w, x.w, e[3]);
              e[4] = fmaf(w, y.x, e[4]); e[5] = fmaf(w, y.y, e[5]); e[6] = fmaf(w, y.z, e[6]); e[7] = fmaf(w, y.w, e[7]);
            }
          const float inv = l > 0.f ? vs / l : 0.f;
#pragma unroll
          for (int d = 0; d < 8; ++d) e[d] *= inv;
          const size_t at = static_cast<size_t>(q0 + rr) * a.o_row + static_cast<size_t>(qh) * a.o_head + d0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t w0 = pack_bf16x2(e[4 * h], e[4 * h + 1]), w1 = pack_bf16x2(e[4 * h + 2], e[4 * h + 3]);
            *reinterpret_cast<uint2*>(a.out + at + 32 * h) = make_uint2(w0, w1);
            if (a.out_q != nullptr) *reinterpret_cast<uint32_t*>(a.out_q + at + 32 * h) = pack_e4m3x4(bf16lo(w0), bf16hi(w0), bf16lo(w1), bf16hi(w1));
          }
        }
      } else if constexpr (kSplit == kUnsplit) {
        // The groups exchange halves: group g finishes outputs 32 g .. 32 g + 31 of the row.  (Tensor work and TMA traffic are finished
        // for both behind the first barrier.)
        float* comb = reinterpret_cast<float*>(smem + L::kCombOff);  // [group][34][128]
        asm volatile("bar.sync 2, 256;" ::: "memory");
        float* give = comb + g * (34 * 128) + r;
        give[0] = m_run;
        give[128] = l_run;
        float h[32];
#pragma unroll
        for (int d = 0; d < 32; ++d) {
          give[(2 + d) * 128] = g == 0 ? o[32 + d] : o[d];
          h[d] = g == 0 ? o[d] : o[32 + d];
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (row_ok && *abort_flag == 0) {
          const float* take = comb + (1 - g) * (34 * 128) + r;
          const float m1 = take[0], l1 = take[128];
          const float m = fmaxf(m_run, m1);
          const float a0 = ex2_approx(m_run - m), a1 = ex2_approx(m1 - m);
          const float l = __fadd_rn(__fmul_rn(l_run, a0), __fmul_rn(l1, a1));  // the same in both groups
          const float vs = a.v_scale ? __ldg(a.v_scale + kvh) : 1.0f;
          const float inv = l > 0.f ? vs / l : 0.f;
          const float s0 = a0 * inv, s1 = a1 * inv;
#pragma unroll
          for (int d = 0; d < 32; ++d) h[d] = h[d] * s0 + take[(2 + d) * 128] * s1;
          write_out(a, static_cast<size_t>(t) * a.o_row + static_cast<size_t>(qh) * a.o_head + g * 32, h);
        }
      } else if constexpr (kSplit == kSplitWorkspace) {
        // Keys shared with other CTAs: the row's part, both groups brought to a common maximum and not yet divided by the row sum, goes
        // to the workspace, and the CTA that draws the last ticket sums them.
        merge_groups(reinterpret_cast<float*>(smem + L::kCombOff), g, r, m_run, l_run, o);
        if (g == 0) {
          const bool good = *abort_flag == 0;
          const int it = qh * gridDim.x + blockIdx.x;  // (head, query tile)
          float* mine = a.partials + (static_cast<size_t>(it) * n_splits + blockIdx.z) * kPartial;
          mine[r] = m_run;
          mine[128 + r] = l_run;
#pragma unroll
          for (int d = 0; d < 64; ++d) mine[(2 + d) * 128 + r] = o[d];
          __threadfence();
          asm volatile("bar.sync 3, 128;" ::: "memory");
          if (r == 0) {
            const int was = atomicAdd(a.tickets + it, *abort_flag == 0 ? 1 : kLostTicket + 1);
            const bool mine_is_last = (was & (kLostTicket - 1)) == n_splits - 1;
            if (mine_is_last) a.tickets[it] = 0;  // ready for the next launch
            *const_cast<volatile int*>(&bars->exchange) = mine_is_last && was < kLostTicket;
          }
          asm volatile("bar.sync 3, 128;" ::: "memory");
          if (*const_cast<volatile int*>(&bars->exchange) != 0 && good && row_ok) {
            __threadfence();
            // sum the shares in order of z: the result does not depend on which CTA came last
            const float* part = a.partials + static_cast<size_t>(it) * n_splits * kPartial;
            float m = -1.0e30f;
            for (int z = 0; z < n_splits; ++z) m = fmaxf(m, __ldcg(part + z * kPartial + r));
            float l = 0.f;
#pragma unroll
            for (int d = 0; d < 64; ++d) o[d] = 0.f;
            for (int z = 0; z < n_splits; ++z) {
              const float* pz = part + z * kPartial;
              const float w = ex2_approx(__ldcg(pz + r) - m);
              l = fmaf(w, __ldcg(pz + 128 + r), l);
#pragma unroll
              for (int d = 0; d < 64; ++d) o[d] = fmaf(w, __ldcg(pz + (2 + d) * 128 + r), o[d]);
            }
            KeyShares::write_row(a, t, qh, kvh, l, o);
          }
        }
      }
    }
    if (kSplit == kHelped && kr.tiles == 0) KeyShares::write_zeros(a, r, g, 2);
  }

  if (kSplit == kSplitCluster && warp < 4) {  // the softmax warps' barriers
    __syncwarp();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace qb

namespace qb {
// e4m3 probabilities: 0 = every second exponential on the FMA pipe (ex2_lin_from_biased), 1 = all on the special-function unit
static int g_attn_exact_exp = [] {
  const char* e = getenv("QB_ATTN_EXACT_EXP");
  return (e != nullptr && e[0] == '1') ? 1 : 0;
}();
}  // namespace qb

using namespace qb;

extern "C" int32_t qb_set_attn_exact_exp(int32_t on) {
  const int32_t was = g_attn_exact_exp;
  g_attn_exact_exp = on ? 1 : 0;
  return was;
}

// How many CTAs share the keys of one (query tile, head).  One when the grid already fills most of the GPU
// (720p: 4 query tiles x 32 heads); otherwise as many as it takes to reach the SM count, while every
// share keeps a few key tiles (360p: 1 x 32 -> 4 shares; a tensor-parallel rank with 2 KV heads: 8).
static int attn_key_splits(const qb_attn_params* p) {
  if (p->kv_splits > 0) return p->kv_splits;
  const int tpf = p->H_spatial * p->W_spatial;
  const int items = ((tpf + kQTile - 1) / kQTile) * p->n_kv_heads * p->gqa_ratio;
  const int tiles = ((p->num_buckets + 1) * (tpf / (p->quilt_factor > 0 ? p->quilt_factor : 1)) + kKeyTile - 1) / kKeyTile;  // at most
  int n = num_sms() / (items > 0 ? items : 1);
  if (n > tiles / 3) n = tiles / 3;
  if (n > 8) n = 8;
  return n < 2 ? 1 : n;
}

// Whether the CTAs that the items leave over help with their keys (owned_tiles, at the longest history; the kernel decides again for
// the keys that are valid).
static bool attn_helped(const qb_attn_params* p, int splits) {
  if (p->kv_splits != 0 || splits != 1) return false;
  const int tpf = p->H_spatial * p->W_spatial, sms = num_sms();
  const long long items = static_cast<long long>((tpf + kQTile - 1) / kQTile) * p->n_kv_heads * p->gqa_ratio;
  const long long tiles = (static_cast<long long>(p->num_buckets + 1) * (tpf / (p->quilt_factor > 0 ? p->quilt_factor : 1)) + kKeyTile - 1) / kKeyTile;  // at most
  return 2 * items > sms && items < sms && tiles < (1 << 24) && owned_tiles(static_cast<int>(items), sms, static_cast<int>(tiles), kHelperCost) < tiles;
}

static cudaLaunchConfig_t attn_config(dim3 grid, int smem_bytes, cudaStream_t st, cudaLaunchAttribute (&attr)[2]) {  // grid.z = CTAs of a cluster
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kAttnThreads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = grid.z;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_dependent_launch ? 2 : 1;
  return cfg;
}

// `splits` CTAs share the keys of each (query tile, head), as a cluster of up to 8 CTAs where the chip holds that many clusters at
// once (B200: 15 of 8 CTAs, 33 of 4, 74 of 2); a wish for more is cut down to what it holds, a number that the caller forced goes
// through the workspace instead.  bf16 comes here for its key splits: where there are none, and with helpers, it goes to the three-group kernel.
template <bool kFp8, bool kLin>
static int32_t launch_attn(const CUtensorMap& tmK, const CUtensorMap& tmV, const AttnArgs& a, int Hq, int splits, bool forced, bool helped, cudaStream_t st) {
  constexpr int kSmem = AttnSmem<kFp8>::kTotal, kClusterSmem = AttnSmem<kFp8, true>::kTotal;
  if constexpr (kFp8) if (helped) {
    static std::atomic<unsigned long long> done{0};
    const int32_t rc = configure_smem(owl_attn_kernel<kFp8, kHelped, kLin>, kSmem, done);
    if (rc != QB_OK) return rc;
    return launch_dep("owl_attn kernel", owl_attn_kernel<kFp8, kHelped, kLin>, dim3(num_sms()), dim3(kAttnThreads), kSmem, st, tmK, tmV, a);
  }
  const unsigned q_tiles = (a.tpf + kQTile - 1) / kQTile;
  const int items = static_cast<int>(q_tiles) * Hq;
  int cluster = splits > 8 ? (forced ? 1 : 8) : splits;
  if (cluster > 1) {
    static std::atomic<unsigned long long> done{0};
    static std::atomic<int> held[9];  // clusters of this many CTAs that run at once (0 = not asked yet)
    const int32_t rc = configure_smem(owl_attn_kernel<kFp8, kSplitCluster, kLin>, kClusterSmem, done);
    if (rc != QB_OK) return rc;
    cudaLaunchAttribute attr[2];
    while (cluster > 1) {
      int n = held[cluster].load(std::memory_order_relaxed);
      if (n == 0) {
        const cudaLaunchConfig_t cfg = attn_config(dim3(q_tiles, Hq, cluster), kClusterSmem, st, attr);
        if (cudaOccupancyMaxActiveClusters(&n, owl_attn_kernel<kFp8, kSplitCluster, kLin>, &cfg) != cudaSuccess || n <= 0) {
          cudaGetLastError();
          n = 1;
        }
        held[cluster].store(n, std::memory_order_relaxed);
      }
      if (items <= n) break;
      cluster = forced ? 1 : cluster - 1;
    }
    if (cluster > 1) {
      const cudaLaunchConfig_t cfg = attn_config(dim3(q_tiles, Hq, cluster), kClusterSmem, st, attr);
      const cudaError_t e = cudaLaunchKernelEx(&cfg, owl_attn_kernel<kFp8, kSplitCluster, kLin>, tmK, tmV, a);
      ++g_launch_count;
      if (e != cudaSuccess) return fail(QB_ERR_LAUNCH, "owl_attn kernel (cluster of %d): %s", cluster, cudaGetErrorString(e));
      return QB_OK;
    }
  }
  if (splits > 1 && forced) {
    static std::atomic<unsigned long long> done{0};
    const int32_t rc = configure_smem(owl_attn_kernel<kFp8, kSplitWorkspace, kLin>, kSmem, done);
    if (rc != QB_OK) return rc;
    return launch_dep("owl_attn kernel", owl_attn_kernel<kFp8, kSplitWorkspace, kLin>, dim3(q_tiles, Hq, splits), dim3(kAttnThreads), kSmem, st, tmK, tmV, a);
  }
  if constexpr (kFp8) {
    static std::atomic<unsigned long long> done{0};
    const int32_t rc = configure_smem(owl_attn_kernel<kFp8, kUnsplit, kLin>, kSmem, done);
    if (rc != QB_OK) return rc;
    return launch_dep("owl_attn kernel", owl_attn_kernel<kFp8, kUnsplit, kLin>, dim3(q_tiles, Hq), dim3(kAttnThreads), kSmem, st, tmK, tmV, a);
  } else {
    return launch_attn3(tmK, tmV, a, Hq, helped, st);
  }
}

// The tickets take a fixed area at the start of the workspace (4096 (query tile, head) items; more only for a
// geometry that has more), so that calls of different geometries that share a workspace agree on where the
// tickets end: one call's partial results never land on tickets that another call expects to find zero.
static size_t attn_ticket_bytes(const qb_attn_params* p) {
  const int tpf = p->H_spatial * p->W_spatial;
  const size_t need = round_up(static_cast<size_t>((tpf + kQTile - 1) / kQTile) * p->n_kv_heads * p->gqa_ratio * sizeof(int), 1024);
  return need > (16u << 10) ? need : (16u << 10);
}

static bool attn_sizes_ok(const qb_attn_params* p) {
  return p != nullptr && p->H_spatial > 0 && p->W_spatial > 0 && p->n_kv_heads > 0 && p->gqa_ratio > 0 && p->num_buckets > 0;
}

extern "C" size_t qb_owl_attn_workspace_bytes(const qb_attn_params* p) {
  if (!attn_sizes_ok(p)) return 0;
  const int n = attn_key_splits(p);
  if (n <= 1) return 0;
  const int tpf = p->H_spatial * p->W_spatial;
  const size_t items = static_cast<size_t>((tpf + kQTile - 1) / kQTile) * p->n_kv_heads * p->gqa_ratio;
  return attn_ticket_bytes(p) + items * n * (66 * 128) * sizeof(float);
}

extern "C" size_t qb_owl_attn_scratch_bytes(const qb_attn_params* p) {
  if (!attn_sizes_ok(p)) return 0;
  if (p->kv_splits > 0) return qb_owl_attn_workspace_bytes(p);  // splits of the kernel's own choice are clusters: no workspace
  if (!attn_helped(p, attn_key_splits(p))) return 0;
  return attn_ticket_bytes(p) + static_cast<size_t>(2 * num_sms()) * kPartial * sizeof(float);
}

extern "C" int32_t qb_owl_attn(const void* qkv, const void* K_cache, const void* Vt_cache, const int32_t* segments,
                               const int32_t* n_segments, const int32_t* frame_t, void* out, void* out_q, const float* rope_xy,
                               const qb_attn_params* p, void* workspace, size_t workspace_bytes, void* stream) {
  QB_REQUIRE(p != nullptr, QB_ERR_INVALID_ARG, "owl_attn: params are NULL");
  QB_REQUIRE(qkv && K_cache && Vt_cache && segments && n_segments && frame_t && out && rope_xy, QB_ERR_INVALID_ARG,
             "owl_attn: NULL pointer");
  QB_REQUIRE(p->quilt_factor >= 1 && (p->H_spatial * p->W_spatial) % p->quilt_factor == 0, QB_ERR_INVALID_ARG,
             "owl_attn: quilt_factor %d does not divide H*W", p->quilt_factor);
  QB_REQUIRE(p->packed_qkv == 0 || p->packed_qkv == 1, QB_ERR_INVALID_ARG, "owl_attn: packed_qkv %d", p->packed_qkv);
  QB_REQUIRE(p->n_kv_heads > 0 && p->gqa_ratio > 0 && p->H_spatial > 0 && p->W_spatial > 0 && p->num_buckets > 0,
             QB_ERR_INVALID_ARG, "owl_attn: sizes must be positive");
  QB_REQUIRE(p->kv_dtype == QB_BF16 || p->kv_dtype == QB_E4M3, QB_ERR_INVALID_ARG, "owl_attn: kv_dtype %d", p->kv_dtype);
  QB_REQUIRE(p->compute_dtype == p->kv_dtype, QB_ERR_UNSUPPORTED,
             "owl_attn: compute_dtype must equal kv_dtype (bf16 cache + bf16 MMAs, or e4m3 cache + e4m3 MMAs)");
  QB_REQUIRE(p->max_segments >= 1, QB_ERR_INVALID_ARG, "owl_attn: max_segments %d", p->max_segments);
  const int tpf = p->H_spatial * p->W_spatial;
  // a quilted cache keeps tpf / quilt_factor tokens per frame (src/quark/kernels/owl_attn/spec.py:79-93); the queries
  // are all tpf tokens either way, and the segment table already counts cached rows
  const int cap = (p->num_buckets + 1) * (tpf / p->quilt_factor);
  QB_REQUIRE(cap % 16 == 0, QB_ERR_UNSUPPORTED, "owl_attn: capacity %d must be a multiple of 16", cap);
  QB_REQUIRE(aligned16(qkv) && aligned16(K_cache) && aligned16(Vt_cache) && aligned16(out) && aligned16(out_q) && aligned16(rope_xy), QB_ERR_ALIGN,
             "owl_attn: pointers must be 16-byte aligned");
  const bool fp8 = p->kv_dtype == QB_E4M3;
  const int es = fp8 ? 1 : 2;
  const int Hq = p->n_kv_heads * p->gqa_ratio;
  CUtensorMap tmK, tmV;
  int32_t rc = make_tmap_2d_sw(&tmK, K_cache, es, static_cast<uint64_t>(p->n_kv_heads) * cap, 64, kKeyTile, 64, fp8 ? 64 : 128);
  if (rc != QB_OK) return rc;
  rc = make_tmap_2d_sw(&tmV, Vt_cache, es, static_cast<uint64_t>(p->n_kv_heads) * 64, cap, 64, fp8 ? 128 : 64, 128);
  if (rc != QB_OK) return rc;

  AttnArgs a{};
  a.qkv = static_cast<const uint16_t*>(qkv);
  a.segments = segments; a.n_segments = n_segments; a.frame_t = frame_t;
  a.out = static_cast<uint16_t*>(out);
  a.out_q = static_cast<uint8_t*>(out_q);
  a.rope_xy = rope_xy;
  a.k_scale = p->k_scale; a.v_scale = p->v_scale;
  a.status = status_word();
  QB_REQUIRE(a.status != nullptr, QB_ERR_CUDA, "owl_attn: device status word unavailable");
  a.tpf = tpf;
  if (p->packed_qkv) {
    a.q_row = (Hq + 2 * p->n_kv_heads) * 64; a.q_head = 64; a.o_row = Hq * 64; a.o_head = 64;
  } else {
    a.q_row = 64; a.q_head = tpf * 64; a.o_row = 64; a.o_head = tpf * 64;
  }
  a.n_q_heads = Hq; a.gqa = p->gqa_ratio; a.capacity = cap; a.max_segments = p->max_segments;

  QB_REQUIRE(p->kv_splits >= 0 && p->kv_splits <= 16, QB_ERR_INVALID_ARG, "owl_attn: kv_splits %d", p->kv_splits);
  const int splits = attn_key_splits(p);
  if (splits > 1 && p->kv_splits > 0) {
    const size_t need = qb_owl_attn_workspace_bytes(p);
    QB_REQUIRE(workspace != nullptr && workspace_bytes >= need, QB_ERR_WORKSPACE, "owl_attn: %d key splits need a workspace of %zu bytes, %zu given",
               splits, need, workspace_bytes);
    QB_REQUIRE(aligned16(workspace), QB_ERR_ALIGN, "owl_attn: workspace must be 16-byte aligned");
    a.tickets = static_cast<int*>(workspace);
    a.partials = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + attn_ticket_bytes(p));
  }
  // the helpers want a workspace; a caller that gives none has one CTA per item
  const bool helped = attn_helped(p, splits) && workspace != nullptr && aligned16(workspace) && workspace_bytes >= qb_owl_attn_scratch_bytes(p);
  if (helped) {
    a.tickets = static_cast<int*>(workspace);
    a.partials = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + attn_ticket_bytes(p));
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool forced = p->kv_splits > 0;
  if (!fp8) return launch_attn<false, false>(tmK, tmV, a, Hq, splits, forced, helped, st);
  return g_attn_exact_exp ? launch_attn<true, false>(tmK, tmV, a, Hq, splits, forced, helped, st) : launch_attn<true, true>(tmK, tmV, a, Hq, splits, forced, helped, st);
}
