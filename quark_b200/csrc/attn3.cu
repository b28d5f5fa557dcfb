// owl_attn with three softmax groups and one accumulator: bf16 without key splits.  (e4m3, and key splits: attn.cu.)
//
// One CTA owns 128 query tokens of one Q head and walks the valid keys in tiles of 128, enumerated from the (start, length)
// segment table, so a masked bucket is never loaded.  512 threads:
//   warp 0        TMA producer: a ring of K tiles [128 keys x 64] and one of V^T tiles [64 x 128 keys] (+ 16 rows of ones)
//   warp 1        one thread issues O += P(j) V(j)          warp 2   one thread issues S(j) = Q K(j)^T
//   warp 3        sines and cosines of the temporal angles
//   warps 4-15    three softmax groups of four warps, one query row per thread; tile j belongs to group j mod 3
// TMEM: three S tiles of 128 columns and one accumulator O of 80 columns (64 outputs and the row sum, which the tensor core makes
// from 16 rows of ones under every V^T tile, of exactly the rounded P that is multiplied with V).  P(j) is written over the
// first columns of S(j) and is the A operand of O += P(j) V(j) from there, so that it takes no shared-memory bandwidth (in bf16, P
// written and read there took as many cycles as the exponentials) and no columns; S(j + 3) waits for PV(j).
//
// A softmax thread reads its row of S twice, 32 columns at a time: once for the maximum, once for P = 2^(score - m).
// m is the maximum that the row was last rescaled to, one value for all groups (m_row in shared memory): the groups settle m in
// the order of the tiles (`turn`, one barrier per group and lane quarter, passed on before the exponentials), and only where
// a tile's maximum exceeds m by more than kSlack does the warp wait for the PV before it and multiply O by 2^(m - m').
//
// What bounds it: the special-function unit (16 exponentials per clock and SM, 1024 cycles per tile; bf16 makes every fourth by a
// polynomial on the FMA pipe) and the trip from P(j) through PV(j) to S(j + 3), some 1200 cycles in which a group has nothing to do;
// hence three groups.  A loop with the same softmax instructions and nothing else takes 965 cycles per tile with three warps per
// scheduler (1180 with all exponentials on the special-function unit), this kernel 1330.  The K and V rings are separate and the loads
// run ahead of the S that runs ahead of the PV: with one ring a stage was held from S to PV, and the next K tiles came too late.
// 720p, us per launch: 56.8 -> 53.6 at 16 buckets, 211 -> 208 at 64, 404 -> 393 at 128, 792 -> 745 at 256.
// Tried and dropped: a whole m (P's rounding is then the same for every m, but the key that m came from no longer has a probability of
// exactly 1: 8 % more error); e4m3 in this form (44.5 against 42.0 us at 720p); key splits in this form (360p bf16 12.8 against 13.5 us,
// but one m for all keys of a CTA makes 2 % more error than one per group); kSlack 8 (52.4 against 53.8 us at 720p, 3 % more error
// where few keys count); kSlack 2, 1, 0 (84, 91, 100 us against 54 on rows that drift: a rescale waits for the PV before it).
// Error against 64 bits, this kernel over three accumulators with an m each (161fee8): keys N(0, 1) 1.000 (16 buckets) to 1.003 (128, one
// accumulator taking the rounding of all additions), rows where few keys count 0.997 to 1.007.
#include <atomic>

#include <cuda.h>

#include "attn_common.cuh"

namespace qb {

int num_sms();

constexpr int kA3Threads = 512;
constexpr int kGroups = 3;
constexpr int kSoftmaxThreads = kGroups * 128;
// setmaxnreg moves registers inside the pool the CTA was given at launch (512 threads x 128 registers): an increase waits until
// other warps of the CTA have released enough, so the budget below must close or the softmax warps would wait for ever.
constexpr int kA3LaunchRegs = 128;
constexpr int kA3CtrlRegs = 104;     // per thread, warps 0-3
constexpr int kA3SoftmaxRegs = 136;  // per thread, warps 4-15
static_assert(128 * kA3CtrlRegs + kSoftmaxThreads * kA3SoftmaxRegs <= kA3Threads * kA3LaunchRegs, "register budget of the CTA");
struct Attn3Smem {
  static constexpr int kStages = 5;                    // of each ring
  static constexpr int kQBytes = kQTile * 64 * 2;      // 16 KB
  static constexpr int kKBytes = kKeyTile * 64 * 2;    // 16 KB
  static constexpr int kVTile = kVRows * 128;          // one 128-byte-wide V^T tile incl. ones rows: 10 KB
  static constexpr int kVBytes = 2 * kVTile;           // keys 0-63, 64-127
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kQOff + kQBytes;
  static constexpr int kVOff = kKOff + kStages * kKBytes;
  static constexpr int kRowOff = kVOff + kStages * kVBytes;  // m of every query row
  static constexpr int kBarOff = kRowOff + kQTile * 4;
  static constexpr int kTotal = kBarOff + 640 + 1024;
  static_assert(kStages >= 4, "S runs three tiles ahead of PV");
  static_assert(kTotal <= 227 * 1024, "shared memory of one CTA");
};

// What follows the rings in shared memory.
struct Attn3Bars {
  uint64_t k_full[Attn3Smem::kStages], k_empty[Attn3Smem::kStages], v_full[Attn3Smem::kStages], v_empty[Attn3Smem::kStages];
  uint64_t s_full[kGroups];   // S(j) is in TMEM
  uint64_t p_full[kGroups];   // P(j) is in TMEM, O is rescaled
  uint64_t pv_done[kGroups];  // O += P(j) V(j) has finished
  uint64_t turn[kGroups][4];  // m of the rows of a lane quarter is settled for the tile before
  uint64_t o_final;           // every PV of a piece has finished
  uint64_t q_ready;
  uint32_t tmem_slot;
  int abort_flag, drain_flag, exchange;
  float tm[16];  // cosines and sines of the temporal angles
  int seg[6];    // the segment table, for tiles that need a mask: tile j of the CTA is tile j + tile_shift of the table
  int tiles, tile_shift;  // kHelped: tiles of an item
};
static_assert(sizeof(Attn3Bars) <= 640, "kBarOff + 640");

// Maximum over a row of S (128 columns from `ts` on), read from the last chunk of 32 columns to the first, which stays in s0.
template <bool kMasked>
__device__ __forceinline__ float row_max(uint32_t ts, int valid, uint32_t (&s0)[32]) {
  uint32_t s1[32];
  float mx[4] = {-1.0e30f, -1.0e30f, -1.0e30f, -1.0e30f};
  tmem_ld32(ts + 96, s1);
#pragma unroll
  for (int c = 3; c >= 0; --c) {
    uint32_t (&s)[32] = (c & 1) ? s1 : s0;
    tmem_wait_ld_into(s);
    if (c > 0) tmem_ld32(ts + (c - 1) * 32, (c & 1) ? s0 : s1);
    if (kMasked) mask_chunk(s, c, valid);
#pragma unroll
    for (int q = 0; q < 16; ++q) mx[q & 3] = max3f(mx[q & 3], __uint_as_float(s[2 * q]), __uint_as_float(s[2 * q + 1]));
  }
  return fmaxf(max3f(mx[0], mx[1], mx[2]), mx[3]);
}

// The row of probabilities 2^(score * sl2 + nshift), rounded, over the first columns of S.  s0 holds the scores of the first chunk.
template <bool kMasked>
__device__ __forceinline__ void row_exp(uint32_t ts, int valid, float sl2, float nshift, uint32_t (&s0)[32]) {
  uint32_t s1[32];
  const uint64_t sl2_2 = pack_f32x2(sl2, sl2), nshift_2 = pack_f32x2(nshift, nshift);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t (&s)[32] = (c & 1) ? s1 : s0;
    if (c > 0) {
      tmem_wait_ld_into(s);
      if (kMasked) mask_chunk(s, c, valid);
    }
    if (c < 3) tmem_ld32(ts + (c + 1) * 32, (c & 1) ? s0 : s1);
    uint32_t w[16];
#pragma unroll
    for (int q = 0; q < 32; q += 2) {
      float e0, e1;
      fma_f32x2(e0, e1, s[q], s[q + 1], sl2_2, nshift_2);
      if ((q & 7) == 6) {  // every fourth on the FMA pipe (57.9 -> 52.3 us)
        ex2_poly_f32x2(e0, e1);
      } else {
        e0 = ex2_approx(e0);
        e1 = ex2_approx(e1);
      }
      w[q >> 1] = pack_bf16x2(e0, e1);
    }
    tmem_st16(ts + c * 16, w);
  }
}

// The softmax warps' tiles j0 .. j1 - 1 of one item, those of their group.
__device__ __forceinline__ void softmax_tiles(uint8_t* smem, uint32_t tmem_base, unsigned* status, float sl2, int j0, int j1, bool whole) {
  using L = Attn3Smem;
  // m is raised (and O rescaled) only when a tile's maximum exceeds it by more than kSlack, so P <= 2^kSlack.
  constexpr float kSlack = 4.0f;
  Attn3Bars* bars = reinterpret_cast<Attn3Bars*>(smem + L::kBarOff);
  volatile int* abort_flag = &bars->abort_flag;
  auto wait_warp = [&](uint64_t& bar, uint32_t parity) { mbar_wait_warp(smem_u32(&bar), parity, abort_flag, status, QB_DEV_WAIT_TIMEOUT_ATTN); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = (warp - 4) >> 2, quarter = warp & 3;
  const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
  const uint32_t ts = tmem_base + g * kKeyTile + lane_addr;  // this thread's row of the group's S, and of P
  const uint32_t tmem_o = tmem_base + kGroups * kKeyTile + lane_addr;
  float* my_m = reinterpret_cast<float*>(smem + L::kRowOff) + quarter * 32 + lane;
  uint64_t* my_turn = &bars->turn[g][quarter];
  uint64_t* next_turn = &bars->turn[g == kGroups - 1 ? 0 : g + 1][quarter];
  int i = (j0 - g + kGroups - 1) / kGroups;  // the group's tiles are j = 3 i + g
  for (int j = kGroups * i + g; j < j1; j += kGroups, ++i) {
    wait_warp(bars->s_full[g], i & 1);
    tc_fence_after();
    int row, valid = kKeyTile;
    if (!whole) locate_tile(bars->seg, j + bars->tile_shift, row, valid);  // (the table is there: Q was staged after it)
    uint32_t s0[32];
    const float m_tile = (valid == kKeyTile ? row_max<false>(ts, valid, s0) : row_max<true>(ts, valid, s0)) * sl2;
    // m is settled tile by tile: after the turn it is what the tiles before this one left
    if (j > 0) {
      wait_warp(*my_turn, g == 0 ? (i - 1) & 1 : i & 1);
    }
    float m = *my_m;
    if (j == j0) {
      m = m_tile;
      *my_m = m;
    } else {
      const bool jump = m_tile > m + kSlack;
      if (__any_sync(0xffffffffu, jump)) {
        // O may be rescaled only when PV(j - 1) has finished.  (S(j - 1) was issued after PV(j - 4), so the barrier is in the
        // phase of tile j - 1 or has finished it.)
        const int gp = g == 0 ? kGroups - 1 : g - 1, ip = g == 0 ? i - 1 : i;
        wait_warp(bars->pv_done[gp], ip & 1);
        const float old = m;
        if (jump) m = m_tile;
        const float alpha = ex2_approx(old - m);
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
        uint32_t lsum = tmem_ld1(tmem_o + 64);
        tmem_wait_ld();
        tmem_loaded(lsum);
        tmem_st1(tmem_o + 64, __float_as_uint(__uint_as_float(lsum) * alpha));
        tmem_wait_st();
        tc_fence_before();
        if (jump) *my_m = m;
      }
    }
    warp_arrive(smem_u32(next_turn), lane);
    const float nshift = -m;
    if (valid == kKeyTile) row_exp<false>(ts, valid, sl2, nshift, s0);
    else row_exp<true>(ts, valid, sl2, nshift, s0);
    tmem_wait_st();
    tc_fence_before();
    warp_arrive(smem_u32(&bars->p_full[g]), lane);
  }
}

// The same as a function of its own, for the kernel with helpers: inlined there, its registers and order changed with whatever surrounded
// it (368 to 399 us at 128 buckets).  A tile takes a fifth longer in it (owned_tiles).  The kernel without is faster with it inlined (52.5 against 55.3 us at 16).
__device__ __noinline__ void softmax_tiles_apart(uint8_t* smem, uint32_t tmem_base, unsigned* status, float sl2, int j0, int j1, bool whole) {
  softmax_tiles(smem, tmem_base, status, sl2, j0, j1, whole);
}

// kHelped: the end of a piece, for the softmax warps.  Group 0 reads O and hands the finished rows on; groups 0 and 1 stage the
// next piece's query rows.  A function of its own, because what it works with (addresses, the places of pieces)
// would otherwise be kept in registers, or spilled, through the loop over the tiles.
__device__ __noinline__ int end_piece3(const AttnArgs& a, uint8_t* smem, uint32_t tmem_o, int piece) {
  using L = Attn3Smem;
  Attn3Bars* b = reinterpret_cast<Attn3Bars*>(smem + L::kBarOff);
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
  if (g == 0) {
    mbar_wait_warp(smem_u32(&b->o_final), piece & 1, abort_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN);
    tc_fence_after();
    read_o<true>(tmem_o, o, l);
  }
  asm volatile("bar.sync 2, 384;" ::: "memory");  // m is final (the first tile of the next piece sets it anew, behind q_ready)
  const float m = reinterpret_cast<const float*>(smem + L::kRowOff)[r];
  const bool good = *abort_flag == 0;
  if (g == 1 && r == 0) b->tile_shift = next.tile0 - (piece + 1) * done.n;  // (read again behind q_ready of the next piece)
  if (next.n > 0) q.stage<false>(smem + L::kQOff, b->tm, &b->q_ready);
  if (g == 0) kr.finish(a, done, r, good, m, l, o, &b->exchange);
  return next.n;
}

template <bool kHelped>
__global__ void __launch_bounds__(kA3Threads, 1)
owl_attn3_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ AttnArgs a) {
  using L = Attn3Smem;
  constexpr int kStages = L::kStages;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kOCol = kGroups * kKeyTile;  // S of group g at columns 128 g, O (80 columns) behind them
  constexpr uint32_t kIdescS = umma_idesc(1, 1, 128, 128);
  constexpr uint32_t kIdescPV = umma_idesc(1, 1, 128, kVRows);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float* m_row = reinterpret_cast<float*>(smem + L::kRowOff);
  Attn3Bars* bars = reinterpret_cast<Attn3Bars*>(smem + L::kBarOff);
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
    for (unsigned i = lane; i < offsetof(Attn3Bars, tmem_slot) / 8; i += 32)
      mbar_init(smem_u32(reinterpret_cast<uint64_t*>(bars) + i), i >= offsetof(Attn3Bars, p_full) / 8 && i < offsetof(Attn3Bars, pv_done) / 8 ? 4 : i == offsetof(Attn3Bars, q_ready) / 8 ? 8 : 1);
    if (lane == 0) {
      *abort_flag = 0;
      *drain_flag = 0;
    }
    fence_barrier_init();
  } else if (threadIdx.x == 96) {
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  // rows of ones under every V^T tile (16 rows x 128 bytes each): the tensor core then returns the row sum of P
  {
    constexpr uint32_t kOnes = 0x3F803F80u;
    for (int i = threadIdx.x; i < kStages * 2 * 128; i += kA3Threads)  // 128 x 16 bytes per tile
      *reinterpret_cast<uint4*>(smem + L::kVOff + (i >> 7) * L::kVTile + 64 * 128 + (i & 127) * 16) = make_uint4(kOnes, kOnes, kOnes, kOnes);
    if (threadIdx.x < kQTile) m_row[threadIdx.x] = -1.0e30f;
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

  // Everything above touched only this CTA's shared memory and TMEM, so it may run while the kernels before this one in the stream are
  // still at work; everything below reads what they wrote.
  grid_dep_launch();
  grid_dep_wait();

  // The table, the query rows with their angles and the frame counter are asked for at once, so that the first K tile is two trips to L2
  // away.
  QueryTile q;
  if (!kHelped && warp >= 4) {
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
  if (kHelped) {
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
  // Registers move from the four control warps to the softmax warps.
  if (warp < 4) {
    setmaxnreg_dec<kA3CtrlRegs>();
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
      // ---------------- TMA producer: K(t), then V(t - 3), in the order in which they are used
      if (elect_one()) {
        int tile = tile0;  // within the item
        int ks = 0, vs = 0;
        uint32_t kph = 1, vph = 1;
        int row[4] = {0, 0, 0, 0}, head[4] = {0, 0, 0, 0};  // of tiles t, t - 1, t - 2, t - 3
        int k_issued = 0, v_issued = 0;
        for (int t = 0; t < n_tiles + kGroups; ++t) {
          if (t < n_tiles) {
            if (kHelped && tile == pc.tile0 + pc.n) {  // on to the next item
              kr.next(pc);
              tile = pc.tile0;
              pc.place(a, q0, qh, kvh);
            }
            int valid;
            locate_tile(seg, tile, row[0], valid);
            head[0] = kvh;
            ++tile;
            if (!wait(bars->k_empty[ks], kph)) break;
            const uint32_t fb = smem_u32(&bars->k_full[ks]);
            mbar_arrive_expect_tx(fb, L::kKBytes);
            tma_load_2d(smem_u32(smem + L::kKOff + ks * L::kKBytes), &tmK, fb, 0, kvh * a.capacity + row[0]);
            ++k_issued;
            if (++ks == kStages) { ks = 0; kph ^= 1; }
          }
          if (t >= kGroups) {
            if (!wait(bars->v_empty[vs], vph)) break;
            const uint32_t fb = smem_u32(&bars->v_full[vs]);
            mbar_arrive_expect_tx(fb, 2 * 64 * 128);
            uint8_t* st = smem + L::kVOff + vs * L::kVBytes;
            tma_load_2d(smem_u32(st), &tmV, fb, row[3], head[3] * 64);
            tma_load_2d(smem_u32(st + L::kVTile), &tmV, fb, row[3] + 64, head[3] * 64);
            ++v_issued;
            if (++vs == kStages) { vs = 0; vph ^= 1; }
          }
#pragma unroll
          for (int i = 3; i > 0; --i) {
            row[i] = row[i - 1];
            head[i] = head[i - 1];
          }
        }
        if (*abort_flag) {
          // Giving up: let the copies already in flight land before this CTA's memory goes away.
          for (int j = max(0, k_issued - kStages); j < k_issued; ++j)
            mbar_wait(smem_u32(&bars->k_full[j % kStages]), (j / kStages) & 1, drain_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN);
          for (int j = max(0, v_issued - kStages); j < v_issued; ++j)
            mbar_wait(smem_u32(&bars->v_full[j % kStages]), (j / kStages) & 1, drain_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN);
        } else {
          // Tail: see the last stage releases land before the CTA can exit.
          for (int j = max(0, n_tiles - kStages); j < n_tiles; ++j)
            if (!wait(bars->k_empty[j % kStages], (j / kStages) & 1) || !wait(bars->v_empty[j % kStages], (j / kStages) & 1)) break;
        }
      }
    } else if (warp == 1) {
      // ---------------- O += P(j) V(j).  Tiles are counted over the pieces of work (kHelped: runs of tiles of one item each, one
      // after the other), so stages, barrier phases and turns run on; only O starts anew.
      if (elect_one()) {
        bool ok = true;
        int j = 0, g = 0, vs = 0;
        uint32_t vph = 0, gph = 0;
        for (int end = kHelped ? pc.n : n_tiles; ok && j < end;) {
          for (const int j0 = j; j < end; ++j) {
            ok = wait(bars->v_full[vs], vph) && wait(bars->p_full[g], gph);
            if (!ok) break;
            tc_fence_after();
            const uint32_t v_addr = smem_u32(smem + L::kVOff + vs * L::kVBytes);
            const uint32_t tp = tmem_base + g * kKeyTile;
            const uint64_t vd0 = umma_desc_k_sw128(v_addr), vd1 = umma_desc_k_sw128(v_addr + L::kVTile);
#pragma unroll
            for (int k = 0; k < 8; ++k) umma_f16_ts(tmem_base + kOCol, tp + 8 * k, (k < 4 ? vd0 : vd1) + 2 * (k & 3), kIdescPV, j > j0 || k > 0);
            umma_commit(smem_u32(&bars->pv_done[g]));
            umma_commit(smem_u32(&bars->v_empty[vs]));
            if (++vs == kStages) { vs = 0; vph ^= 1; }
            if (++g == kGroups) { g = 0; gph ^= 1; }
          }
          if (ok && late(blockIdx.x == gridDim.x - 1, abort_flag, a.status, QB_DEV_WAIT_TIMEOUT_ATTN)) ok = false;
          if (ok) umma_commit(smem_u32(&bars->o_final));
          if (kHelped) {
            kr.next(pc);
            end += pc.n;
          }
        }
      }
    } else {
      // ---------------- S(j) = Q K(j)^T, as soon as the PV before it in the group's columns has read P(j - 3)
      if (elect_one()) {
        const uint32_t q_addr = smem_u32(smem + L::kQOff);
        bool ok = true;
        int j = 0, g = 0, ks = 0;
        uint32_t kph = 0, gph = 1;  // parity of pv_done of tile j - 3
        int piece = 0;
        for (int end = kHelped ? pc.n : n_tiles; ok && j < end; ++piece) {
          ok = wait(bars->q_ready, piece & 1);
          for (; ok && j < end; ++j) {
            ok = wait(bars->k_full[ks], kph) && (j < kGroups || wait(bars->pv_done[g], gph));
            if (!ok) break;
            tc_fence_after();
            const uint32_t k_addr = smem_u32(smem + L::kKOff + ks * L::kKBytes), ts = tmem_base + g * kKeyTile;
            const uint64_t qd = umma_desc_k_sw128(q_addr), kd = umma_desc_k_sw128(k_addr);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_f16(ts, qd + 2 * k, kd + 2 * k, kIdescS, k > 0);
            umma_commit(smem_u32(&bars->s_full[g]));
            umma_commit(smem_u32(&bars->k_empty[ks]));
            if (++ks == kStages) { ks = 0; kph ^= 1; }
            if (++g == kGroups) { g = 0; gph ^= 1; }
          }
          if (kHelped) {
            kr.next(pc);
            end += pc.n;
          }
        }
      }
    }
  } else {
    setmaxnreg_inc<kA3SoftmaxRegs>();
    // ---------------- softmax groups: one query row per thread, group g takes tiles j = 3 i + g
    const int g = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int t = q0 + r;
    const bool row_ok = t < a.tpf;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_o = tmem_base + kOCol + lane_addr;

    if (g < 2) {
      asm volatile("bar.sync 4, 288;" ::: "memory");  // the temporal angles
      if (!kHelped || pc.n > 0) q.stage<false>(smem + L::kQOff, bars->tm, &bars->q_ready);  // (else nothing was requested)
    }
    // every segment a multiple of the tile (720p: 512 keys a bucket): no tile needs a mask, so none is looked up
    const bool whole = ((seg[1] | seg[3] | seg[5]) & (kKeyTile - 1)) == 0;
    int j0 = 0, j1 = kHelped ? pc.n : n_tiles;
    // What the end of a piece needs is worked out there from its number, so that it takes no registers in the loop.
    bool more = !kHelped || pc.n > 0;

    for (int piece = 0; more; ++piece) {
      if (kHelped && piece > 0) {
        const KeyShares again(a, *const_cast<volatile int*>(&bars->tiles), kHelperCost);
        again.at(again.first_item + piece).place(a, q0, qh, kvh);
      }
      const float ks = a.k_scale ? __ldg(a.k_scale + kvh) : 1.0f;
      const float sl2 = ks * 0.125f * 1.4426950408889634f;  // scores -> log2 domain, 1/sqrt(64) folded in
      if (kHelped) softmax_tiles_apart(smem, tmem_base, a.status, sl2, j0, j1, whole);
      else softmax_tiles(smem, tmem_base, a.status, sl2, j0, j1, whole);
      if constexpr (kHelped) {
        const int n = end_piece3(a, smem, tmem_o, piece);
        j0 = j1;
        j1 += n;
        more = n > 0;
        continue;
      }
      more = false;

      // ---------------- the CTA's result: 64 outputs, still scaled by 2^-m, and the row sum in column 64
      if (g < 2) {  // 32 of the outputs each
        float o[32];
#pragma unroll
        for (int d = 0; d < 32; ++d) o[d] = 0.f;
        if (n_tiles > 0) {
          const float vs = a.v_scale ? __ldg(a.v_scale + kvh) : 1.0f;
          wait_warp(bars->o_final, 0);
          tc_fence_after();
          uint32_t oo[32];
          tmem_ld32(tmem_o + g * 32, oo);
          uint32_t lsum = tmem_ld1(tmem_o + 64);
          tmem_wait_ld_into(oo);
          tmem_loaded(lsum);
          const float l = __uint_as_float(lsum);
          const float inv = l > 0.f ? vs / l : 0.f;
#pragma unroll
          for (int d = 0; d < 32; ++d) o[d] = __uint_as_float(oo[d]) * inv;
        }
        if (row_ok && *abort_flag == 0) write_out(a, static_cast<size_t>(t) * a.o_row + static_cast<size_t>(qh) * a.o_head + g * 32, o);
      }
    }
    if (kHelped && kr.tiles == 0) KeyShares::write_zeros(a, r, g, kGroups);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// With helpers where the call has a workspace for them, otherwise one (query tile, head) per CTA.
int32_t launch_attn3(const CUtensorMap& tmK, const CUtensorMap& tmV, const AttnArgs& a, int Hq, bool helped, cudaStream_t st) {
  auto kernel = helped ? owl_attn3_kernel<true> : owl_attn3_kernel<false>;
  static std::atomic<unsigned long long> done[2];
  const int32_t rc = configure_smem(kernel, Attn3Smem::kTotal, done[helped]);
  if (rc != QB_OK) return rc;
  const dim3 grid = helped ? dim3(num_sms()) : dim3((a.tpf + kQTile - 1) / kQTile, Hq);
  return launch_dep("owl_attn kernel (three groups)", kernel, grid, dim3(kA3Threads), Attn3Smem::kTotal, st, tmK, tmV, a);
}

}  // namespace qb
