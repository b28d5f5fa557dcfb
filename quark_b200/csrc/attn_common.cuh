// Pieces shared by the two attention kernels (attn.cu: two softmax groups over 128-key tiles; attn4.cu: three groups
// over 64-key chunks): the kernel arguments and a few instruction wrappers.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "rope.cuh"
#include "sm100.cuh"

namespace qb {

struct AttnArgs {
  const uint16_t* qkv;
  const int32_t* segments;
  const int32_t* n_segments;
  const int32_t* frame_t;
  uint16_t* out;
  uint8_t* out_q;  // optional e4m3 copy of the output
  const float* rope_xy;
  const float* k_scale;
  const float* v_scale;
  unsigned int* status;
  int tpf, n_q_heads, gqa, capacity, max_segments;
  // Q of token t, head h starts at qkv + t * q_row + h * q_head (16-bit words), its output row at out + t * o_row +
  // h * o_head: the packed projection has q_row = qkv_dim, q_head = 64, o_row = Hq * 64, o_head = 64; the head-major
  // layout [Hq * tpf, 64] of Q and of the output has 64 and tpf * 64 for both
  int q_row, q_head, o_row, o_head;
  // Key splits (gridDim.z > 1): CTA z walks its share of the key tiles and leaves (m, row sum, 64 outputs)
  // per query row in `partials`; the CTA that draws the last ticket of a (query tile, head) sums the
  // shares in order of z and writes the output.
  float* partials;  // [heads][query tiles][splits][66][128]; with helpers: [2][heads][query tiles][66][128]
  int* tickets;     // [heads][query tiles], zero between launches
};

__device__ __forceinline__ float ex2_approx(float x);

// A ticket for a partial result that must not be used (a wait of its CTA ran out): the CTA that draws the last ticket, which counts
// them in the lower bits, then writes no row of the item.
constexpr int kLostTicket = 1 << 16;

constexpr int kPartial = 66 * 128;  // floats of a partial result: m and row sum of 128 rows, then 64 x 128 outputs

// What the softmax warps do next: `n` more tiles (0: nothing) of an item, the tile0-th first, `done` tiles into the CTA's work.
struct NextPiece {
  int item, n, tile0, done, kvh;
};

// A run of key tiles of one item, an item being one (query tile, head).
struct Piece {
  int n = 0, tile0 = 0, item = 0;
  __device__ __forceinline__ void place(const AttnArgs& a, int& q0, int& qh, int& kvh) const {
    const int q_tiles = (a.tpf + 127) / 128;
    qh = item / q_tiles;
    q0 = (item - qh * q_tiles) * 128;
    kvh = qh / a.gqa;
  }
};

// How many of an item's `tiles` key tiles its own CTA keeps when `sms` CTAs work on `items` items (sms / 2 < items < sms): the CTAs left
// over are helpers that take the last tiles of up to `per` items each, one item after the other.  `cost` is what a piece costs a helper
// on top of its tiles (the query tile, O, the trip of the partial result through the workspace), in tiles.  Where less than
// the meeting of the two parts would be saved (a session's first frames, or 720p's ring of 16 buckets) the item stays whole.
// 720p, 512 queries x 32 heads (20 helpers of up to 7 items), us per launch: 128 buckets e4m3 344 -> 319, bf16 427 -> 395; 64 buckets
// 174 -> 169 and 221 -> 210; 96 items of 256 queries, 64 buckets 91 -> 73 and 120 -> 98.
// The owners of the items that share a K / V head still walk its keys side by side, and so do the helpers, one after the other: equal
// ranges of the row of all tiles (every CTA the end of one item and the start of the next) balance better but read each key from
// DRAM once per query tile and head (720p, 128 buckets: 339 us against 344 unsplit).
__host__ __device__ inline int owned_tiles(int items, int sms, int tiles, int cost) {
  const int per = (items + (sms - items) - 1) / (sms - items);
  const int keep = static_cast<int>((static_cast<long long>(per) * (tiles + cost) + per) / (per + 1));
  return keep + 2 * cost < tiles ? keep : tiles;
}
constexpr int kHelperCost = 7, kHelperCost4 = 18;  // tiles of 128 keys (attn.cu), chunks of 64 (attn4.cu); 5 to 12 and 10 to 24 were tried

struct KeyShares {
  int tiles = 0, keep = 0, items = 0, first_item = 0, last_item = 0;  // this CTA's items: [first_item, last_item)
  bool helper = false;
  __device__ __forceinline__ KeyShares() {}
  __device__ __forceinline__ KeyShares(const AttnArgs& a, int n_tiles, int cost) : tiles(n_tiles) {
    items = (a.tpf + 127) / 128 * a.n_q_heads;
    const int helpers = static_cast<int>(gridDim.x) - items, c = blockIdx.x;
    keep = owned_tiles(items, gridDim.x, tiles, cost);
    helper = c >= items;
    first_item = helper ? (c - items) * items / helpers : c;
    last_item = helper ? (c - items + 1) * items / helpers : c + 1;
  }
  __device__ __forceinline__ int piece_tiles() const { return helper ? tiles - keep : keep; }
  __device__ __forceinline__ int all_tiles() const { return (last_item - first_item) * piece_tiles(); }
  __device__ __forceinline__ Piece at(int item) const {
    Piece p;
    p.item = item;
    p.tile0 = helper ? keep : 0;
    p.n = item < last_item ? piece_tiles() : 0;
    return p;
  }
  __device__ __forceinline__ Piece first() const { return at(first_item); }
  __device__ __forceinline__ void next(Piece& p) const { p = at(p.item + 1); }

  // One query row's result, still to be divided by the row sum.
  __device__ __forceinline__ static void write_row(const AttnArgs& a, int t, int qh, int kvh, float l, const float (&o)[64]) {
    const float vs = a.v_scale ? __ldg(a.v_scale + kvh) : 1.0f;
    const float inv = l > 0.f ? vs / l : 0.f;
    const size_t at = static_cast<size_t>(t) * a.o_row + static_cast<size_t>(qh) * a.o_head;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) w[q] = pack_bf16x2(o[8 * v + 2 * q] * inv, o[8 * v + 2 * q + 1] * inv);
      *reinterpret_cast<uint4*>(a.out + at + v * 8) = make_uint4(w[0], w[1], w[2], w[3]);
      if (a.out_q != nullptr)  // narrowed from the bf16-rounded values: equals a separate bf16 -> e4m3 cast
        *reinterpret_cast<uint2*>(a.out_q + at + v * 8) = make_uint2(pack_e4m3x4(bf16lo(w[0]), bf16hi(w[0]), bf16lo(w[1]), bf16hi(w[1])),
                                                                     pack_e4m3x4(bf16lo(w[2]), bf16hi(w[2]), bf16lo(w[3]), bf16hi(w[3])));
    }
  }

  // The 128 threads of group 0, one row each: writes the rows of a whole item; otherwise leaves them in the workspace and, as the
  // second of the item's two CTAs, sums both parts (the same bits whichever CTA is the second).
  __device__ __forceinline__ void finish(const AttnArgs& a, const Piece& p, int r, bool good, float m, float l, float (&o)[64], int* exchange) const {
    int q0, qh, kvh;
    p.place(a, q0, qh, kvh);
    const int t = q0 + r;
    const bool row = good && t < a.tpf;
    if (p.n == tiles) {
      if (row) write_row(a, t, qh, kvh, l, o);
      return;
    }
    float* owner = a.partials + static_cast<size_t>(p.item) * kPartial + r;
    float* other = owner + static_cast<size_t>(items) * kPartial;
    float* mine = helper ? other : owner;
    mine[0] = m;
    mine[128] = l;
#pragma unroll
    for (int d = 0; d < 64; ++d) mine[(2 + d) * 128] = o[d];
    __threadfence();
    asm volatile("bar.sync 3, 128;" ::: "memory");
    if (r == 0) {
      const int was = atomicAdd(a.tickets + p.item, good ? 1 : kLostTicket + 1);
      const bool last = (was & (kLostTicket - 1)) == 1;
      if (last) a.tickets[p.item] = 0;  // ready for the next launch
      *exchange = last && was < kLostTicket;
    }
    asm volatile("bar.sync 3, 128;" ::: "memory");
    if (*exchange == 0) return;
    __threadfence();
    const float* theirs = helper ? owner : other;
    const float m1 = __ldcg(theirs), l1 = __ldcg(theirs + 128);
    float o1[64];
#pragma unroll
    for (int d = 0; d < 64; ++d) o1[d] = __ldcg(theirs + (2 + d) * 128);
    const float top = fmaxf(m, m1);
    const float wm = ex2_approx(m - top), wt = ex2_approx(m1 - top);
    l = __fadd_rn(__fmul_rn(l, wm), __fmul_rn(l1, wt));  // (contracted, it would depend on whose product is rounded)
#pragma unroll
    for (int d = 0; d < 64; ++d) o[d] = __fadd_rn(__fmul_rn(o[d], wm), __fmul_rn(o1[d], wt));
    if (row) write_row(a, t, qh, kvh, l, o);
  }

  // No valid key at all: every output row is zero.  Thread (r, part) of `parts` writes its share of row r of the CTA's items.
  __device__ __forceinline__ static void write_zeros(const AttnArgs& a, int r, int part, int parts) {
    const int items = (a.tpf + 127) / 128 * a.n_q_heads;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      Piece p;
      p.item = item;
      int q0, qh, kvh;
      p.place(a, q0, qh, kvh);
      if (q0 + r >= a.tpf) continue;
      const size_t at = static_cast<size_t>(q0 + r) * a.o_row + static_cast<size_t>(qh) * a.o_head;
      for (int v = part; v < 8; v += parts) {
        *reinterpret_cast<uint4*>(a.out + at + v * 8) = make_uint4(0, 0, 0, 0);
        if (a.out_q != nullptr) *reinterpret_cast<uint2*>(a.out_q + at + v * 8) = make_uint2(0, 0);
      }
    }
  }
};

#ifndef QB_EX2_VOLATILE
#define QB_EX2_VOLATILE 0
#endif
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
#if QB_EX2_VOLATILE
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
#else
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
#endif
  return y;
}
// One arrival for the whole warp: an mbarrier arrival is an atomic on shared memory.  __syncwarp orders the
// lanes' earlier writes (and fences) before lane 0's arrival, which releases them to the waiting thread.
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// UMMA descriptor for a K-major tile with 64-byte rows and the 64-byte swizzle (fp8, head_dim 64).
__device__ __forceinline__ uint64_t umma_desc_k_sw64(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(512 >> 4) << 32;  // 8 rows x 64 B
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(4) << 61;         // SWIZZLE_64B
  return d;
}

// 2^x for an e4m3 probability without the special-function unit, in three instructions of the FMA / integer pipes:
// the caller adds 1.5 * 2^15 to x inside the multiply-add that forms x (so v = x rounded to 8 fractional bits, sitting in
// the low mantissa bits of v), and the float whose exponent field is floor(x) + 127 and whose mantissa is the fraction
// is v's bit pattern times 2^15 plus a constant: 2^floor(x) * (1 + frac(x) - 0.052), the chord of 2^x lowered by 0.052 so
// that its mean error over the fraction is near zero (-5.2 % .. +2.3 %; an e4m3 code is 6.25 % wide; in a simulation of
// 8192-key rows the output's 1 - cosine against exact arithmetic goes from 3.6e-4 to 4.3e-4 at worst).  x is clamped at -120 (the result then
// narrows to zero).  Every second probability of a row is built this way in the kLin instantiations of the e4m3 kernel
// (the default; qb_set_attn_exact_exp(1) or QB_ATTN_EXACT_EXP=1 selects the instantiations that use the special-function
// unit for every element): the exponentials no longer queue behind one another there, at the same number of
// instructions issued.  Measured at 720p, 8320 keys, us per launch: 52.0 exact; 49.5 with the turn passing at chunk 2 as
// in the exact kernel; 46.5 with the turn passing before chunk 0 (the groups then overlap almost fully, which the exact
// kernel cannot afford: 62.6); 47.9 without turns; 3 / 5 of every 8 elements instead of 4: 51.6 / 47.2; all: 56.0.
constexpr float kLinMagic = 49152.0f;  // 1.5 * 2^15: floats in [2^15, 2^16) have an ulp of 2^-8
// (The clamp is a maximum on the ALU pipe, the busiest one of the kernel at 58 %; moving it to the FMA pipe as a
// saturating multiply-add followed by a second multiply-add costs one instruction more and measured 49.5 against 46.5 us:
// what counts is the number of instructions issued.)
__device__ __forceinline__ float ex2_lin_from_biased(float v) {
  v = fmaxf(v, kLinMagic - 120.0f);
  constexpr uint32_t kC = 0x3F800000u - 0x47400000u * 32768u - 436208u;  // 0x47400000 = bits of 49152.0f; 436208 = 0.052 * 2^23
  return __uint_as_float(__float_as_uint(v) * 32768u + kC);
}

}  // namespace qb
