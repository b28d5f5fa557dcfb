// Pieces shared by the two attention kernels (attn.cu: two softmax groups, e4m3 and key splits; attn3.cu: three groups, bf16 without key
// splits): the kernel arguments, the ways to share keys, the query tile, and a few instruction wrappers.
#pragma once

#include <atomic>

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
// 720p, 512 queries x 32 heads (20 helpers of up to 7 items), 64 / 128 / 256 buckets, e4m3: 143, 272, 517 us,
// with the items whole 150, 295, 577; cost 12 149 at 64, the rest alike; cost 16 and more loses up to 9 %.  bf16: 208, 392, 745 us and whole
// 192, 372, 721, since a tile takes a fifth longer in its kernel with helpers; kept, because two accumulators share the
// additions (error at 128 buckets over that of three accumulators, keys N(0, 1): 0.3 against 0.4 % more, few keys that count: 0.4 against 0.8).
// The owners of the items that share a K / V head still walk its keys side by side, and so do the helpers, one after the other: equal
// ranges of the row of all tiles (every CTA the end of one item and the start of the next) balance better but read each key from
// DRAM once per query tile and head (720p, 128 buckets: 339 us against 344 unsplit).
__host__ __device__ inline int owned_tiles(int items, int sms, int tiles, int cost) {
  const int per = (items + (sms - items) - 1) / (sms - items);
  const int keep = static_cast<int>((static_cast<long long>(per) * (tiles + cost) + per) / (per + 1));
  return keep + 2 * cost < tiles ? keep : tiles;
}
constexpr int kHelperCost = 9;

// Outputs of a query row (divided by the row sum already) and their e4m3 copy, narrowed from the bf16-rounded values: it equals a
// separate cast.
template <int kN>
__device__ __forceinline__ void write_out(const AttnArgs& a, size_t at, const float (&o)[kN]) {
#pragma unroll
  for (int v = 0; v < kN / 8; ++v) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = pack_bf16x2(o[8 * v + 2 * q], o[8 * v + 2 * q + 1]);
    *reinterpret_cast<uint4*>(a.out + at + v * 8) = make_uint4(w[0], w[1], w[2], w[3]);
    if (a.out_q != nullptr)
      *reinterpret_cast<uint2*>(a.out_q + at + v * 8) = make_uint2(pack_e4m3x4(bf16lo(w[0]), bf16hi(w[0]), bf16lo(w[1]), bf16hi(w[1])),
                                                                   pack_e4m3x4(bf16lo(w[2]), bf16hi(w[2]), bf16lo(w[3]), bf16hi(w[3])));
  }
}

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
    float y[64];
#pragma unroll
    for (int d = 0; d < 64; ++d) y[d] = o[d] * inv;
    write_out(a, at, y);
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
// Two multiply-adds in one instruction: x = a * s + t, s and t being pairs.
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void fma_f32x2(float& x0, float& x1, uint32_t a0, uint32_t a1, uint64_t s, uint64_t t) {
  asm("{\n\t.reg .b64 A, D;\n\tmov.b64 A, {%2, %3};\n\tfma.rn.f32x2 D, A, %4, %5;\n\tmov.b64 {%0, %1}, D;\n\t}"
      : "=f"(x0), "=f"(x1)
      : "r"(a0), "r"(a1), "l"(s), "l"(t));
}
__device__ __forceinline__ void add_f32x2(uint64_t& acc, uint32_t a0, uint32_t a1) {
  asm("{\n\t.reg .b64 A;\n\tmov.b64 A, {%1, %2};\n\tadd.rn.f32x2 %0, %0, A;\n\t}" : "+l"(acc) : "r"(a0), "r"(a1));
}
__device__ __forceinline__ float sum_f32x2(uint64_t a, uint64_t b) {
  float a0, a1, b0, b1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(b));
  return (a0 + a1) + (b0 + b1);
}
// 2^x for two values on the FMA and integer pipes: x = n + f with n = round(x) in the low mantissa bits of x + 1.5 * 2^23, a
// polynomial for 2^f on [-0.5, 0.5] (least squares with 2^0 = 1 held, weighted until the relative error is level: 9.1e-8, evaluated in f32
// 1.7e-7, below the 2^-22 of ex2.approx; a degree less made 2.7e-6 of it), times 2^n.  As with ex2.approx.ftz, NaN stays NaN and what would be
// below 2^-126, -inf among it, is 0: x is clamped at -127 by a maximum that keeps NaN, and the bits of 2^-127 come out as those of 0.
__device__ __forceinline__ void ex2_poly_f32x2(float& x0, float& x1) {
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x0) : "f"(-127.0f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x1) : "f"(-127.0f));
  const uint64_t x = pack_f32x2(x0, x1), magic = pack_f32x2(12582912.0f, 12582912.0f), nmagic = pack_f32x2(-12582912.0f, -12582912.0f),
                 none = pack_f32x2(-1.0f, -1.0f);
  uint64_t t, f, p;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(x), "l"(magic));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(f) : "l"(t), "l"(nmagic));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(f) : "l"(f), "l"(none), "l"(x));
  p = pack_f32x2(0.0013264727f, 0.0013264727f);
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(p) : "l"(f), "l"(pack_f32x2(0.009671513f, 0.009671513f)));
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(p) : "l"(f), "l"(pack_f32x2(0.055507336f, 0.055507336f)));
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(p) : "l"(f), "l"(pack_f32x2(0.24022242f, 0.24022242f)));
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(p) : "l"(f), "l"(pack_f32x2(0.693147f, 0.693147f)));
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(p) : "l"(f), "l"(pack_f32x2(1.0f, 1.0f)));
  uint32_t t0, t1;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(t0), "=r"(t1) : "l"(t));
  const uint64_t s = pack_f32x2(__uint_as_float((t0 << 23) + 0x3F800000u), __uint_as_float((t1 << 23) + 0x3F800000u));
  asm("mul.rn.ftz.f32x2 %0, %0, %1;" : "+l"(p) : "l"(s));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(p));
}
// Four f32 -> four packed e4m3, joined by the conversions themselves.
__device__ __forceinline__ uint32_t merge_e4m3x4(float a, float b, float c, float d) {
  uint32_t r;
  asm("{\n\t.reg .b16 l, h;\n\tcvt.rn.satfinite.e4m3x2.f32 l, %2, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 h, %4, %3;\n\tmov.b32 %0, {l, h};\n\t}"
      : "=r"(r)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
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
// (the default; qb_set_attn_exact_exp(1) or QB_ATTN_EXACT_EXP=1 selects the instantiations without it): the exponentials no longer queue
// behind one another at the special-function unit.  Measured at 720p, 8320 keys, us per launch: 41.4 against 57.0 without.
constexpr float kLinMagic = 49152.0f;  // 1.5 * 2^15: floats in [2^15, 2^16) have an ulp of 2^-8
// (The clamp is a maximum on the ALU pipe, the busiest one of the kernel at 58 %; moving it to the FMA pipe as a
// saturating multiply-add followed by a second multiply-add costs one instruction more and measured 49.5 against 46.5 us:
// what counts is the number of instructions issued.)
__device__ __forceinline__ float ex2_lin_from_biased(float v) {
  v = fmaxf(v, kLinMagic - 120.0f);
  constexpr uint32_t kC = 0x3F800000u - 0x47400000u * 32768u - 436208u;  // 0x47400000 = bits of 49152.0f; 436208 = 0.052 * 2^23
  return __uint_as_float(__float_as_uint(v) * 32768u + kC);
}

constexpr int kQTile = 128;
constexpr int kKeyTile = 128;
constexpr int kVRows = 80;  // of a V^T tile: 64 channels + 16 rows of ones (row sum of P)

// Which 128-key tile is the j-th valid one?  Returns its first cache row and how many of its
// keys are valid.  Segments are (start, length) pairs; zero-length entries are legal.
__device__ __forceinline__ void locate_tile(const int* seg, int j, int& row, int& valid) {
  row = 0;
  valid = 0;
  bool found = false;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int nt = (seg[2 * i + 1] + kKeyTile - 1) / kKeyTile;
    if (!found && j < nt) {
      row = seg[2 * i] + j * kKeyTile;
      valid = min(kKeyTile, seg[2 * i + 1] - j * kKeyTile);
      found = true;
    }
    j -= nt;
  }
}

// Whether the keys of a (query tile, head) are shared by gridDim.z CTAs, and how their results are brought together: through the
// workspace (see AttnArgs::partials), or, the CTAs being one thread-block cluster, in shared memory.  The unsplit kernel is an
// instantiation of its own so that none of this reaches its instruction stream.  kHelped: the CTAs that
// the items leave over take a part of the keys of several items each (KeyShares).
enum { kUnsplit = 0, kSplitWorkspace = 1, kSplitCluster = 2, kHelped = 3 };

// The table on its way; returns n_segments.
__device__ __forceinline__ int request_table(const AttnArgs& a, int (&seg)[6]) {
  const int nseg = *after_wait(a.n_segments);
  const int32_t* table = after_wait(a.segments);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    seg[2 * i] = i < a.max_segments ? table[2 * i] : 0;
    seg[2 * i + 1] = i < a.max_segments ? table[2 * i + 1] : 0;
  }
  return nseg;
}

// What was requested, checked (ordinary loads: the table is the work of the kernel before).  Returns the number of key tiles, the same in
// every thread; a malformed table is reported and counts as empty.
__device__ __forceinline__ int load_table(const AttnArgs& a, int nseg, int (&seg)[6]) {
  nseg = min(nseg, a.max_segments);
  bool ok = true;
  int n = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (i >= nseg) seg[2 * i] = seg[2 * i + 1] = 0;
    if (seg[2 * i] < 0 || seg[2 * i + 1] < 0 || (seg[2 * i] & 15) != 0 || seg[2 * i] + seg[2 * i + 1] > a.capacity) ok = false;
    n += (seg[2 * i + 1] + kKeyTile - 1) / kKeyTile;
  }
  if (ok) return n;
#pragma unroll
  for (int i = 0; i < 6; ++i) seg[i] = 0;
  if (threadIdx.x == 0) atomicOr(a.status, QB_DEV_BAD_SEGMENT);
  return 0;
}

// The query tile: 128 rows of 8 units of 16 bytes, four units to a thread of groups 0 and 1 (256 threads): unit (n & 7) of row n >> 3, n =
// the thread's number + 256 i.  (A row per thread and group, as the tensor core will want them, made every load touch 32 lines: 2500
// cycles until the last one was here.)
struct QueryTile {
  uint4 x[4];      // 8 values: 4 pairs to rotate
  float2 c[4], s[4];  // spatial units (0..3): cosines and sines of the two angles of the 4 pairs

  __device__ __forceinline__ static int number() { return static_cast<int>(threadIdx.x) - 128; }  // (the softmax warps start at thread 128)
  // The rows' angles.  Behind grid_dep_wait like the rows: the table may be the work of a kernel before (qb_rope_table_build).
  __device__ __forceinline__ void request_angles(const AttnArgs& a, int q0) {
    const int n = number(), u = n & 7;
    if (n >= 256 || u >= 4) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = q0 + (n >> 3) + 32 * i;
      c[i] = s[i] = make_float2(0.f, 0.f);
      if (t >= a.tpf) continue;
      const float* xy = a.rope_xy + static_cast<size_t>(t) * 16 + 2 * u;
      asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(c[i].x), "=f"(c[i].y) : "l"(xy) : "memory");
      asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(s[i].x), "=f"(s[i].y) : "l"(xy + 8) : "memory");
    }
  }
  // The rows.  (volatile: ordinary loads were moved down to where they are used, behind the segment table.)
  __device__ __forceinline__ void request(const AttnArgs& a, int q0, int qh) {
    const int n = number(), u = n & 7;
    if (n >= 256) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = q0 + (n >> 3) + 32 * i;
      x[i] = make_uint4(0, 0, 0, 0);
      if (t >= a.tpf) continue;
      const uint16_t* src = a.qkv + static_cast<size_t>(t) * a.q_row + static_cast<size_t>(qh) * a.q_head + 8 * u;
      asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x[i].x), "=r"(x[i].y), "=r"(x[i].z), "=r"(x[i].w) : "l"(src) : "memory");
    }
  }
  // Rotated (RoPE; `tm`: cosines and sines of the temporal angles), narrowed and stored to shared memory, K-major and swizzled like a TMA
  // tile: pair p = 4 u + j of a row becomes its values p and 32 + p.
  template <bool kFp8>
  __device__ __forceinline__ void stage(uint8_t* q_s, const float* tm, uint64_t* q_ready) {
    const int n = number(), u = n & 7;
    if (n >= 256) return;
    float2 ct, st;
    if (u >= 4) {
      ct = make_float2(tm[2 * u - 8], tm[2 * u - 7]);
      st = make_float2(tm[2 * u], tm[2 * u + 1]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = (n >> 3) + 32 * i;
      const float2 co = u < 4 ? c[i] : ct, si = u < 4 ? s[i] : st;
      const uint32_t w[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
      float y0[4], y1[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float cc = j < 2 ? co.x : co.y, ss = j < 2 ? si.x : si.y;
        const float x0 = bf16lo(w[j]), x1 = bf16hi(w[j]);
        y0[j] = __fsub_rn(__fmul_rn(x0, cc), __fmul_rn(x1, ss));
        y1[j] = __fadd_rn(__fmul_rn(x1, cc), __fmul_rn(x0, ss));
      }
      if (kFp8) {  // 64-byte rows; 16-byte unit XOR ((row >> 1) & 3)
        uint8_t* row = q_s + r * 64 + (u & 3) * 4;
        const int sw = (r >> 1) & 3;
        *reinterpret_cast<uint32_t*>(row + (((u >> 2) ^ sw) << 4)) = pack_e4m3x4(y0[0], y0[1], y0[2], y0[3]);
        *reinterpret_cast<uint32_t*>(row + ((((u >> 2) + 2) ^ sw) << 4)) = pack_e4m3x4(y1[0], y1[1], y1[2], y1[3]);
      } else {  // 128-byte rows; unit XOR (row & 7)
        uint8_t* row = q_s + r * 128 + (u & 1) * 8;
        const int sw = r & 7;
        *reinterpret_cast<uint2*>(row + (((u >> 1) ^ sw) << 4)) = make_uint2(pack_bf16x2(y0[0], y0[1]), pack_bf16x2(y0[2], y0[3]));
        *reinterpret_cast<uint2*>(row + ((((u >> 1) + 4) ^ sw) << 4)) = make_uint2(pack_bf16x2(y1[0], y1[1]), pack_bf16x2(y1[2], y1[3]));
      }
    }
    fence_proxy_async_smem();
    tc_fence_before();
    warp_arrive(smem_u32(q_ready), threadIdx.x & 31);
  }
};

// Keys from `valid` on of the 32 columns that start at c * 32 count nothing: -inf.
__device__ __forceinline__ void mask_chunk(uint32_t (&s)[32], int c, int valid) {
#pragma unroll
  for (int q = 0; q < 32; ++q)
    if (c * 32 + q >= valid) s[q] = 0xff800000u;
}

// A row's result: 64 outputs and, where the tensor core made it (kSum), the row sum, still scaled by 2^(kPShift - m).
template <bool kSum>
__device__ __forceinline__ void read_o(uint32_t tmem_o, float (&o)[64], float& l) {
  uint32_t oo[2][32];
  tmem_ld32(tmem_o, oo[0]);
  tmem_ld32(tmem_o + 32, oo[1]);
  uint32_t lsum = kSum ? tmem_ld1(tmem_o + 64) : 0;
  tmem_wait_ld_into(oo[0]);
  tmem_loaded(oo[1]);
  tmem_loaded(lsum);
#pragma unroll
  for (int d = 0; d < 64; ++d) o[d] = __uint_as_float(oo[d >> 5][d & 31]);
  if (kSum) l = __uint_as_float(lsum);
}

// The shared memory of a kernel, once per device (`done`: a bit per device).
template <typename K>
int32_t configure_smem(K kernel, int smem_bytes, std::atomic<unsigned long long>& done) {  // once per device
  int dev = 0;
  QB_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 64 && (done.load(std::memory_order_relaxed) >> dev & 1) != 0) return QB_OK;
  QB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_relaxed);
  return QB_OK;
}

}  // namespace qb
