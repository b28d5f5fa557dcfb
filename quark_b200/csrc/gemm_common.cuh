// What the two GEMM kernels share (gemm.cu: tiles of one CTA; gemm_pair.cu: tiles of a pair of CTAs): their arguments, the
// epilogue on 8 columns, the exchange of K slices inside a cluster and the epilogue of the QKV projection.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "rope.cuh"
#include "sm100.cuh"

namespace qb {

constexpr int kBM = 128;          // rows of A per CTA = TMEM lanes
constexpr int kRowBytes = 128;    // bytes of K per stage row = one swizzle atom
constexpr int kGemmThreads = 320; // 10 warps: TMA, MMA, 2 x 4 epilogue (two warps per TMEM lane quarter)

// What the QKV projection's fused epilogue needs beyond the GEMM: per-head RMS norm of Q and K, value
// residual on V, RoPE(K) and the KV-cache append happen on the accumulator tile, before anything is
// written (the stand-alone kernels are in qkv_post.cu and kv.cu; results are bit-identical to them).
struct QkvTail {
  const uint16_t* qkv_first;  // may be null: no value residual
  const float* lamb;
  const int32_t* frame_t;
  const int32_t* frozen;
  void* K_cache;
  void* Vt_cache;
  int32_t* segments;
  int32_t* n_segments;
  const float* rope_xy;
  const float* k_scale;  // optional per-KV-head cache scales (see qb_kv_params)
  const float* v_scale;
  int n_q_heads, n_kv_heads, tpf, nb, pd, max_segments, kv_fp8;
  // Quilt: the cache keeps tokens qoff, qoff + quilt, ... of the frame (tpf / quilt of them); slots, capacity and the
  // segment table are those of a frame of tpf / quilt tokens (src/quark/kernels/kv_cache_update/reference.py:201-207)
  int quilt, qoff;
  float eps;
};

struct GemmArgs {
  int M, N, K;
  int a_rows;  // rows of A in a box: 128, or M rounded up to 8 below that (rows past it hold what was there: never stored)
  int kb_total, kb_per_split, splits;
  int cluster;  // K slices are the CTAs of one thread-block cluster and are summed through distributed shared memory
  int through_bf16;  // an e4m3 C is rounded to bf16 first (grouped GEMM)
  int b_const;  // no kernel still in flight writes B (weights): its first tiles are fetched ahead of the grid dependency
  int c_dtype, activation, rows_per_gate;
  const float* a_scale;
  const float* w_scale;
  const uint16_t* bias;
  const uint16_t* gate;
  const uint16_t* residual;
  void* C;
  float* partials;
  int* counters;
  unsigned int* status;
  QkvTail qkv;  // for the instantiations whose epilogue is that of the QKV projection
  // Row-parallel GEMM of a tensor-parallel rank: row m of the bf16 partial goes to the rank that owns that row in the
  // cross-GPU reduction (m / tp_rpo), into that rank's staging area for partials from this rank (peer-mapped memory,
  // plain stores over NVLink): tp_dst[owner] + (m % tp_rpo) * N.  tp_world == 0: the ordinary output C.
  int tp_world, tp_rpo;
  uint16_t* tp_dst[8];
  // Grouped GEMM (mixture of experts, gemm_grouped.cu): the 128-row tile i of A belongs to expert tile_expert[i] and is multiplied
  // with rows [expert * N, expert * N + N) of B; a tile with expert -1 is skipped.
  const int* tile_expert;
  // Pairs of CTAs only: the walk over the tiles (see tile_at in gemm_pair.cu) and the shared memory's layout
  int tiles_m, n_tiles, group_m, stages, scratch;
};

// Applies the epilogue to 8 consecutive columns of one row and stores them.
__device__ __forceinline__ void epilogue_store8(const GemmArgs& g, float (&v)[8], int m, int n) {
  if (g.a_scale != nullptr || g.w_scale != nullptr) {
    const float sa = g.a_scale ? *g.a_scale : 1.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= g.w_scale ? sa * __ldg(g.w_scale + n + j) : sa;
  }
  if (g.bias != nullptr) {
    const uint4 b = *reinterpret_cast<const uint4*>(g.bias + n);  // may be the output of the kernel before (MLPFusion)
    const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] += bf16lo(w[j]);
      v[2 * j + 1] += bf16hi(w[j]);
    }
  }
  if (g.activation == 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = silu_fast(v[j]);
  }
  if (g.gate != nullptr) {
    const size_t grow = static_cast<size_t>(m / g.rows_per_gate) * g.N;
    const uint4 gt = *reinterpret_cast<const uint4*>(g.gate + grow + n);
    const uint4 rs = *reinterpret_cast<const uint4*>(g.residual + static_cast<size_t>(m) * g.N + n);
    const uint32_t gw[4] = {gt.x, gt.y, gt.z, gt.w};
    const uint32_t rw[4] = {rs.x, rs.y, rs.z, rs.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __fadd_rn(bf16lo(rw[j]), __fmul_rn(bf16lo(gw[j]), v[2 * j]));
      v[2 * j + 1] = __fadd_rn(bf16hi(rw[j]), __fmul_rn(bf16hi(gw[j]), v[2 * j + 1]));
    }
  }
  const size_t off = static_cast<size_t>(m) * g.N + n;
  if (g.c_dtype == QB_BF16) {
    uint4 o;
    o.x = pack_bf16x2(v[0], v[1]);
    o.y = pack_bf16x2(v[2], v[3]);
    o.z = pack_bf16x2(v[4], v[5]);
    o.w = pack_bf16x2(v[6], v[7]);
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(g.C) + off) = o;
  } else if (g.c_dtype == QB_E4M3) {
    uint2 o;
    o.x = pack_e4m3x4(v[0], v[1], v[2], v[3]);
    o.y = pack_e4m3x4(v[4], v[5], v[6], v[7]);
    *reinterpret_cast<uint2*>(static_cast<uint8_t*>(g.C) + off) = o;
  } else {
    float4* dst = reinterpret_cast<float4*>(static_cast<float*>(g.C) + off);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// The same on values that were fetched ahead: `col` points at this column's scale, with the bias BN and the gate 2 BN words
// further, and `rs` is the residual.
template <int BN>
__device__ __forceinline__ void epilogue_store8_staged(const GemmArgs& g, float (&v)[8], int m, int n, const float* col, const uint4& rs) {
  if (g.a_scale != nullptr || g.w_scale != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= col[j];
  }
  if (g.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += col[BN + j];
  }
  if (g.activation == 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = silu_fast(v[j]);
  }
  if (g.gate != nullptr) {
    const uint32_t rw[4] = {rs.x, rs.y, rs.z, rs.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __fadd_rn(bf16lo(rw[j]), __fmul_rn(col[2 * BN + 2 * j], v[2 * j]));
      v[2 * j + 1] = __fadd_rn(bf16hi(rw[j]), __fmul_rn(col[2 * BN + 2 * j + 1], v[2 * j + 1]));
    }
  }
  const size_t off = static_cast<size_t>(m) * g.N + n;
  if (g.c_dtype == QB_BF16) {
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(g.C) + off) =
        make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
  } else if (g.c_dtype == QB_E4M3) {
    *reinterpret_cast<uint2*>(static_cast<uint8_t*>(g.C) + off) = make_uint2(pack_e4m3x4(v[0], v[1], v[2], v[3]), pack_e4m3x4(v[4], v[5], v[6], v[7]));
  } else {
    float4* dst = reinterpret_cast<float4*>(static_cast<float*>(g.C) + off);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// Where slice s's partial sums of columns [4 c4, 4 c4 + 4) of a row lie among a CTA's 128 / S = `rows` rows, in 16-byte units:
// consecutive rows (the lanes of a pushing warp) are neighbours, and the exclusive-or spreads the column groups of a row (the
// lanes that read them) over the banks.
template <int BN>
__device__ __forceinline__ int slice_unit(int s, int c4, int row, int rows) {
  return (s * (BN / 4) + c4) * rows + (row ^ ((c4 >> 1) & 7));
}

// K slices of a cluster: this thread's half row of the partial tile into the scratch area of the CTA that finishes the row.
template <int CG, int BN>
__device__ __forceinline__ void push_slices(uint8_t* scratch, uint32_t taddr, int split, int rank, int row, int half, int splits) {
  const int rows = kBM / splits;
  const uint32_t base = map_to_cta(smem_u32(scratch), CG * (row / rows) + rank);
#pragma unroll
  for (int c = 0; c < BN / 64; ++c) {
    uint32_t r[32];
    tmem_ld32(taddr + half * (BN / 2) + c * 32, r);
    tmem_wait_ld_into(r);
#pragma unroll
    for (int v = 0; v < 8; ++v)
      st_dsmem_v4(base + 16 * slice_unit<BN>(split, half * (BN / 8) + c * 8 + v, row % rows, rows), r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
  }
}

// A CTA whose slice is missing (a wait ran out) tells the CTAs that would sum it, in front of the cluster barrier behind which they
// do; they write no row of the tile then.
template <int CG>
__device__ __forceinline__ void tell_lost(volatile int* lost_flag, int rank, int splits) {
  for (int s = 0; s < splits; ++s) st_dsmem(map_to_cta(smem_u32(const_cast<const int*>(lost_flag)), CG * s + rank), 1);
}
// The same for slices through the workspace: what such a CTA adds to the tile's counter, whose lower half counts the tickets.
constexpr int kLostTicket = 1 << 16;

// Whether `ok` holds for all 256 epilogue threads (a barrier of theirs).
__device__ __forceinline__ bool all_of_epilogue(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "bar.red.and.pred p, 2, 256, q;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1 : 0)
      : "memory");
  return r != 0;
}

// After the cluster barrier: this CTA's rows of the tile, 8 columns at a time per thread (neighbouring threads take neighbouring
// groups of a row, so that whole lines are read and written), summed in slice order.  pre[k][0]: the residuals.
template <int BN>
__device__ __forceinline__ void finish_slices(const GemmArgs& g, const float4* parts, const float* col, int m0, int n0, int row0, int rows, bool one_gate,
                                              const uint4 (&pre)[BN / 32][2]) {
  const int et = threadIdx.x - 64, c8 = et % (BN / 8);
#pragma unroll
  for (int k = 0; k < BN / 32; ++k) {
    const int r = et / (BN / 8) + 256 / (BN / 8) * k;
    const int m = m0 + row0 + r, n = n0 + c8 * 8;
    if (r >= rows || m >= g.M || n >= g.N) continue;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < g.splits; ++s) {
      const float4 x = parts[slice_unit<BN>(s, 2 * c8, r, rows)], y = parts[slice_unit<BN>(s, 2 * c8 + 1, r, rows)];
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
      v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
    }
    if (one_gate) epilogue_store8_staged<BN>(g, v, m, n, col + c8 * 8, pre[k][0]);
    else epilogue_store8(g, v, m, n);
  }
}

// Row m of the output in bytes.
__device__ __forceinline__ uint8_t* row_of_c(const GemmArgs& g, int m) {
  if (g.tp_world != 0) {
    const int owner = m / g.tp_rpo;
    return reinterpret_cast<uint8_t*>(g.tp_dst[owner] + static_cast<size_t>(m - owner * g.tp_rpo) * g.N);
  }
  const int es = g.c_dtype == QB_BF16 ? 2 : g.c_dtype == QB_E4M3 ? 1 : 4;
  return static_cast<uint8_t*>(g.C) + static_cast<size_t>(m) * g.N * es;
}

// The plain epilogue on 16 columns of one row: r the accumulator, `col` at the first column's scale (bias BN, gate 2 BN words
// further), `res` the residual.  Kept small and called in a loop: unrolled over the half row, with every branch in it, the
// epilogue's instructions cost more to fetch (0.5 us a launch) than they took to run.
template <int BN>
__device__ __forceinline__ void epilogue16(const GemmArgs& g, const uint32_t (&r)[16], int m, int n, const float* col, const uint4* res, bool one_gate,
                                           uint8_t* c_row, bool wide, bool store) {
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
  if (g.a_scale != nullptr || g.w_scale != nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] *= col[j];
  }
  if (g.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] += col[BN + j];
  }
  if (g.activation == 1) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = silu_fast(v[j]);
  }
  const bool second = n + 8 < g.N;
  if (g.gate != nullptr) {
    const uint4 x = res[0], y = second ? res[1] : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t rw[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    if (one_gate) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[2 * j] = __fadd_rn(bf16lo(rw[j]), __fmul_rn(col[2 * BN + 2 * j], v[2 * j]));
        v[2 * j + 1] = __fadd_rn(bf16hi(rw[j]), __fmul_rn(col[2 * BN + 2 * j + 1], v[2 * j + 1]));
      }
    } else {  // the tile spans several gate rows
      const uint32_t* gt = reinterpret_cast<const uint32_t*>(g.gate + static_cast<size_t>(m / g.rows_per_gate) * g.N + n);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t w = j < 4 || second ? gt[j] : 0u;
        v[2 * j] = __fadd_rn(bf16lo(rw[j]), __fmul_rn(bf16lo(w), v[2 * j]));
        v[2 * j + 1] = __fadd_rn(bf16hi(rw[j]), __fmul_rn(bf16hi(w), v[2 * j + 1]));
      }
    }
  }
  if (!store) {  // (the values still have to be worked out: see the caller)
#pragma unroll
    for (int j = 0; j < 16; ++j) asm volatile("" ::"f"(v[j]));
    return;
  }
  if (g.c_dtype == QB_BF16) {
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
    uint4* d = reinterpret_cast<uint4*>(c_row + 2 * n);
    if (wide) {
      st_global_v8(d, w);
    } else {
      d[0] = make_uint4(w[0], w[1], w[2], w[3]);
      if (second) d[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  } else if (g.c_dtype == QB_E4M3) {
    if (g.through_bf16) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __bfloat162float(__float2bfloat16_rn(v[j]));
    }
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = pack_e4m3x4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    if (wide) {
      *reinterpret_cast<uint4*>(c_row + n) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      *reinterpret_cast<uint2*>(c_row + n) = make_uint2(w[0], w[1]);
      if (second) *reinterpret_cast<uint2*>(c_row + n + 8) = make_uint2(w[2], w[3]);
    }
  } else {
    float4* d = reinterpret_cast<float4*>(c_row + 4 * n);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < 2 || second) d[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  }
}

// ---------------------------------------------------------------- fused epilogue of the QKV projection
// The accumulator tile (BN / 64 heads) goes through shared memory to a layout of four threads per (token, head), 16 elements
// each: a warp then reads and writes 128-byte rows, the head's sum of squares is two shuffles, and each thread needs four
// cosines and four sines.  Arithmetic, rounding points and summation order are those of qkv_post.cu (and through it of
// head_rmsnorm, value_residual_packed and kv_cache_update), so the bytes written are the same.  V is transposed through
// shared memory, two channels at a time.
// What bounds it is the chain of one round (about 0.4 us for a Q head: sum, shuffles, square root, reciprocal) and, before this
// was a loop, fetching its instructions: they run once per launch, after other kernels have had the instruction caches.  In a
// frame the rounds unrolled, with the divisions by run-time sizes and the loads of the cache scales in each of them, took 4.9 us
// (Q heads 4.5, V heads 7.9) at 720p bf16 and 3.2 (V heads 5.2) at 360p; as a loop on shifts, with what the rounds share
// prepared while the main loop runs, 2.4 (2.1, 3.8) and 2.5 (2.8).  Two rounds side by side were slower again (2.7): more
// instructions.

struct QkvFrame {  // where this frame's rows go
  int ft, slot, L, cap, tpf_c;
  bool ring;
};
__device__ __forceinline__ QkvFrame qkv_frame(const QkvTail& q) {
  QkvFrame f;
  f.ft = *after_wait(q.frame_t);  // written on the device: ordinary loads, after the grid dependency
  f.tpf_c = q.tpf / q.quilt;      // tokens of a frame that the cache keeps
  f.L = q.nb * f.tpf_c;
  f.cap = f.L + f.tpf_c;
  f.slot = (f.ft + q.pd - 1) / q.pd % q.nb;
  f.ring = f.ft % q.pd == 0 && *after_wait(q.frozen) == 0;
  return f;
}

// One thread of the grid writes the segment table.
__device__ __forceinline__ void qkv_segments(const QkvTail& q, const QkvFrame& f) {
  const int bucket = (f.ft + q.pd - 1) / q.pd;
  int sg[6] = {0, 0, 0, 0, 0, 0};
  int n = 2;
  if (f.ft % q.pd == 0 && bucket >= q.nb) {
    sg[1] = f.slot * f.tpf_c;
    sg[2] = (f.slot + 1) * f.tpf_c;
    sg[3] = (q.nb - f.slot - 1) * f.tpf_c;
    sg[4] = f.L;
    sg[5] = f.tpf_c;
    n = 3;
  } else {
    sg[1] = min(bucket, q.nb) * f.tpf_c;
    sg[2] = f.L;
    sg[3] = f.tpf_c;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i)
    if (i < 2 * q.max_segments) q.segments[i] = sg[i];
  for (int i = 6; i < 2 * q.max_segments; ++i) q.segments[i] = 0;
  q.n_segments[0] = n;
}

__device__ __forceinline__ int qkv_kind(const QkvTail& q, int col) {  // 0 Q, 1 K, 2 V
  return col < q.n_q_heads * 64 ? 0 : col < (q.n_q_heads + q.n_kv_heads) * 64 ? 1 : 2;
}

__device__ __forceinline__ int log2i(int x) { return 31 - __clz(x); }  // x: a power of two

// What the rounds of qkv_finish share, in shared memory before the main loop ends: the frame's temporal cosines and sines, the
// reciprocals of the cache scales of the tile's heads (1 without scales: multiplying by it changes no bit) and the mix factor.
struct QkvShared {
  float tm[16], inv[2], lam;
};
template <int BN>
__device__ __forceinline__ void qkv_share(const QkvTail& q, const QkvFrame& f, int et, int n0, QkvShared* sh) {
  if (et < 8) temporal_cos_sin(f.ft, et, sh->tm);
  if (et >= 32 && et < 32 + BN / 64) {
    const int head = (n0 >> 6) + et - 32 - q.n_q_heads, vh = head - q.n_kv_heads;
    const float* sc = vh >= 0 ? q.v_scale : q.k_scale;
    sh->inv[et - 32] = sc != nullptr && head >= 0 && vh < q.n_kv_heads ? __fdiv_rn(1.0f, __ldg(sc + (vh >= 0 ? vh : head))) : 1.0f;
  }
  if (et == 64) sh->lam = q.qkv_first != nullptr ? *after_wait(q.lamb) : 0.f;
}

// What round k of qkv_finish needs from global memory: cosines and sines of a K head's positions, or the first block's V.
template <int BN>
__device__ __forceinline__ void qkv_fetch(const GemmArgs& g, int et, int row0, int rows, int m0, int n0, int k, uint4 (&pre)[2]) {
  const QkvTail& q = g.qkv;
  pre[0] = pre[1] = make_uint4(0u, 0u, 0u, 0u);
  const int idx = et + 256 * k, l = idx & 3, rh = idx >> 2;
  const int hd = rh >> log2i(rows), t = m0 + row0 + (rh & (rows - 1)), col = n0 + hd * 64;
  if (hd >= BN / 64 || t >= g.M || col >= g.N) return;
  const int kind = qkv_kind(q, col);
  if (kind == 1 && l < 2) {
    const uint4* rp = reinterpret_cast<const uint4*>(after_wait(q.rope_xy) + static_cast<size_t>(t) * 16);
    pre[0] = rp[l];
    pre[1] = rp[2 + l];
  } else if (kind == 2 && q.qkv_first != nullptr) {  // written earlier in this pass
    const uint4* fp = reinterpret_cast<const uint4*>(after_wait(q.qkv_first) + static_cast<size_t>(t) * g.N + col + 16 * l);
    pre[0] = fp[0];
    pre[1] = fp[1];
  }
}

// Rows [row0, row0 + rows) of the tile to the packed QKV and the caches.  One K slice: the tile is in `vt` (pitch BN + 8); S
// slices: the partial sums are in `partials` and `vt` (pitch 72) takes the V rows.  `col` holds the tile's per-column scales, `sh`
// what qkv_share left there, `pre` the first two rounds' qkv_fetch.  Run by the 256 epilogue threads together.
template <int BN, bool kCacheFp8>
__device__ __forceinline__ void qkv_finish(const GemmArgs& g, const float4* partials, uint16_t* vt, const float* col, const QkvShared* sh, const QkvFrame& fr, int splits, int row0,
                                           int rows, int m0, int n0, uint4 (&pre)[2][2]) {
  constexpr int kEs = kCacheFp8 ? 1 : 2;
  const QkvTail& q = g.qkv;
  const int et = threadIdx.x - 64, lrows = log2i(rows), lquilt = log2i(q.quilt);
  const int k_off = q.n_q_heads * 64, v_off = (q.n_q_heads + q.n_kv_heads) * 64;
  const bool mix = q.qkv_first != nullptr;
  const float lam = sh->lam;
  const int vpitch = splits == 1 ? BN + 8 : 72;
  const int rounds = max(rows * (BN / 64) / 64, 1);
#pragma unroll 1
  for (int k = 0; k < rounds; ++k) {
    const uint4 p0 = pre[0][0], p1 = pre[0][1];
    pre[0][0] = pre[1][0];
    pre[0][1] = pre[1][1];
    if (k + 2 < rounds) qkv_fetch<BN>(g, et, row0, rows, m0, n0, k + 2, pre[1]);
    const int idx = et + 256 * k, l = idx & 3, rh = idx >> 2;
    const int hd = rh >> lrows, row = rh & (rows - 1), t = m0 + row0 + row, c0 = n0 + hd * 64;
    if (hd >= BN / 64 || c0 >= g.N) continue;  // uniform over the warp
    const int kind = qkv_kind(q, c0);
    uint16_t* staged = vt + row * vpitch + hd * 64 + 16 * l;
    float f[16];
    if (splits == 1) {  // already scaled and rounded
      const uint4 a = *reinterpret_cast<const uint4*>(staged), b = *reinterpret_cast<const uint4*>(staged + 8);
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        f[2 * j] = bf16lo(w[j]);
        f[2 * j + 1] = bf16hi(w[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) f[j] = 0.f;
      for (int s = 0; s < splits; ++s) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const float4 x = partials[slice_unit<BN>(s, hd * 16 + 4 * l + v, row, rows)];
          f[4 * v] += x.x; f[4 * v + 1] += x.y; f[4 * v + 2] += x.z; f[4 * v + 3] += x.w;
        }
      }
      const bool scaled = g.a_scale != nullptr || g.w_scale != nullptr;
#pragma unroll
      for (int j = 0; j < 16; ++j) f[j] = __bfloat162float(__float2bfloat16_rn(scaled ? f[j] * col[hd * 64 + 16 * l + j] : f[j]));
    }
    uint32_t o[8];  // the 16 elements as they go to qkv_out
    if (kind < 2) {
      float sa = 0.f, sb = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) sa += f[j] * f[j];
#pragma unroll
      for (int j = 8; j < 16; ++j) sb += f[j] * f[j];
      float ss = sa + sb;
      ss += __shfl_xor_sync(0xffffffffu, ss, 1);
      ss += __shfl_xor_sync(0xffffffffu, ss, 2);
      const float inv = 1.0f / sqrtf(ss * (1.0f / 64.0f) + q.eps);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = pack_bf16x2(__fmul_rn(f[2 * j], inv), __fmul_rn(f[2 * j + 1], inv));
    } else if (mix) {
      const uint32_t vf[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = f[2 * j], b = f[2 * j + 1];
        o[j] = pack_bf16x2(__fadd_rn(a, __fmul_rn(lam, __fsub_rn(bf16lo(vf[j]), a))), __fadd_rn(b, __fmul_rn(lam, __fsub_rn(bf16hi(vf[j]), b))));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = pack_bf16x2(f[2 * j], f[2 * j + 1]);
    }
    if (kind == 2) {
      *reinterpret_cast<uint4*>(staged) = make_uint4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<uint4*>(staged + 8) = make_uint4(o[4], o[5], o[6], o[7]);
    }
    if (t >= g.M) continue;
    st_global_v8(static_cast<uint16_t*>(g.C) + static_cast<size_t>(t) * g.N + c0 + 16 * l, o);
    const int tq = t - q.qoff;
    if (kind == 1 && tq >= 0 && (tq & (q.quilt - 1)) == 0) {  // this token is one of those the cache keeps
      // rotate what the stand-alone append would read back (the bf16-rounded normalised K): thread l holds pairs 8 l .. 8 l + 7,
      // whose angles are 4 (x, y, or half of the temporal ones); a cache row is the pairs' first outputs, then their second
      const int head = (c0 - k_off) >> 6, tc = tq >> lquilt;
      const float inv_k = sh->inv[hd];
      float cs[4], sn[4];
      if (l < 2) {
        cs[0] = __uint_as_float(p0.x); cs[1] = __uint_as_float(p0.y); cs[2] = __uint_as_float(p0.z); cs[3] = __uint_as_float(p0.w);
        sn[0] = __uint_as_float(p1.x); sn[1] = __uint_as_float(p1.y); sn[2] = __uint_as_float(p1.z); sn[3] = __uint_as_float(p1.w);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          cs[i] = sh->tm[4 * (l - 2) + i];
          sn[i] = sh->tm[8 + 4 * (l - 2) + i];
        }
      }
      float y0[8], y1[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x0 = bf16lo(o[j]), x1 = bf16hi(o[j]);
        y0[j] = __fmul_rn(__fsub_rn(__fmul_rn(x0, cs[j >> 1]), __fmul_rn(x1, sn[j >> 1])), inv_k);
        y1[j] = __fmul_rn(__fadd_rn(__fmul_rn(x1, cs[j >> 1]), __fmul_rn(x0, sn[j >> 1])), inv_k);
      }
      uint8_t* kc = static_cast<uint8_t*>(q.K_cache);
      uint8_t* tail = kc + (static_cast<size_t>(head) * fr.cap + fr.L + tc) * (64 * kEs) + l * (8 * kEs);
      uint8_t* rr = kc + (static_cast<size_t>(head) * fr.cap + static_cast<size_t>(fr.slot) * fr.tpf_c + tc) * (64 * kEs) + l * (8 * kEs);
      if (kCacheFp8) {
        const uint2 w0 = make_uint2(pack_e4m3x4(y0[0], y0[1], y0[2], y0[3]), pack_e4m3x4(y0[4], y0[5], y0[6], y0[7]));
        const uint2 w1 = make_uint2(pack_e4m3x4(y1[0], y1[1], y1[2], y1[3]), pack_e4m3x4(y1[4], y1[5], y1[6], y1[7]));
        *reinterpret_cast<uint2*>(tail) = w0;
        *reinterpret_cast<uint2*>(tail + 32) = w1;
        if (fr.ring) {
          *reinterpret_cast<uint2*>(rr) = w0;
          *reinterpret_cast<uint2*>(rr + 32) = w1;
        }
      } else {
        const uint4 w0 = make_uint4(pack_bf16x2(y0[0], y0[1]), pack_bf16x2(y0[2], y0[3]), pack_bf16x2(y0[4], y0[5]), pack_bf16x2(y0[6], y0[7]));
        const uint4 w1 = make_uint4(pack_bf16x2(y1[0], y1[1]), pack_bf16x2(y1[2], y1[3]), pack_bf16x2(y1[4], y1[5]), pack_bf16x2(y1[6], y1[7]));
        *reinterpret_cast<uint4*>(tail) = w0;
        *reinterpret_cast<uint4*>(tail + 64) = w1;
        if (fr.ring) {
          *reinterpret_cast<uint4*>(rr) = w0;
          *reinterpret_cast<uint4*>(rr + 64) = w1;
        }
      }
    }
  }
  if (min(n0 + BN, g.N) <= v_off) return;  // no V head in this tile (the same for all threads)
  asm volatile("bar.sync 2, 256;" ::: "memory");
  // transposed 16-byte stores, two channels x (8 | 16) consecutive cached tokens per thread, neighbouring threads taking
  // neighbouring token vectors so that whole 32-byte sectors are written.  The tile's cached tokens are its rows qoff,
  // qoff + quilt, ... (m0 + row0 is a multiple of the quilt factor).
  constexpr int kTokPerVec = 16 / kEs;
  const int vec_per_ch = (rows >> lquilt) / kTokPerVec;
  const int ljw = vec_per_ch > 1 ? 1 : 0;  // two vectors (a whole sector) side by side where there are two
  uint8_t* vc = static_cast<uint8_t*>(q.Vt_cache);
#pragma unroll 1
  for (int hd = 0; hd < BN / 64; ++hd) {
    const int c0 = n0 + hd * 64;
    if (c0 < v_off || c0 >= g.N) continue;
    const int head = (c0 - v_off) >> 6;
    const float inv_v = sh->inv[hd];
    const uint16_t* src = vt + hd * 64;
#pragma unroll 1
    for (int v = et; v < 32 * vec_per_ch; v += 256) {
      const int d = ((v >> ljw) & 31) * 2, j = ((v >> (5 + ljw)) << ljw) + (v & ljw);
      const int c1 = j * kTokPerVec;                      // first cached token of the vector, inside these rows
      const int c_abs = ((m0 + row0) >> lquilt) + c1;       // ... and inside the frame's cached tokens
      if (c_abs + kTokPerVec > fr.tpf_c) continue;
      uint32_t x[kTokPerVec];
#pragma unroll
      for (int i = 0; i < kTokPerVec; ++i) x[i] = *reinterpret_cast<const uint32_t*>(src + (q.qoff + ((c1 + i) << lquilt)) * vpitch + d);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t w[4];
        if (kCacheFp8) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float e[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) e[b] = __fmul_rn(h == 0 ? bf16lo(x[(4 * i + b) % kTokPerVec]) : bf16hi(x[(4 * i + b) % kTokPerVec]), inv_v);
            w[i] = pack_e4m3x4(e[0], e[1], e[2], e[3]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t a = x[2 * i], b = x[2 * i + 1];
            if (q.v_scale != nullptr)
              w[i] = h == 0 ? pack_bf16x2(__fmul_rn(bf16lo(a), inv_v), __fmul_rn(bf16lo(b), inv_v)) : pack_bf16x2(__fmul_rn(bf16hi(a), inv_v), __fmul_rn(bf16hi(b), inv_v));
            else
              w[i] = h == 0 ? __byte_perm(a, b, 0x5410) : __byte_perm(a, b, 0x7632);
          }
        }
        const uint4 ov = make_uint4(w[0], w[1], w[2], w[3]);
        const size_t ch = (static_cast<size_t>(head) * 64 + d + h) * fr.cap;
        *reinterpret_cast<uint4*>(vc + (ch + fr.L + c_abs) * kEs) = ov;
        if (fr.ring) *reinterpret_cast<uint4*>(vc + (ch + static_cast<size_t>(fr.slot) * fr.tpf_c + c_abs) * kEs) = ov;
      }
    }
  }
}

struct GemmPlan {
  int cg;  // CTAs per tile: 1 (gemm.cu) or a pair (gemm_pair.cu)
  int bn, splits, kb_total, kb_per_split;
  int cluster;  // slices summed inside a thread-block cluster instead of through the workspace
  size_t counters_bytes, aq_bytes, partial_bytes;
};

// Tensor maps and launch of the grouped kernel, and of the pair kernel for a plan with cg == 2.
int32_t launch_gemm_grouped(int bn, const void* A, const void* B, int n_experts, const GemmArgs& g, bool fp8, cudaStream_t st);
int32_t launch_gemm_pair(const GemmPlan& pl, const void* A, const void* B, const GemmArgs& g, bool fp8, cudaStream_t st);
int32_t make_tmap_2d_sw(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols,
                        int swizzle_bytes);

}  // namespace qb
