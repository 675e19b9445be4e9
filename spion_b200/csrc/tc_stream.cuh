// What the streaming kernels (tc_fwd_stream.cu, tc_bwd_stream.cu) share: the order in which a CTA walks its lines (block rows or
// block columns) and the pairs of entries of a line.
#pragma once
#include "tc_tiles.cuh"

namespace tc {

// Unit ordinal -> (b,h) matrix and rank of its line.  by_rank: the longest lines of all matrices first (even shares of long and
// short lines); else matrix by matrix, so that tiles shared by the lines of a matrix stay in L2, the lines rotated from matrix to
// matrix so that no CTA meets the long ones every time.
struct UnitMap {
  int nb, BH, by_rank;
  __device__ __forceinline__ void at(int u, int& bh, int& rank) const {
    if (by_rank) { rank = u / BH; bh = u - rank * BH; }
    else { bh = u / nb; rank = u - bh * nb + bh % nb; if (rank >= nb) rank -= nb; }
  }
};
// The streamed matrices of all (b,h) pairs stay in L2 (126 MB) whatever the order of the lines; beyond that the order has to keep the
// lines of one matrix together.
inline int order_by_rank(const spion_ctx* c) { return (size_t)2 * c->BH * c->L * c->d * 2 <= (size_t)80 << 20; }

// A walk over units first, first + step, ... < total: unit ordinal i, pair k of its line.  The record of the next unit is requested a
// unit early.  rec[rank] = {line, first pair, pairs, entries}.
struct Walk {
  UnitMap um;
  const int4* rec;
  int first, step, n_my;                              // units of this walk
  int i, k, bh, bh_n;
  int4 cur, nxt;
  __device__ __forceinline__ int4 record(int x, int& b) const {
    if (x >= n_my) { b = 0; return make_int4(0, 0, 0, 0); }
    int rank;
    um.at(first + x * step, b, rank);
    return rec[rank];
  }
  __device__ __forceinline__ void init(const UnitMap& m, const int4* r, int f, int s, int total) {
    um = m; rec = r; first = f; step = s;
    n_my = total > f ? (total - f + s - 1) / s : 0;
    i = 0; k = 0;
    cur = record(0, bh);
    nxt = record(1, bh_n);
  }
  __device__ __forceinline__ bool valid() const { return i < n_my; }
  __device__ __forceinline__ int pairs() const { return cur.z; }
  __device__ __forceinline__ int cnt() const { return min(2, cur.w - 2 * k); }          // entries of pair k
  __device__ __forceinline__ bool last() const { return k + 1 == cur.z; }
  __device__ __forceinline__ void shift() { ++i; k = 0; cur = nxt; bh = bh_n; nxt = record(i + 1, bh_n); }
  __device__ __forceinline__ void skip() { while (i < n_my && cur.w == 0) shift(); }      // lines without entries
  __device__ __forceinline__ void next() { if (++k >= cur.z) { shift(); skip(); } }
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two fp32 values per instruction, each rounded as fmaf / + would; three-way maximum.
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint64_t pack2(float a, float b) { return pack2(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint32_t (&w)[4]) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// Raw scores of 32 keys with their penalties: (s - pad / scale) scale = s scale - pad.  Done in place, in the few blocks whose keys
// have different ones, so that the arithmetic behind it has one form only (two forms cost 20 % of the forward in registers).
__device__ __forceinline__ void take_penalty(uint32_t (&s)[32], const float* kp, float inv_scale) {
#pragma unroll
  for (int x = 0; x < 32; ++x) s[x] = __float_as_uint(fmaf(kp[x], -inv_scale, __uint_as_float(s[x])));
}

// The penalties of a block's 64 keys: one value for all of them (zero: no padded keys), or different ones.  Padding is a tail of the
// sequence, so a block in which they differ is one per sequence; all others take the value with the row's constant, not key by key (256 matrices,
// L = 4096, d 32, 10 %, 25 % of the keys padded: forward, columns, rows 224, 335, 298 us with a penalty per key of every padded block).
// Half a warp, four keys per lane: pen_load is requested early, pen_of gives the block's value and whether a key differs from it.
struct Pen4 { float x[4]; };
__device__ __forceinline__ void pen_load(Pen4& p, const float* lo, const float* hi) {       // of the first and the second 32 keys
#pragma unroll
  for (int i = 0; i < 4; ++i) p.x[i] = (i < 2 ? lo : hi)[(threadIdx.x & 15) + 16 * (i & 1)];
}
__device__ __forceinline__ void pen_load(Pen4& p, const float* kp) { pen_load(p, kp, kp + 32); }
__device__ __forceinline__ float pen_of(const Pen4& p, uint32_t& mixed) {      // whole warp; mixed: bit 0, lanes 0-15, bit 1, lanes 16-31
  const float first = __shfl_sync(0xffffffffu, p.x[0], threadIdx.x & 16);
  bool other = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) other |= p.x[i] != first;           // a NaN differs from itself
  const uint32_t all = __ballot_sync(0xffffffffu, other);
  mixed = ((all & 0xffffu) ? 1u : 0u) | ((all >> 16) ? 2u : 0u);
  return first;
}

}  // namespace tc
