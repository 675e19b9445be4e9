// Fused fp32 kernels of the block-sparse attention path on the CUDA cores: the calls with too little work for those of mma_fused.cu (see
// use_mma below).  Fusing removes the S / dP round trips through memory that the staged kernels of simt_attn.cu make.
//
//   fused_fwd_kernel   per block row:  S = Q K^T -> sparse row softmax -> P (written once) -> O = P V
//                      replaces models/block_attn.cu:453-487 (cusparseSDDMM, scale_softmax_kernel, cusparseSpMM)
//   fused_bwd_row      per block row:  dP = dO V^T -> dS = (dP.P - P rowsum(dP.P)) scale -> dQ = dS K
//                      replaces models/block_attn.cu:498-516
//   fused_bwd_col      per block col:  dK = dS^T Q, dV = P^T dO      (models/block_attn.cu:526-536)
//
// A row of blocks can be arbitrarily long, so nothing but one tile is ever held on chip: pass 1 of the
// forward kernel leaves the scaled scores in the P tiles themselves (global memory, normally still in
// L2 when they are read back) while it accumulates the row maximum and denominator on line; pass 2
// reads them back, writes the probabilities over them and feeds the second product.  The backward
// row kernel does the same with dP in the dS tiles.
//
// Bound by latencies at these sizes, and by the FMA pipes: scalar multiply-adds reach 47 TFLOP/s on this chip (register ports) and packed
// pairs 61, so the loops use pairs.  A bs x bs tile is computed by bs^2 / 16 threads with 4 x 4 micro-tiles.  The threads of one (b,h)
// matrix run on their own, with a barrier of their own.  Tiles are unpadded, the 16-byte pieces of row i exchanged by i / 4 (mod 8): a
// thread owns contiguous rows and four contiguous columns, so value tiles move in 16-byte pieces, and the reads take no bank twice.
//
// Layouts: operands through (row, column) strides, value tiles through tile_address(); only
// layouts whose tile rows are contiguous (element CSR, block tiles) are accepted.
#include <cooperative_groups.h>

#include <atomic>

#include "fp32_tiles.cuh"

using namespace fp32;

namespace {

// R: rows of a tile per thread
template <int BS, int D, int R>
struct Cfg {
  static constexpr int TX = BS / 4;            // threads along a tile row
  static constexpr int NT = BS * BS / (4 * R); // threads per (b,h) problem
  static constexpr int CTA = NT > 128 ? NT : 128;
  static constexpr int G = CTA / NT;           // problems per CTA
  static constexpr int TN = D / TX;            // output columns per thread in the bs x d products
  static constexpr int TILE = BS * D;          // floats of an operand tile
  static constexpr int VALS = BS * BS;         // ... of a value tile
  static constexpr int RESIDENT = 2;           // CTAs per SM
  static_assert(TN == 2 || TN == 4 || TN == 8, "unsupported shape");
};

// A CTA has W > 1 groups of NT threads that share a block row, or (W == 1) G groups with a problem each.
template <int BS, int D, int R, int W> constexpr int cta_threads() { return W > 1 ? W * Cfg<BS, D, R>::NT : Cfg<BS, D, R>::CTA; }
template <int BS, int D, int R, int W> constexpr int cta_groups() { return W > 1 ? W : Cfg<BS, D, R>::G; }
template <int BS, int D, int R, int W> constexpr int cta_resident(int n) { return W > 1 ? 512 / (W * Cfg<BS, D, R>::NT) : n; }

// float offset of 16-byte piece `piece` of row `row` in a tile of COLS columns
template <int COLS>
__device__ __forceinline__ int at(int row, int piece) { return row * COLS + ((piece ^ ((row >> 2) & 7)) << 2); }
struct Swizzle {
  template <int COLS>
  static __device__ __forceinline__ int at(int row, int piece) { return ::at<COLS>(row, piece); }
};

// column of the thread's y-th output in a bs x d product: groups of 4 (or 2) contiguous columns
template <int BS, int D, int R>
__device__ __forceinline__ int out_col(int tx, int y) {
  using C = Cfg<BS, D, R>;
  if (C::TN == 2) return tx * 2 + y;
  return (y >> 2) * (C::TX * 4) + tx * 4 + (y & 3);
}

// the thread's columns of row `row` of a [bs x d] tile
template <int BS, int D, int R>
__device__ __forceinline__ void load_vec(const float* tile, int row, int tx, float (&b)[Cfg<BS, D, R>::TN]) {
  using C = Cfg<BS, D, R>;
  if constexpr (C::TN == 2) {
    const float2 v = *reinterpret_cast<const float2*>(tile + at<D>(row, tx >> 1) + (tx & 1) * 2);
    b[0] = v.x; b[1] = v.y;
  } else {
#pragma unroll
    for (int g4 = 0; g4 < C::TN / 4; ++g4) {
      const float4 v = *reinterpret_cast<const float4*>(tile + at<D>(row, g4 * C::TX + tx));
      b[4 * g4] = v.x; b[4 * g4 + 1] = v.y; b[4 * g4 + 2] = v.z; b[4 * g4 + 3] = v.w;
    }
  }
}

// Packed pairs of fp32: one instruction, two multiply-adds per lane.  The FMA pipe is no faster for it, but the loops below were
// limited by issue slots (two multiply-adds in three instructions).
using pair_t = unsigned long long;
__device__ __forceinline__ pair_t pack2(float x, float y) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(pair_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(pair_t& acc, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
struct Quad { pair_t lo, hi; };
__device__ __forceinline__ Quad load_quad(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return Quad{v.x, v.y};
}

// out[x][y] = sum_n A[row0+x][n] * B[tx*4+y][n], x = 0..3   (both tiles [bs x d] in shared memory; row0 a multiple of four; even and
// odd n in one sum each).
template <int BS, int D>
__device__ __forceinline__ void tile_abt(const float* As, const float* Bs, int row0, int tx, float (&out)[4][4]) {
  pair_t acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = 0ull;
#pragma unroll 2
  for (int n = 0; n < D / 4; ++n) {
    Quad a[4], b[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) b[y] = load_quad(Bs + at<D>(tx * 4, n) + y * D);
#pragma unroll
    for (int x = 0; x < 4; ++x) a[x] = load_quad(As + at<D>(row0, n) + x * D);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) fma2(acc[x][y], a[x].lo, b[y].lo);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) fma2(acc[x][y], a[x].hi, b[y].hi);
  }
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const float2 v = unpack2(acc[x][y]);
      out[x][y] = v.x + v.y;
    }
}

// The thread's R x TN sums of a bs x d product, rows in pairs: v[x][y] = (row ty*R + 2 x, row ty*R + 2 x + 1), column out_col(y).
template <int BS, int D, int R>
struct Sums {
  pair_t v[R / 2][Cfg<BS, D, R>::TN];
  __device__ __forceinline__ Sums() {
#pragma unroll
    for (int x = 0; x < R / 2; ++x)
#pragma unroll
      for (int y = 0; y < Cfg<BS, D, R>::TN; ++y) v[x][y] = 0ull;
  }
};

// W groups: the first adds the sums of the others, in their order.  `place`: this group's shared memory, bs x d floats that nobody reads
// any more once every thread of the group is here.
template <int BS, int D, int R, int W>
__device__ __forceinline__ void join_sums(float* place, int group_floats, int g, int t, Sums<BS, D, R>& s) {
  using C = Cfg<BS, D, R>;
  constexpr int NT = C::NT;
  pair_t* mine = reinterpret_cast<pair_t*>(place) + t;            // pair i of thread t at i * NT + t
  if (g > 0) {
#pragma unroll
    for (int x = 0; x < R / 2; ++x)
#pragma unroll
      for (int y = 0; y < C::TN; ++y) mine[(x * C::TN + y) * NT] = s.v[x][y];
  }
  __syncthreads();
  if (g == 0) {
#pragma unroll
    for (int q = 1; q < W; ++q) {
      const pair_t* theirs = reinterpret_cast<const pair_t*>(place + q * group_floats) + t;
#pragma unroll
      for (int x = 0; x < R / 2; ++x)
#pragma unroll
        for (int y = 0; y < C::TN; ++y) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s.v[x][y]) : "l"(theirs[(x * C::TN + y) * NT]));
    }
  }
}

// acc += sum_i Vt[i][rows] * B[i][columns]   (Vt: [bs x bs] value tile, transposed use; B: [bs x d])
template <int BS, int D, int R>
__device__ __forceinline__ void tile_atb(const float* Vt, const float* Bs, int ty, int tx, Sums<BS, D, R>& acc) {
  using C = Cfg<BS, D, R>;
#pragma unroll 4
  for (int i = 0; i < BS; ++i) {
    pair_t a[R / 2];
#pragma unroll
    for (int x = 0; x < R / 4; ++x) {
      const Quad v = load_quad(Vt + at<BS>(i, R / 4 * ty + x));
      a[2 * x] = v.lo;
      a[2 * x + 1] = v.hi;
    }
    float b[C::TN];
    load_vec<BS, D, R>(Bs, i, tx, b);
#pragma unroll
    for (int y = 0; y < C::TN; ++y) {
      const pair_t bb = pack2(b[y], b[y]);
#pragma unroll
      for (int x = 0; x < R / 2; ++x) fma2(acc.v[x][y], a[x], bb);
    }
  }
}

// Four rows of the thread's values of a tile into shared memory, transposed (16-byte piece `piece` of each row there), so that tile_atb multiplies with the tile itself.
template <int BS>
__device__ __forceinline__ void put_transposed(float* Vt, int piece, int tx, const float (&v)[4][4]) {
#pragma unroll
  for (int y = 0; y < 4; ++y)
    *reinterpret_cast<float4*>(Vt + at<BS>(tx * 4 + y, piece)) = make_float4(v[0][y], v[1][y], v[2][y], v[3][y]);
}

template <int TX>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = TX / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int TX>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = TX / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// store the thread's R x TN outputs of a bs x d product
template <int BS, int D, int R>
__device__ __forceinline__ void store_out(float* __restrict__ out, OperandLayout lo, int row0, int ty, int tx,
                                          const Sums<BS, D, R>& sums) {
  using C = Cfg<BS, D, R>;
  float acc[R][C::TN];
#pragma unroll
  for (int x = 0; x < R / 2; ++x)
#pragma unroll
    for (int y = 0; y < C::TN; ++y) {
      const float2 v = unpack2(sums.v[x][y]);
      acc[2 * x][y] = v.x;
      acc[2 * x + 1][y] = v.y;
    }
  const bool vec = lo.sd == 1 && (lo.sl & 3) == 0 && vec_ok(out);
#pragma unroll
  for (int x = 0; x < R; ++x) {
    float* o = out + (long long)(row0 + ty * R + x) * lo.sl;
    if (C::TN >= 4 && vec) {
#pragma unroll
      for (int g4 = 0; g4 < C::TN / 4; ++g4)
        *reinterpret_cast<float4*>(o + out_col<BS, D, R>(tx, 4 * g4)) =
            make_float4(acc[x][4 * g4], acc[x][4 * g4 + 1], acc[x][4 * g4 + 2], acc[x][4 * g4 + 3]);
    } else {
#pragma unroll
      for (int y = 0; y < C::TN; ++y) o[(long long)out_col<BS, D, R>(tx, y) * lo.sd] = acc[x][y];
    }
  }
}

// Shared memory of the two-pass kernels: the row's own operand (pass 1) and the value tile (pass 2) take turns.
template <int BS, int D, int R> constexpr int ONE = Cfg<BS, D, R>::TILE > Cfg<BS, D, R>::VALS ? Cfg<BS, D, R>::TILE : Cfg<BS, D, R>::VALS;
template <int BS, int D, int R> __host__ __device__ constexpr int two_pass_floats() { return ONE<BS, D, R> + 2 * Cfg<BS, D, R>::TILE; }

// ------------------------------------------------------------------------------ forward
//   v = S*scale - keypad[col];  m = max(floor, max v);  Z = sum exp(v-m) + (L-n_i) exp(-m);  P = exp(v-m)/Z
// The K (pass 1) and V (pass 2) tiles are double-buffered: the copy of tile k+1 is in flight while
// tile k is used.  Every thread keeps the maximum and the sum of its own columns of a row; the threads of a row join them
// once, after the last tile.
// W > 1: W groups of threads take a share of the row's blocks each; maxima and denominators are joined between the passes, O at the end.
template <int BS, int D, int R, int W>
__global__ void __launch_bounds__(cta_threads<BS, D, R, W>(), cta_resident<BS, D, R, W>(Cfg<BS, D, R>::RESIDENT)) fused_fwd_kernel(const float* __restrict__ Q, OperandLayout lq,
                                                           const float* __restrict__ K, OperandLayout lk,
                                                           const float* __restrict__ V, OperandLayout lv,
                                                           const float* __restrict__ keypad, float floor_v, float* P,
                                                           ValueLayout vl, float* __restrict__ O, OperandLayout lo,
                                                           Pattern p, int BH, int L, float scale) {
  using C = Cfg<BS, D, R>;
  extern __shared__ __align__(16) float smem[];
  const int g = threadIdx.x / C::NT, t = threadIdx.x % C::NT;
  const int ty = t / C::TX, tx = t % C::TX;
  const int r = blockIdx.x, bh = W > 1 ? blockIdx.y : blockIdx.y * C::G + g;
  if (bh >= BH) return;
  float* Qs = smem + g * two_pass_floats<BS, D, R>();
  float* Bs = Qs + ONE<BS, D, R>;                                // two buffers: K tiles, then V tiles
  float* Ps = Qs;                                               // pass 2

  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const int* cols = p.col_idx + rp;
  const int k0 = W > 1 ? nblk * g / W : 0, k1 = W > 1 ? nblk * (g + 1) / W : nblk;      // this group's blocks
  const Operand Kb(K, lk, bh), Vb(V, lv, bh);
  float* Pb = P + (long long)bh * vl.bh_stride;
  const float* kp = keypad ? keypad + (long long)bh * L + tx * 4 : nullptr;
  const bool vec = vec_ok(Pb);
  const RowTiles rt = RowTiles::of<BS>(vl, rp, nblk);
  float* mine = Pb + rt.base + ty * R * rt.si + tx * 4;         // the thread's values of the row's first tile
  const float scale2 = scale * LOG2_E;                          // scores in base-2 units

  int c_cur = k0 < k1 ? cols[k0] : 0, c_nxt = k0 + 1 < k1 ? cols[k0 + 1] : 0;
  load_tile<Swizzle, BS, D, C::NT>(Qs, Operand(Q, lq, bh), r * BS, t);
  if (k0 < k1) load_tile<Swizzle, BS, D, C::NT>(Bs + (k0 & 1) * C::TILE, Kb, c_cur * BS, t);
  cp_async_commit();

  // ---- pass 1: scores into the P tiles, running maximum and denominator per row
  float m[R], l[R];
#pragma unroll
  for (int x = 0; x < R; ++x) { m[x] = floor_v * LOG2_E; l[x] = 0.f; }
  for (int k = k0; k < k1; ++k) {
    const int c = c_cur;
    if (k + 1 < k1)
      load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Kb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < k1 ? cols[k + 2] : 0;
    float pad[4] = {0.f, 0.f, 0.f, 0.f};
    if (kp) {
#pragma unroll
      for (int y = 0; y < 4; ++y) pad[y] = kp[c * BS + y] * LOG2_E;
    }
    cp_async_wait<1>();
    group_sync<C::NT>(g);                                        // tile k (and Q) have landed
    float* tile = mine + (long long)k * rt.step;
#pragma unroll
    for (int half = 0; half < R / 4; ++half) {
      float acc[4][4];
      tile_abt<BS, D>(Qs, Bs + (k & 1) * C::TILE, ty * R + half * 4, tx, acc);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float &mx = m[half * 4 + x], &lx = l[half * 4 + x];
#pragma unroll
        for (int y = 0; y < 4; ++y) acc[x][y] = fmaf(acc[x][y], scale2, -pad[y]);
        store_vals(tile + (half * 4 + x) * rt.si, make_float4(acc[x][0], acc[x][1], acc[x][2], acc[x][3]), vec);
        const float m_new = fmaxf(mx, fmaxf(fmaxf(acc[x][0], acc[x][1]), fmaxf(acc[x][2], acc[x][3])));
        const float s = (ex2(acc[x][0] - m_new) + ex2(acc[x][1] - m_new)) + (ex2(acc[x][2] - m_new) + ex2(acc[x][3] - m_new));
        lx = fmaf(lx, ex2(mx - m_new), s);
        mx = m_new;
      }
    }
    group_sync<C::NT>(g);                                        // buffer k&1 may be refilled
  }
  c_cur = k0 < k1 ? cols[k0] : 0;
  c_nxt = k0 + 1 < k1 ? cols[k0 + 1] : 0;
  if (k0 < k1) load_tile<Swizzle, BS, D, C::NT>(Bs + (k0 & 1) * C::TILE, Vb, c_cur * BS, t);
  cp_async_commit();
  float inv[R];
#pragma unroll
  for (int x = 0; x < R; ++x) {
    const float row_m = group_max<C::TX>(m[x]);
    const float z = group_sum<C::TX>(l[x] * ex2(m[x] - row_m));
    m[x] = row_m;
    inv[x] = z;
  }
  if (W > 1) {                                                   // join the groups' maxima and sums
    float2* stat = reinterpret_cast<float2*>(smem + W * two_pass_floats<BS, D, R>());       // [W][BS]
    if (tx == 0) {
#pragma unroll
      for (int x = 0; x < R; ++x) stat[g * BS + ty * R + x] = make_float2(m[x], inv[x]);
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < R; ++x) {
      float row_m = m[x], z = 0.f;
#pragma unroll
      for (int q = 0; q < W; ++q) row_m = fmaxf(row_m, stat[q * BS + ty * R + x].x);
#pragma unroll
      for (int q = 0; q < W; ++q) z = fmaf(stat[q * BS + ty * R + x].y, ex2(stat[q * BS + ty * R + x].x - row_m), z);
      m[x] = row_m;
      inv[x] = z;
    }
  }
#pragma unroll
  for (int x = 0; x < R; ++x) inv[x] = 1.0f / (inv[x] + (float)(L - nblk * BS) * ex2(-m[x]));

  // ---- pass 2: probabilities over the scores, O = P V
  Sums<BS, D, R> o;
  float4 sc[R];                                                  // scores of the tile about to be used
  auto fetch_scores = [&](int k) {
    const float* tile = mine + (long long)k * rt.step;
#pragma unroll
    for (int x = 0; x < R; ++x) sc[x] = load_vals(tile + x * rt.si, vec);
  };
  if (k0 < k1) fetch_scores(k0);
  for (int k = k0; k < k1; ++k) {
    if (k + 1 < k1)
      load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Vb, c_nxt * BS, t);
    cp_async_commit();
    float* tile = mine + (long long)k * rt.step;
#pragma unroll
    for (int half = 0; half < R / 4; ++half) {
      float pr[4][4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int i = half * 4 + x;
        const float v[4] = {sc[i].x, sc[i].y, sc[i].z, sc[i].w};
#pragma unroll
        for (int y = 0; y < 4; ++y) pr[x][y] = inv[i] == 0.f ? 0.f : ex2(v[y] - m[i]) * inv[i];
        store_vals(tile + i * rt.si, make_float4(pr[x][0], pr[x][1], pr[x][2], pr[x][3]), vec);
      }
      put_transposed<BS>(Ps, R / 4 * ty + half, tx, pr);
    }
    if (k + 1 < k1) fetch_scores(k + 1);                       // in flight during the product below
    c_cur = c_nxt;
    c_nxt = k + 2 < k1 ? cols[k + 2] : 0;
    cp_async_wait<1>();
    group_sync<C::NT>(g);                                        // V tile k has landed, Ps is complete
    tile_atb<BS, D, R>(Ps, Bs + (k & 1) * C::TILE, ty, tx, o);
    group_sync<C::NT>(g);                                        // Ps and buffer k&1 may be overwritten
  }
  cp_async_wait<0>();
  if (W > 1) {
    group_sync<C::NT>(g);
    join_sums<BS, D, R, W>(Qs, two_pass_floats<BS, D, R>(), g, t, o);
    if (g > 0) return;
  }
  store_out<BS, D, R>(O + (long long)bh * lo.bh_stride, lo, r * BS, ty, tx, o);
}

// ------------------------------------------------------------------------------ backward, row side
//   t = dP.P ; s = rowsum(t) ; dS = (t - P s) scale ; dQ = dS K     (models/block_attn.cu:90-130, :498-516)
template <int BS, int D, int R, int W>
__global__ void __launch_bounds__(cta_threads<BS, D, R, W>(), cta_resident<BS, D, R, W>(Cfg<BS, D, R>::RESIDENT)) fused_bwd_row_kernel(const float* __restrict__ dO, OperandLayout ldo,
                                                               const float* __restrict__ V, OperandLayout lv,
                                                               const float* __restrict__ K, OperandLayout lk,
                                                               const float* __restrict__ P, ValueLayout vp, float* dS,
                                                               ValueLayout vds, float* __restrict__ dQ,
                                                               OperandLayout ldq, Pattern p, int BH, float scale) {
  using C = Cfg<BS, D, R>;
  extern __shared__ __align__(16) float smem[];
  const int g = threadIdx.x / C::NT, t = threadIdx.x % C::NT;
  const int ty = t / C::TX, tx = t % C::TX;
  const int r = blockIdx.x, bh = W > 1 ? blockIdx.y : blockIdx.y * C::G + g;
  if (bh >= BH) return;
  float* As = smem + g * two_pass_floats<BS, D, R>();              // dO tile
  float* Bs = As + ONE<BS, D, R>;                                // two buffers: V tiles, then K tiles
  float* Ss = As;                                               // dS tile, pass 2

  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const int* cols = p.col_idx + rp;
  const int k0 = W > 1 ? nblk * g / W : 0, k1 = W > 1 ? nblk * (g + 1) / W : nblk;      // this group's blocks
  const Operand Vb(V, lv, bh), Kb(K, lk, bh);
  const RowTiles rp_t = RowTiles::of<BS>(vp, rp, nblk), rs_t = RowTiles::of<BS>(vds, rp, nblk);
  const float* Pb = P + (long long)bh * vp.bh_stride + rp_t.base + ty * R * rp_t.si + tx * 4;   // the thread's values of the first tile
  float* dSb = dS + (long long)bh * vds.bh_stride + rs_t.base + ty * R * rs_t.si + tx * 4;
  const bool vec_p = vec_ok(Pb), vec_s = vec_ok(dSb);

  int c_cur = k0 < k1 ? cols[k0] : 0, c_nxt = k0 + 1 < k1 ? cols[k0 + 1] : 0;
  load_tile<Swizzle, BS, D, C::NT>(As, Operand(dO, ldo, bh), r * BS, t);
  if (k0 < k1) load_tile<Swizzle, BS, D, C::NT>(Bs + (k0 & 1) * C::TILE, Vb, c_cur * BS, t);
  cp_async_commit();

  // ---- pass 1: dP into the dS tiles, row sums of dP.P
  float s[R];
#pragma unroll
  for (int x = 0; x < R; ++x) s[x] = 0.f;
  for (int k = k0; k < k1; ++k) {
    if (k + 1 < k1)
      load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Vb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < k1 ? cols[k + 2] : 0;
    float4 pv[R];                                                // requested before the wait: both latencies overlap
#pragma unroll
    for (int x = 0; x < R; ++x) pv[x] = load_vals(Pb + (long long)k * rp_t.step + x * rp_t.si, vec_p);
    cp_async_wait<1>();
    group_sync<C::NT>(g);
#pragma unroll
    for (int half = 0; half < R / 4; ++half) {
      float acc[4][4];
      tile_abt<BS, D>(As, Bs + (k & 1) * C::TILE, ty * R + half * 4, tx, acc);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int i = half * 4 + x;
        s[i] = fmaf(acc[x][0], pv[i].x, s[i]);
        s[i] = fmaf(acc[x][1], pv[i].y, s[i]);
        s[i] = fmaf(acc[x][2], pv[i].z, s[i]);
        s[i] = fmaf(acc[x][3], pv[i].w, s[i]);
        store_vals(dSb + (long long)k * rs_t.step + i * rs_t.si, make_float4(acc[x][0], acc[x][1], acc[x][2], acc[x][3]), vec_s);
      }
    }
    group_sync<C::NT>(g);
  }
#pragma unroll
  for (int x = 0; x < R; ++x) s[x] = group_sum<C::TX>(s[x]);
  if (W > 1) {
    float* stat = smem + W * two_pass_floats<BS, D, R>();        // [W][BS]
    if (tx == 0) {
#pragma unroll
      for (int x = 0; x < R; ++x) stat[g * BS + ty * R + x] = s[x];
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < R; ++x) {
      s[x] = 0.f;
#pragma unroll
      for (int q = 0; q < W; ++q) s[x] += stat[q * BS + ty * R + x];
    }
  }

  // ---- pass 2: dS over dP, dQ = dS K
  Sums<BS, D, R> o;
  c_cur = k0 < k1 ? cols[k0] : 0;
  c_nxt = k0 + 1 < k1 ? cols[k0 + 1] : 0;
  if (k0 < k1) load_tile<Swizzle, BS, D, C::NT>(Bs + (k0 & 1) * C::TILE, Kb, c_cur * BS, t);
  cp_async_commit();
  for (int k = k0; k < k1; ++k) {
    if (k + 1 < k1)
      load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Kb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < k1 ? cols[k + 2] : 0;
#pragma unroll
    for (int half = 0; half < R / 4; ++half) {
      float ds[4][4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int i = half * 4 + x;
        float* e = dSb + (long long)k * rs_t.step + i * rs_t.si;
        const float4 dp = load_vals(e, vec_s), pv = load_vals(Pb + (long long)k * rp_t.step + i * rp_t.si, vec_p);
        ds[x][0] = (dp.x * pv.x - pv.x * s[i]) * scale;
        ds[x][1] = (dp.y * pv.y - pv.y * s[i]) * scale;
        ds[x][2] = (dp.z * pv.z - pv.z * s[i]) * scale;
        ds[x][3] = (dp.w * pv.w - pv.w * s[i]) * scale;
        store_vals(e, make_float4(ds[x][0], ds[x][1], ds[x][2], ds[x][3]), vec_s);
      }
      put_transposed<BS>(Ss, R / 4 * ty + half, tx, ds);
    }
    cp_async_wait<1>();
    group_sync<C::NT>(g);
    tile_atb<BS, D, R>(Ss, Bs + (k & 1) * C::TILE, ty, tx, o);
    group_sync<C::NT>(g);
  }
  cp_async_wait<0>();
  if (W > 1) {
    group_sync<C::NT>(g);
    join_sums<BS, D, R, W>(As, two_pass_floats<BS, D, R>(), g, t, o);
    if (g > 0) return;
  }
  store_out<BS, D, R>(dQ + (long long)bh * ldq.bh_stride, ldq, r * BS, ty, tx, o);
}

// Row backward when O is at hand: rowsum(dP.P) = rowsum(dO.O) (delta), so dS of a tile needs nothing
// from the other tiles of its row and one pass suffices.  Two stages per block, V tile (for dP) and
// K tile (for dQ); the copy of one is in flight while the other is used.
template <int BS, int D, int R, int W>
__global__ void __launch_bounds__(cta_threads<BS, D, R, W>(), cta_resident<BS, D, R, W>(Cfg<BS, D, R>::RESIDENT)) fused_bwd_row_delta_kernel(const float* __restrict__ dO, OperandLayout ldo,
                                                                     const float* __restrict__ O, OperandLayout lo,
                                                                     const float* __restrict__ V, OperandLayout lv,
                                                                     const float* __restrict__ K, OperandLayout lk,
                                                                     const float* __restrict__ P, ValueLayout vp,
                                                                     float* __restrict__ dS, ValueLayout vds,
                                                                     float* __restrict__ dQ, OperandLayout ldq,
                                                                     Pattern p, int BH, float scale) {
  using C = Cfg<BS, D, R>;
  extern __shared__ __align__(16) float smem[];
  const int g = threadIdx.x / C::NT, t = threadIdx.x % C::NT;
  const int ty = t / C::TX, tx = t % C::TX;
  const int r = blockIdx.x, bh = W > 1 ? blockIdx.y : blockIdx.y * C::G + g;
  if (bh >= BH) return;
  float* As = smem + g * (3 * C::TILE + C::VALS);               // dO tile
  float* Vs = As + C::TILE;
  float* Ks = As + 2 * C::TILE;
  float* Ss = As + 3 * C::TILE;                                 // dS tile

  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const int* cols = p.col_idx + rp;
  const int k0 = W > 1 ? nblk * g / W : 0, k1 = W > 1 ? nblk * (g + 1) / W : nblk;      // this group's blocks
  const Operand Vb(V, lv, bh), Kb(K, lk, bh);
  const RowTiles rp_t = RowTiles::of<BS>(vp, rp, nblk), rs_t = RowTiles::of<BS>(vds, rp, nblk);
  const float* Pb = P + (long long)bh * vp.bh_stride + rp_t.base + ty * R * rp_t.si + tx * 4;   // the thread's values of the first tile
  float* dSb = dS + (long long)bh * vds.bh_stride + rs_t.base + ty * R * rs_t.si + tx * 4;
  const bool vec_p = vec_ok(Pb), vec_s = vec_ok(dSb);

  int c_cur = k0 < k1 ? cols[k0] : 0, c_nxt = k0 + 1 < k1 ? cols[k0 + 1] : 0;
  load_tile<Swizzle, BS, D, C::NT>(As, Operand(dO, ldo, bh), r * BS, t);
  if (k0 < k1) load_tile<Swizzle, BS, D, C::NT>(Vs, Vb, c_cur * BS, t);
  cp_async_commit();
  if (k0 < k1) load_tile<Swizzle, BS, D, C::NT>(Ks, Kb, c_cur * BS, t);
  cp_async_commit();

  float delta[R];
#pragma unroll
  for (int x = 0; x < R; ++x) delta[x] = 0.f;
  Sums<BS, D, R> o;
  float4 pv[R];                                                  // the tile's probabilities, requested one tile ahead
  auto fetch_p = [&](int k) {
#pragma unroll
    for (int x = 0; x < R; ++x) pv[x] = load_vals(Pb + (long long)k * rp_t.step + x * rp_t.si, vec_p);
  };
  if (k0 < k1) fetch_p(k0);

  for (int k = k0; k < k1; ++k) {
    cp_async_wait<1>();
    group_sync<C::NT>(g);                                        // V tile k (and dO) have landed
    if (k == k0) {
      const float* Ob = O + (long long)bh * lo.bh_stride + (long long)(r * BS + ty * R) * lo.sl;
#pragma unroll
      for (int x = 0; x < R; ++x) {
        float a = 0.f, d[C::TN];
        load_vec<BS, D, R>(As, ty * R + x, tx, d);
#pragma unroll
        for (int y = 0; y < C::TN; ++y) a = fmaf(d[y], Ob[(long long)x * lo.sl + (long long)out_col<BS, D, R>(tx, y) * lo.sd], a);
        delta[x] = group_sum<C::TX>(a);
      }
    }
#pragma unroll
    for (int half = 0; half < R / 4; ++half) {
      float acc[4][4];
      tile_abt<BS, D>(As, Vs, ty * R + half * 4, tx, acc);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int i = half * 4 + x;
        const float pr[4] = {pv[i].x, pv[i].y, pv[i].z, pv[i].w};
#pragma unroll
        for (int y = 0; y < 4; ++y) acc[x][y] = pr[y] * (acc[x][y] - delta[i]) * scale;
        store_vals(dSb + (long long)k * rs_t.step + i * rs_t.si, make_float4(acc[x][0], acc[x][1], acc[x][2], acc[x][3]), vec_s);
      }
      put_transposed<BS>(Ss, R / 4 * ty + half, tx, acc);
    }
    group_sync<C::NT>(g);                                        // Ss complete, V buffer free
    if (k + 1 < k1) {
      load_tile<Swizzle, BS, D, C::NT>(Vs, Vb, c_nxt * BS, t);
      fetch_p(k + 1);
    }
    cp_async_commit();
    cp_async_wait<1>();
    group_sync<C::NT>(g);                                        // K tile k has landed
    tile_atb<BS, D, R>(Ss, Ks, ty, tx, o);
    group_sync<C::NT>(g);                                        // Ss and the K buffer are free
    if (k + 1 < k1) load_tile<Swizzle, BS, D, C::NT>(Ks, Kb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < k1 ? cols[k + 2] : 0;
  }
  cp_async_wait<0>();
  if (W > 1) {
    group_sync<C::NT>(g);
    join_sums<BS, D, R, W>(As, 3 * C::TILE + C::VALS, g, t, o);
    if (g > 0) return;
  }
  store_out<BS, D, R>(dQ + (long long)bh * ldq.bh_stride, ldq, r * BS, ty, tx, o);
}

// ------------------------------------------------------------------------------ backward, column side
//   dK[c] = sum_r dS(r,c)^T Q[r],  dV[c] = sum_r P(r,c)^T dO[r]     (models/block_attn.cu:526-536)
// Two stages per entry of the column: (dS, Q) for dK and (P, dO) for dV; the copy of one stage is in
// flight while the other is used.
// A cluster of SPLIT_WAYS CTAs per column: there is room for them, and discovered masks have columns that every row selects; one CTA would
// walk such a column long after the others are done.  The CTAs of the cluster take a share of its entries each and the
// first adds the others' sums, in their order, through distributed shared memory.  Columns below SPLIT_MIN entries
// are left to the first CTA; the others end at once.  Eight CTAs per column were slower than four (16 matrices, L = 1024, blocks
// of 32 at 15 %: 57 against 24 us, 41 without a split).
constexpr int SPLIT_WAYS = 4, SPLIT_MIN = 3;
template <int BS, int D, int R>
__global__ void __launch_bounds__(Cfg<BS, D, R>::CTA, Cfg<BS, D, R>::RESIDENT) fused_bwd_col_kernel(const float* __restrict__ dS, ValueLayout vds,
                                                               const float* __restrict__ P, ValueLayout vp,
                                                               const float* __restrict__ Q, OperandLayout lq,
                                                               const float* __restrict__ dO, OperandLayout ldo,
                                                               float* __restrict__ dK, OperandLayout ldk,
                                                               float* __restrict__ dV, OperandLayout ldv, Pattern p,
                                                               int BH) {
  using C = Cfg<BS, D, R>;
  extern __shared__ __align__(16) float smem[];
  const int g = threadIdx.x / C::NT, t = threadIdx.x % C::NT;
  const int ty = t / C::TX, tx = t % C::TX;
  const int c = blockIdx.x / SPLIT_WAYS, part = blockIdx.x % SPLIT_WAYS;
  const int bh_raw = blockIdx.y * C::G + g;
  const bool active = bh_raw < BH;
  const int bh = active ? bh_raw : BH - 1;                      // the cluster barriers take every thread
  int e0 = p.col_ptr[c], e1 = p.col_ptr[c + 1];
  const bool shared = e1 - e0 >= SPLIT_MIN;
  if (!shared && (part > 0 || !active)) return;
  if (shared) {
    const int first = e0, n = e1 - e0;
    e0 = first + n * part / SPLIT_WAYS;
    e1 = active ? first + n * (part + 1) / SPLIT_WAYS : e0;
  }
  float* dSs = smem + g * (2 * C::TILE + 2 * C::VALS);
  float* Qs = dSs + C::VALS;
  float* Ps = Qs + C::TILE;
  float* Os = Ps + C::VALS;

  const float* dSb = dS + (long long)bh * vds.bh_stride;
  const float* Pb = P + (long long)bh * vp.bh_stride;
  const Operand Qb(Q, lq, bh), dOb(dO, ldo, bh);

  Sums<BS, D, R> ak, av;

  auto fetch_k = [&](int r, int blk) {                          // stage A: dS tile and Q rows of entry (r, blk)
    long long b1, s1, t1;
    tile_address(vds, p, r, c, blk, b1, s1, t1);
    load_tile<Swizzle, BS, BS, C::NT>(dSs, Operand(dSb + b1, (int)s1), 0, t);
    load_tile<Swizzle, BS, D, C::NT>(Qs, Qb, r * BS, t);
  };
  auto fetch_v = [&](int r, int blk) {                          // stage B: P tile and dO rows
    long long b2, s2, t2;
    tile_address(vp, p, r, c, blk, b2, s2, t2);
    load_tile<Swizzle, BS, BS, C::NT>(Ps, Operand(Pb + b2, (int)s2), 0, t);
    load_tile<Swizzle, BS, D, C::NT>(Os, dOb, r * BS, t);
  };
  int r_cur = e0 < e1 ? p.row_idx[e0] : 0, b_cur = e0 < e1 ? p.csc_pos[e0] : 0;
  if (e0 < e1) fetch_k(r_cur, b_cur);
  cp_async_commit();
  for (int e = e0; e < e1; ++e) {
    const int r_nxt = e + 1 < e1 ? p.row_idx[e + 1] : 0, b_nxt = e + 1 < e1 ? p.csc_pos[e + 1] : 0;
    fetch_v(r_cur, b_cur);                                       // stage B was released at the end of the last iteration
    cp_async_commit();
    cp_async_wait<1>();
    group_sync<C::NT>(g);                                        // stage A has landed
    tile_atb<BS, D, R>(dSs, Qs, ty, tx, ak);
    group_sync<C::NT>(g);                                        // stage A may be refilled
    if (e + 1 < e1) fetch_k(r_nxt, b_nxt);
    cp_async_commit();
    cp_async_wait<1>();
    group_sync<C::NT>(g);                                        // stage B has landed
    tile_atb<BS, D, R>(Ps, Os, ty, tx, av);
    group_sync<C::NT>(g);
    r_cur = r_nxt;
    b_cur = b_nxt;
  }
  cp_async_wait<0>();
  if (shared) {                                                  // the same for all CTAs of the cluster
    auto cluster = cooperative_groups::this_cluster();
    group_sync<C::NT>(g);                                        // the tiles are read: their place takes the sums
    pair_t* mine = reinterpret_cast<pair_t*>(dSs) + t;           // pair i of thread t at i * NT + t
    if (part > 0) {
#pragma unroll
      for (int x = 0; x < R / 2; ++x)
#pragma unroll
        for (int y = 0; y < C::TN; ++y) {
          mine[(x * C::TN + y) * C::NT] = ak.v[x][y];
          mine[(R / 2 * C::TN + x * C::TN + y) * C::NT] = av.v[x][y];
        }
    }
    cluster.sync();
    if (part == 0) {
      auto add = [](pair_t& sum, pair_t v) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum) : "l"(v)); };
      for (int q = 1; q < SPLIT_WAYS; ++q) {
        const pair_t* theirs = cluster.map_shared_rank(mine, q);
#pragma unroll
        for (int x = 0; x < R / 2; ++x)
#pragma unroll
          for (int y = 0; y < C::TN; ++y) {
            add(ak.v[x][y], theirs[(x * C::TN + y) * C::NT]);
            add(av.v[x][y], theirs[(R / 2 * C::TN + x * C::TN + y) * C::NT]);
          }
      }
    }
    cluster.sync();                                              // nobody leaves while its sums are read
    if (part > 0 || !active) return;
  }
  store_out<BS, D, R>(dK + (long long)bh * ldk.bh_stride, ldk, c * BS, ty, tx, ak);
  store_out<BS, D, R>(dV + (long long)bh * ldv.bh_stride, ldv, c * BS, ty, tx, av);
}

template <int BS, int D, int R, int W> constexpr size_t smem_two_pass() {
  return sizeof(float) * (cta_groups<BS, D, R, W>() * two_pass_floats<BS, D, R>() + (W > 1 ? 2 * W * BS : 0));
}
template <int BS, int D, int R, int W> constexpr size_t smem_row() {
  return sizeof(float) * cta_groups<BS, D, R, W>() * (3 * Cfg<BS, D, R>::TILE + Cfg<BS, D, R>::VALS);
}
template <int BS, int D, int R> constexpr size_t smem_col() { return sizeof(float) * Cfg<BS, D, R>::G * (2 * Cfg<BS, D, R>::TILE + 2 * Cfg<BS, D, R>::VALS); }

template <int BS, int D, int R, int W>
int set_attrs() {
  static std::atomic<bool> done[64];
  int dev = 0;
  SPION_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return SPION_OK;
  SPION_CUDA_TRY(cudaFuncSetAttribute(fused_fwd_kernel<BS, D, R, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_two_pass<BS, D, R, W>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(fused_bwd_row_kernel<BS, D, R, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_two_pass<BS, D, R, W>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(fused_bwd_row_delta_kernel<BS, D, R, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_row<BS, D, R, W>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(fused_bwd_col_kernel<BS, D, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_col<BS, D, R>()));
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return SPION_OK;
}

template <int BS, int D, int R, int W>
int fwd_launch(const float* Q, OperandLayout lq, const float* K, OperandLayout lk, const float* V, OperandLayout lv,
               const float* keypad, float floor_v, float* P, ValueLayout vl, float* O, OperandLayout lo, Pattern p,
               int BH, int L, float scale, cudaStream_t st) {
  int rc = set_attrs<BS, D, R, W>();
  if (rc) return rc;
  const dim3 grid(p.nb, W > 1 ? BH : (BH + Cfg<BS, D, R>::G - 1) / Cfg<BS, D, R>::G);
  fused_fwd_kernel<BS, D, R, W><<<grid, cta_threads<BS, D, R, W>(), smem_two_pass<BS, D, R, W>(), st>>>(Q, lq, K, lk, V, lv, keypad, floor_v, P, vl, O, lo, p, BH,
                                                               L, scale);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

template <int BS, int D, int R, int W>
int bwd_launch(const float* Q, OperandLayout lq, const float* K, OperandLayout lk, const float* V, OperandLayout lv,
               const float* P, ValueLayout vp, const float* O, OperandLayout lo, const float* dO, OperandLayout ldo,
               float* dS, ValueLayout vds, float* dQ, OperandLayout ldq, float* dK, OperandLayout ldk, float* dV,
               OperandLayout ldv, Pattern p, int BH, float scale, cudaStream_t st, spion_ctx* prof) {
  int rc = set_attrs<BS, D, R, W>();
  if (rc) return rc;
  const dim3 grid(p.nb, W > 1 ? BH : (BH + Cfg<BS, D, R>::G - 1) / Cfg<BS, D, R>::G);
  if (O)
    fused_bwd_row_delta_kernel<BS, D, R, W><<<grid, cta_threads<BS, D, R, W>(), smem_row<BS, D, R, W>(), st>>>(dO, ldo, O, lo, V, lv, K, lk, P, vp, dS, vds,
                                                                           dQ, ldq, p, BH, scale);
  else
    fused_bwd_row_kernel<BS, D, R, W><<<grid, cta_threads<BS, D, R, W>(), smem_two_pass<BS, D, R, W>(), st>>>(dO, ldo, V, lv, K, lk, P, vp, dS, vds, dQ, ldq, p,
                                                                     BH, scale);
  SPION_LAUNCH_CHECK();
  if (prof) prof_mark(prof, SPION_STAGE_BWD_ROW);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.nb * SPLIT_WAYS, (BH + Cfg<BS, D, R>::G - 1) / Cfg<BS, D, R>::G);
  cfg.blockDim = dim3(Cfg<BS, D, R>::CTA);
  cfg.dynamicSmemBytes = smem_col<BS, D, R>();
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = SPLIT_WAYS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  SPION_CUDA_TRY(cudaLaunchKernelEx(&cfg, fused_bwd_col_kernel<BS, D, R>, (const float*)dS, vds, P, vp, Q, lq, dO, ldo, dK, ldk, dV, ldv, p, BH));
  SPION_LAUNCH_CHECK();
  if (prof) prof_mark(prof, SPION_STAGE_SPMM_DKDV);
  return SPION_OK;
}

}  // namespace

bool simt_fused_supports(int bs, int d, int BH, int value_mode) {
  return (bs == 32 || bs == 64) && (d == 32 || d == 64) && BH >= 1 && (BH + 3) / 4 <= 65535 &&
         (value_mode == VAL_ELEMCSR || value_mode == VAL_BLOCKTILE);
}

// Which calls the kernels of mma_fused.cu serve: those with work for most schedulers.  Their warps do twice (block 32) or half (64) of what
// the threads of a row do here, and nobody shares a row there, so the uneven rows of small calls are better shared by groups of threads (up to four
// rows of blocks of 32 per SM, see row_groups).  us of forward, rows and columns there and here, in a graph (a band of two blocks and random ones):
//   blocks of 32, d 32: rows of 5 blocks 256 51, 46; 304 56, 50; 416 57, 57; 480 60, 71; 512 (of 4.8) 53, 64; 1024 90, 120.  Rows of 8 384 85, 75; 448 87, 78;
//     480 86, 91.  Rows of 12, 24, 45: two or three matrices 456 rows 0.85, 0.87, 0.86 times the speed there, 500 0.86, 0.88, 0.83, 540 0.89, 0.90,
//     0.84; four or eight matrices 448 0.86 - 0.98, 512 1.01 - 1.09; 768 and more 1.09 - 1.20.
//   d 64, whose threads here have twice the work: rows of 5 256 77, 78; 304 93, 83; 320 89, 88; 512 102, 120.  Rows of 12, 24, 45: 300 0.86, 0.79,
//     0.89 times the speed there, 320 0.87 - 0.92, 380 0.91 - 0.95, 384 0.84 - 0.99 (with a full column 0.89 - 1.24), 456 and more 1.01 - 1.20
//   blocks of 64, d 32: 144 rows of 5 87, 85; 160 of 5 100, 114;  d 64: 160 of 5 170, 165; 176 of 5 191, 162; 192 of 5 166, 171; 224 of 5 183, 206
//     (with a full column: 160 of 7 1.05 times as long there, 192 of 7 0.88; all of equal length: 176 rows of 6 0.81)
// Few blocks in all stay here although rows of two are faster there (512 rows, d 32: 27, 38): up to that size a pass is host time.
static bool use_mma(const Pattern& p, int d, int BH, int nnzb) {
  const long long sms = sm_count(), rows = (long long)p.nb * BH, blocks = (long long)nnzb * BH;
  if (p.bs == 64) return 4 * rows >= (d == 64 ? 5 : 4) * sms && (blocks > 5 * sms || rows > 2 * sms);
  return rows > 8 * sms || (blocks > 10 * sms && (d == 64 ? 2 * rows > 5 * sms : rows > 4 * sms || (BH >= 4 && 5 * rows > 16 * sms)));
}

// Groups of threads that share the blocks of a row (forward and row kernels; columns are shared by a cluster).  They pay
// where the rows have blocks to share and some are longer than others, and lose in a second wave of CTAs with equal rows.  us of the forward
// and of the row kernel with one group, two (and four); masks with a band of two blocks and random ones unless stated:
//   blocks of 32: four up to one CTA per SM (d 32, 128 rows of 5 blocks, the longest 8: 16.6, 10.5, 9.1 and 15.6, 9.9, 8.5), two up to four
//     (d 32, 384 rows of 8 35.6, 25.2, 26.7 and 32.8, 23.9, 24.9, of 5 23.8, 18.9, 21.1; 592 of 2 10.8, 10.4, 15.3 and 12.0, 10.2, 13.9, but 512 of 2
//     10.2, 11.3, 15.1; d 64, 288 rows of two blocks 12.0, 8.3, 12.5 and 12.3, 9.6, 13.5).  d 64: half the registers make the row kernel slower
//     from 512 rows on (of two blocks 15.7, 20.3; 384 rows of 8 56.5, 45.9), so its line is three CTAs per SM.
//   blocks of 64 (512 threads for two groups): d 64, 128 rows of 10 blocks 74, 69 and 73, 63; 192 rows of 3 blocks 48, 44 and 47, 41, of 4
//     62, 53 and 61, 49 (all of 4: 39.8, 42.8 and 38.9, 40.1); 288 rows of 3 48, 52 and 47, 48, of 8 131, 133 and 126, 122; rows of two blocks:
//     128 13.3, 13.4 and 13.2, 12.4, 192 21.5, 24.6 and 21.3, 22.9.  So three CTAs for two SMs, and one per SM if the rows are short.
//   rows of one block: the joins are pure cost (blocks of 32, d 64, 512 rows: 8.0, 8.9 and 8.4, 10.1; blocks of 64, 128 rows 8.1, 8.9).
// A pass of up to about 500 short rows is host time whatever the groups (90 us forward + backward).
static int row_groups(int bs, int d, long long rows, long long nnzb, int nb, bool backward) {
  const long long sms = sm_count();
  if (2 * nnzb < 3LL * nb) return 1;                  // most rows have one block
  if (bs == 64) return 2 * rows <= (nnzb < 3LL * nb ? 2 : 3) * sms ? 2 : 1;
  return rows <= sms ? 4 : rows <= (backward && d == 64 ? 3 : 4) * sms ? 2 : 1;
}
#define SPION_FUSED_DISPATCH(FN, BACKWARD, ...)                                                      \
  do {                                                                                               \
    const int ways = row_groups(p.bs, d, (long long)p.nb * BH, nnzb, p.nb, BACKWARD);                \
    if (p.bs == 32 && d == 32)                                                                       \
      return ways == 4 ? FN<32, 32, 4, 4>(__VA_ARGS__) : ways == 2 ? FN<32, 32, 4, 2>(__VA_ARGS__) : FN<32, 32, 4, 1>(__VA_ARGS__); \
    if (p.bs == 32 && d == 64)                                                                       \
      return ways == 4 ? FN<32, 64, 4, 4>(__VA_ARGS__) : ways == 2 ? FN<32, 64, 4, 2>(__VA_ARGS__) : FN<32, 64, 4, 1>(__VA_ARGS__); \
    if (p.bs == 64 && d == 32) return ways == 2 ? FN<64, 32, 4, 2>(__VA_ARGS__) : FN<64, 32, 4, 1>(__VA_ARGS__); \
    if (p.bs == 64 && d == 64) return ways == 2 ? FN<64, 64, 4, 2>(__VA_ARGS__) : FN<64, 64, 4, 1>(__VA_ARGS__); \
    return SPION_ERR_UNSUPPORTED;                                                                    \
  } while (0)

// A launch has groups of matrices along gridDim.y, and a group is one matrix for blocks of 64 (simt_full.cu, mma_fused.cu), two or four for
// blocks of 32: calls with more matrices run in equal slices.
constexpr int MOST_MATRICES = 65535;
static int slice(int BH) {
  const int n = (BH + MOST_MATRICES - 1) / MOST_MATRICES;
  return (BH + n - 1) / n;
}

// The full mask has kernels of its own (simt_full.cu).
int simt_fused_forward(const float* Q, OperandLayout lq, const float* K, OperandLayout lk, const float* V,
                       OperandLayout lv, const float* keypad, float floor_v, float* P, ValueLayout vl, float* O,
                       OperandLayout lo, Pattern p, int BH, int L, int d, float scale, cudaStream_t st, int nnzb) {
  if (!simt_fused_supports(p.bs, d, BH, vl.mode)) return SPION_ERR_UNSUPPORTED;
  if (BH > MOST_MATRICES) {
    const int per = slice(BH);
    for (long long b = 0; b < BH; b += per) {
      const int rc = simt_fused_forward(Q + b * lq.bh_stride, lq, K + b * lk.bh_stride, lk, V + b * lv.bh_stride, lv, keypad ? keypad + b * L : nullptr,
                                        floor_v, P + b * vl.bh_stride, vl, O + b * lo.bh_stride, lo, p, min(per, BH - (int)b), L, d, scale, st, nnzb);
      if (rc) return rc;
    }
    return SPION_OK;
  }
  if (nnzb == p.nb * p.nb) return simt_full_forward(Q, lq, K, lk, V, lv, keypad, floor_v, P, vl, O, lo, p, BH, L, d, scale, st);
  if (use_mma(p, d, BH, nnzb)) return mma_fused_forward(Q, lq, K, lk, V, lv, keypad, floor_v, P, vl, O, lo, p, BH, L, d, scale, st);
  SPION_FUSED_DISPATCH(fwd_launch, false, Q, lq, K, lk, V, lv, keypad, floor_v, P, vl, O, lo, p, BH, L, scale, st);
}

int simt_fused_backward(const float* Q, OperandLayout lq, const float* K, OperandLayout lk, const float* V,
                        OperandLayout lv, const float* P, ValueLayout vp, const float* O, OperandLayout lo,
                        const float* dO, OperandLayout ldo, float* dS, ValueLayout vds, float* dQ, OperandLayout ldq,
                        float* dK, OperandLayout ldk, float* dV, OperandLayout ldv, Pattern p, int BH, int d,
                        float scale, cudaStream_t st, spion_ctx* prof, int nnzb) {
  if (!simt_fused_supports(p.bs, d, BH, vp.mode) || vds.mode != vp.mode) return SPION_ERR_UNSUPPORTED;
  if (BH > MOST_MATRICES) {
    const int per = slice(BH);
    for (long long b = 0; b < BH; b += per) {
      const int rc = simt_fused_backward(Q + b * lq.bh_stride, lq, K + b * lk.bh_stride, lk, V + b * lv.bh_stride, lv, P + b * vp.bh_stride, vp,
                                         O ? O + b * lo.bh_stride : nullptr, lo, dO + b * ldo.bh_stride, ldo, dS + b * vds.bh_stride, vds,
                                         dQ + b * ldq.bh_stride, ldq, dK + b * ldk.bh_stride, ldk, dV + b * ldv.bh_stride, ldv, p,
                                         min(per, BH - (int)b), d, scale, st, prof, nnzb);
      if (rc) return rc;
    }
    return SPION_OK;
  }
  if (nnzb == p.nb * p.nb && O)
    return simt_full_backward(Q, lq, K, lk, V, lv, P, vp, O, lo, dO, ldo, dS, vds, dQ, ldq, dK, ldk, dV, ldv, p, BH, d, scale, st, prof);
  if (use_mma(p, d, BH, nnzb)) return mma_fused_backward(Q, lq, K, lk, V, lv, P, vp, O, lo, dO, ldo, dS, vds, dQ, ldq, dK, ldk, dV, ldv, p, BH, d, scale, st, prof, nnzb,
                                                      prof ? prof->longest_col : -1);
  SPION_FUSED_DISPATCH(bwd_launch, true, Q, lq, K, lk, V, lv, P, vp, O, lo, dO, ldo, dS, vds, dQ, ldq, dK, ldk, dV, ldv, p, BH,
                       scale, st, prof);
}
