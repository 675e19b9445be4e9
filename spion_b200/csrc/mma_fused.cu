// fp32 block-sparse attention of calls that fill the chip: the kernels of simt_fused.cu with their products on the tensor cores.
//
//   mma_fwd_kernel        per block row:     S = Q K^T -> sparse row softmax -> P (written once) -> O = P V
//   mma_bwd_row_kernel    per block row:     dP = dO V^T -> dS = P (dP - delta) scale -> dQ = dS K
//   mma_bwd_row2_kernel   the same when the caller has no O: dP is left in the dS tiles until rowsum(dP.P) is known
//   mma_bwd_col_kernel    per block column:  dK = dS^T Q, dV = P^T dO
//
// Precision.  Every fp32 operand is split into three bf16 parts (8 + 8 + 8 significant bits: exact from 2^-110 up) and the six partial
// products of weight 2^0, 2^-8 and 2^-16 are accumulated in fp32; the dropped ones are below 2^-25 of the product.  The tensor cores
// truncate a sum at every step, so each 16 terms of a contraction get accumulators of their own, the small products first, and are added
// in fp32: one truncated step at full weight per 16 terms where a chain of FMAs rounds 16 times.  The parts of an infinity are NaN where
// an fp32 product is an infinity or a number, and the last part of a value below 2^-110 ends at the smallest bf16 number: a warp that meets a
// result that is not finite, or smaller than 2^-100 and not zero, forms all of its rows again in plain fp32.
//
// mma.sync and not tcgen05: a tile of a 32-wide mask has 32 rows, P and dS stay in the registers that the next product takes them from,
// and the parts of an operand are made where it is used.  tcgen05 operands would go through shared memory three times as large.
// Bound by the legacy tensor path and the FMA pipes together: one m16n8k16 takes two cycles of an SM (six of them carry 1.3 times the
// multiply-adds of the FMA pipes in that time), and fp32 additions and multiplications of other warps wait for it and it for them (measured:
// their times add up; integer work overlaps by half).  So what is left out around the products counts: no check per tile, no select per value.
// Without products the kernels take 60 % of their time, products alone 45 %.
// us of forward, rows, columns, the FMA kernels before (8 x 4 micro-tiles) and now: 512 matrices, L = 1024, d 32, 155 blocks of 32 362, 314, 262
// -> 261, 245, 228; 128 matrices, L = 2048, 104 blocks of 64, d 32 263, 240, 234 -> 199, 184, 162, d 64 409, 384, 344 -> 335, 361, 308;
// 15 matrices, L = 3008, d 64, 8 % and a full column 140, 132, 158 -> 109, 119, 86 (132 without the overlap, see SHARED).  Relative error against fp64 of O, dQ, dK, dV in the first: 2.9,
// 3.0, 3.0, 2.8e-7 before, 1.6, 2.0, 2.0, 1.5e-7 now.
//
// A warp does MT x 16 rows of a tile, 32 columns at a time.  Fragment layouts leave the order of the contraction and of the columns open as
// long as both sides agree; they are chosen so that every read of shared memory and every access to a value tile is a 16-byte piece:
//   kappa(j, n) = 16 (j / 2) + 4 (n / 2) + 2 (j % 2) + n % 2    key of slot n of n-tile j: a thread's values are two pieces of four keys
//   d = 4 g + t                                                 column of slot g of n-tile t in the bs x d products
#include <cooperative_groups.h>

#include <atomic>

#include "fp32_tiles.cuh"

using namespace fp32;

namespace {

// MT: 16-row tiles per warp, two at most at head_dim 32 and one at 64: the sums of a product take MT * d / 2 registers.
template <int BS, int D, int MT>
struct Cfg {
  static constexpr int WR = 16 * MT;             // rows per warp
  static constexpr int NT = 32 * BS / WR;        // threads per (b,h) problem
  static constexpr int CTA = 128;
  static constexpr int G = CTA / NT;             // problems per CTA
  static constexpr int KS = D / 16;              // steps of a contraction over the head dimension
  static constexpr int NH = D / 32;              // groups of four n-tiles in a bs x d product
  static constexpr int TILE = BS * D, VALS = BS * BS;
  static constexpr int FRAGS = KS * MT * 3 * 32 * 4;      // floats: parts of the warp's rows of a fixed operand, ready as A fragments
  static constexpr int RESIDENT = 3;
};

// float offset of 16-byte piece `piece` of row `row`: the eight lanes of a read phase (two rows and four pieces, or four rows of every
// fourth and two pieces) meet eight different groups of banks
struct Swizzle {
  template <int COLS>
  static __device__ __forceinline__ int at(int row, int piece) {
    return row * COLS + ((piece ^ ((((row >> 2) & 3) << 1) ^ ((row & 1) << 2))) << 2);
  }
};

__device__ __forceinline__ int kappa(int j, int n) { return 16 * (j >> 1) + 4 * (n >> 1) + 2 * (j & 1) + (n & 1); }

__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
// Two values -> their leading, middle and last eight bits, as pairs of bf16.  (Masks in place of the roundings make the dropped products
// four times as large: dQ at d 64 3.9e-7 from fp64 instead of 2.3e-7, FMA kernels 3.5e-7.  Two tf32 parts and three products: 3.1e-7, 3 % faster.)
__device__ __forceinline__ void split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x, y);
  x -= __uint_as_float(hi << 16);
  y -= __uint_as_float(hi & 0xffff0000u);
  mid = pack_bf16(x, y);
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  lo = pack_bf16(x, y);
}

struct FragA { uint32_t p[3][4]; };              // parts of a 16 x 16 tile
struct FragB { uint32_t p[3][2]; };              // parts of a 16 x 8 tile
// q0, q1: four consecutive terms of rows g and g + 8
__device__ __forceinline__ FragA frag_a(float4 q0, float4 q1) {
  FragA f;
  split(q0.x, q0.y, f.p[0][0], f.p[1][0], f.p[2][0]);
  split(q1.x, q1.y, f.p[0][1], f.p[1][1], f.p[2][1]);
  split(q0.z, q0.w, f.p[0][2], f.p[1][2], f.p[2][2]);
  split(q1.z, q1.w, f.p[0][3], f.p[1][3], f.p[2][3]);
  return f;
}
__device__ __forceinline__ FragB frag_b(float a, float b, float c, float d) {
  FragB f;
  split(a, b, f.p[0][0], f.p[1][0], f.p[2][0]);
  split(c, d, f.p[0][1], f.p[1][1], f.p[2][1]);
  return f;
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_zero(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
// sum[m][n] += A[m] B[n] over 16 terms
template <int MT>
__device__ __forceinline__ void products(float (&sum)[MT][4][4], const FragA (&a)[MT], const FragB (&b)[4]) {
  constexpr int PA[6] = {0, 1, 2, 0, 1, 0}, PB[6] = {2, 1, 0, 1, 0, 0};       // smallest first
  float f[MT][4][4];
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (i == 0) mma_zero(f[m][n], a[m].p[PA[i]], b[n].p[PB[i]]);
        else mma(f[m][n], a[m].p[PA[i]], b[n].p[PB[i]]);
      }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) sum[m][n][x] += f[m][n][x];
}
template <int MT>
__device__ __forceinline__ void clear(float (&v)[MT][4][4]) {
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) v[m][n][x] = 0.f;
}
// Whether sums are what plain fp32 gives: finite (see split), and zero or at least 2^-100, a bound above which terms that have lost bits count for
// nothing: with n terms of factors around f an error of sqrt(n) f 2^-134 in all.
template <int MT>
__device__ __forceinline__ bool as_fp32(const float (&v)[MT][4][4]) {
  float probe = 0.f;
  uint32_t least = 0xffffffffu;                  // twice the bits less one: zeros are the largest
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        probe = fmaf(0.f, v[m][n][x], probe);
        least = min(least, 2u * __float_as_uint(v[m][n][x]) - 1u);
      }
  return probe == 0.f && least >= 2u * __float_as_uint(0x1p-100f) - 1u;
}

__device__ __forceinline__ float4 piece(const float* p) { return *reinterpret_cast<const float4*>(p); }

// The warp's rows of a [bs x d] tile -> A fragments in its part of shared memory.
template <int BS, int D, int MT>
__device__ __forceinline__ void make_frags(float* frags, const float* tile, int row0, int lane) {
  using C = Cfg<BS, D, MT>;
  const int g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int s = 0; s < C::KS; ++s)
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int row = row0 + 16 * m + g;
      const FragA f = frag_a(piece(tile + Swizzle::at<D>(row, 4 * s + c)), piece(tile + Swizzle::at<D>(row + 8, 4 * s + c)));
#pragma unroll
      for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(frags + (((s * MT + m) * 3 + p) * 32 + lane) * 4) = make_uint4(f.p[p][0], f.p[p][1], f.p[p][2], f.p[p][3]);
    }
}

// out = A B^T: the warp's rows (as fragments) by rows key0 .. key0 + 31 of a [bs x d] tile.  out[m][j][..]: keys kappa(j, 2 c + i), rows g, g + 8.
template <int BS, int D, int MT>
__device__ __forceinline__ void tile_abt(const float* frags, const float* tile, int key0, int lane, float (&out)[MT][4][4]) {
  using C = Cfg<BS, D, MT>;
  const int g = lane >> 2, c = lane & 3;
  clear(out);
#pragma unroll
  for (int s = 0; s < C::KS; ++s) {
    FragB b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 q = piece(tile + Swizzle::at<D>(key0 + kappa(j, g), 4 * s + c));
      b[j] = frag_b(q.x, q.y, q.z, q.w);
    }
    FragA a[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const uint4 v = *reinterpret_cast<const uint4*>(frags + (((s * MT + m) * 3 + p) * 32 + lane) * 4);
        a[m].p[p][0] = v.x; a[m].p[p][1] = v.y; a[m].p[p][2] = v.z; a[m].p[p][3] = v.w;
      }
    products(out, a, b);
  }
}

// sum += A B over 16 rows of a [bs x d] tile, row0 + 4 c .. + 3 of them this thread's
template <int D, int MT>
__device__ __forceinline__ void tile_ab(const FragA (&a)[MT], const float* tile, int row0, int lane, float (&sum)[D / 32][MT][4][4]) {
  const int g = lane >> 2, row = row0 + 4 * (lane & 3);
#pragma unroll
  for (int h = 0; h < D / 32; ++h) {
    float4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = piece(tile + Swizzle::at<D>(row + i, 8 * h + g));
    const FragB b[4] = {frag_b(q[0].x, q[1].x, q[2].x, q[3].x), frag_b(q[0].y, q[1].y, q[2].y, q[3].y),
                        frag_b(q[0].z, q[1].z, q[2].z, q[3].z), frag_b(q[0].w, q[1].w, q[2].w, q[3].w)};
    products(sum[h], a, b);
  }
}

// Row `row` of slot (m, half) of a bs x d product: columns 32 h + 8 c + 4 i + t.
template <int D, int MT>
__device__ __forceinline__ void store_row(float* out, long long sd, bool vec, const float (&sum)[D / 32][MT][4][4], int m, int half, int c) {
#pragma unroll
  for (int h = 0; h < D / 32; ++h)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float* o = out + (32 * h + 8 * c + 4 * i) * sd;
      const float4 v = make_float4(sum[h][m][0][2 * half + i], sum[h][m][1][2 * half + i], sum[h][m][2][2 * half + i], sum[h][m][3][2 * half + i]);
      if (vec) *reinterpret_cast<float4*>(o) = v;
      else o[0] = v.x, o[sd] = v.y, o[2 * sd] = v.z, o[3 * sd] = v.w;
    }
}
template <int D, int MT>
__device__ __forceinline__ bool all_as_fp32(const float (&sum)[D / 32][MT][4][4]) {
  bool ok = true;
#pragma unroll
  for (int h = 0; h < D / 32; ++h) ok = ok && as_fp32(sum[h]);
  return ok;
}

// The thread's values of 32 columns: piece jj of row slot (m, half).
__device__ __forceinline__ float4 quad(const float (&v)[4][4], int jj, int half) {
  return make_float4(v[2 * jj][2 * half], v[2 * jj][2 * half + 1], v[2 * jj + 1][2 * half], v[2 * jj + 1][2 * half + 1]);
}

__device__ __forceinline__ float quad_max(float v) {             // over the four lanes that share a row
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ------------------------------------------------------------------------------ plain fp32, by one warp, in the order of the terms
// Bound by the latency of its loads.  us of forward, rows, columns, 512 matrices, L = 1024, d 32, 155 blocks of 32: no such row 269, 252, 238; one infinity
// in V 359, 379, 239; dO of 1e-35, all rows again, 269, 2629, 1657.  (Term by term with a test after each, that infinity took 700 us more.)
__device__ __forceinline__ float4 load4(const Operand& o, int i, int n) {
  const float* p = o.base + i * o.s_row + n * o.s_col;
  return o.pieces ? piece(p) : make_float4(p[0], p[o.s_col], p[2 * o.s_col], p[3 * o.s_col]);
}
// WR rows of A by the rows of B's blocks -> value tiles.  Lanes are keys, whose rows of B stay in registers.
template <int BS, int D, int WR>
__device__ __forceinline__ void plain_abt(const Operand& A, int row0, const Operand& B, const int* cols, int nblk, float* out, int si, int step, int lane) {
  for (int k = 0; k < nblk; ++k)
    for (int j = lane; j < BS; j += 32) {
      float4 b[D / 4];
#pragma unroll
      for (int n = 0; n < D / 4; ++n) b[n] = load4(B, cols[k] * BS + j, 4 * n);
      for (int x = 0; x < WR; ++x) {
        float s = 0.f;
#pragma unroll
        for (int n = 0; n < D / 4; ++n) {
          const float4 q = load4(A, row0 + x, 4 * n);
          s = fmaf(q.w, b[n].w, fmaf(q.z, b[n].z, fmaf(q.y, b[n].y, fmaf(q.x, b[n].x, s))));
        }
        out[x * si + (long long)k * step + j] = s;
      }
    }
}
// WR rows of value tiles by B.  Lanes are columns of B.
template <int BS, int D, int WR>
__device__ __forceinline__ void plain_ab(const float* vals, int si, int step, const Operand& B, const int* cols, int nblk, float* out, long long sl, long long sd,
                                         int lane) {
  const bool vec = vec_ok(vals);
  for (int n = lane; n < D; n += 32) {
    float o[WR] = {};
    for (int k = 0; k < nblk; ++k)
      for (int j = 0; j < BS; j += 4) {
        float b[4];
#pragma unroll
        for (int y = 0; y < 4; ++y) b[y] = B.base[(cols[k] * BS + j + y) * B.s_row + n * B.s_col];
#pragma unroll
        for (int x = 0; x < WR; ++x) {
          const float4 v = load_vals(vals + x * si + (long long)k * step + j, vec);
          o[x] = fmaf(v.w, b[3], fmaf(v.z, b[2], fmaf(v.y, b[1], fmaf(v.x, b[0], o[x]))));
        }
      }
#pragma unroll
    for (int x = 0; x < WR; ++x) out[x * sl + n * sd] = o[x];
  }
}

// ------------------------------------------------------------------------------ forward
struct FwdArgs {
  const float *Q, *K, *V, *keypad;
  OperandLayout lq, lk, lv, lo;
  float floor_v, scale;
  float *P, *O;
  ValueLayout vl;
  Pattern p;
  int BH, L;
};

// Rows row0 .. row0 + WR - 1 of block row r
template <int BS, int D, int MT>
__device__ __noinline__ void redo_fwd(const FwdArgs& a, int bh, int r, int row0, int lane) {
  constexpr int WR = Cfg<BS, D, MT>::WR;
  const Operand Qb(a.Q, a.lq, bh), Kb(a.K, a.lk, bh), Vb(a.V, a.lv, bh);
  const int rp = a.p.row_ptr[r], nblk = a.p.row_ptr[r + 1] - rp;
  const int* cols = a.p.col_idx + rp;
  const RowTiles rt = RowTiles::of<BS>(a.vl, rp, nblk);
  const float* kp = a.keypad ? a.keypad + (long long)bh * a.L : nullptr;
  float* P0 = a.P + (long long)bh * a.vl.bh_stride + rt.base + row0 * rt.si;
  plain_abt<BS, D, WR>(Qb, r * BS + row0, Kb, cols, nblk, P0, rt.si, rt.step, lane);
  for (int x = 0; x < WR; ++x) {                   // a lane reads and writes what it has written
    float* Pr = P0 + x * rt.si;
    float m = a.floor_v * LOG2_E, l = 0.f;
    for (int k = 0; k < nblk; ++k)
      for (int j = lane; j < BS; j += 32) {
        float* e = Pr + (long long)k * rt.step + j;
        const float v = fmaf(*e, a.scale * LOG2_E, kp ? -kp[cols[k] * BS + j] * LOG2_E : 0.f), m_new = fmaxf(m, v);
        *e = v;
        l = fmaf(l, ex2(m - m_new), ex2(v - m_new));
        m = m_new;
      }
    const float row_m = warp_max(m), z = warp_sum(l * ex2(m - row_m));
    const float inv = 1.0f / (z + (float)(a.L - nblk * BS) * ex2(-row_m));
    for (int k = 0; k < nblk; ++k)
      for (int j = lane; j < BS; j += 32) {
        float* e = Pr + (long long)k * rt.step + j;
        *e = inv == 0.f ? 0.f : ex2(*e - row_m) * inv;
      }
  }
  __syncwarp();
  plain_ab<BS, D, WR>(P0, rt.si, rt.step, Vb, cols, nblk, a.O + (long long)bh * a.lo.bh_stride + (r * BS + row0) * a.lo.sl, a.lo.sl, a.lo.sd, lane);
}

//   v = S*scale - keypad[col];  m = max(floor, max v);  Z = sum exp(v-m) + (L-n_i) exp(-m);  P = exp(v-m)/Z
// Two passes over the blocks of a row, as in simt_fused.cu: the scaled scores wait in the P tiles (normally still in L2) while the row
// maximum and the denominator are accumulated on line.  K (pass 1) and V (pass 2) tiles are double-buffered.
template <int BS, int D, int MT>
__global__ void __launch_bounds__(128, (Cfg<BS, D, MT>::RESIDENT)) mma_fwd_kernel(const __grid_constant__ FwdArgs a) {
  using C = Cfg<BS, D, MT>;
  extern __shared__ __align__(16) float smem[];
  const int g0 = threadIdx.x / C::NT, t = threadIdx.x % C::NT, lane = t & 31;
  const int r = blockIdx.x, bh = blockIdx.y * C::G + g0;
  if (bh >= a.BH) return;
  float* Bs = smem + g0 * (C::NT / 32 * C::FRAGS + 2 * C::TILE);        // two buffers: K tiles, then V tiles
  float* frags = Bs + 2 * C::TILE + (t >> 5) * C::FRAGS;
  const int row0 = (t >> 5) * C::WR, g = lane >> 2, c = lane & 3;

  const int rp = a.p.row_ptr[r], nblk = a.p.row_ptr[r + 1] - rp;
  const int* cols = a.p.col_idx + rp;
  const Operand Kb(a.K, a.lk, bh), Vb(a.V, a.lv, bh);
  float* Pb = a.P + (long long)bh * a.vl.bh_stride;
  const float* kp = a.keypad ? a.keypad + (long long)bh * a.L + 4 * c : nullptr;
  const bool vec = vec_ok(Pb);
  const RowTiles rt = RowTiles::of<BS>(a.vl, rp, nblk);
  float* mine = Pb + rt.base + (row0 + g) * rt.si + 4 * c;              // row slot (m, h): + (16 m + 8 h) si; piece jj: + 16 jj
  const float scale2 = a.scale * LOG2_E;                                // scores in base-2 units

  int c_cur = nblk > 0 ? cols[0] : 0, c_nxt = nblk > 1 ? cols[1] : 0;
  load_tile<Swizzle, BS, D, C::NT>(Bs + C::TILE, Operand(a.Q, a.lq, bh), r * BS, t);
  cp_async_commit();
  if (nblk > 0) load_tile<Swizzle, BS, D, C::NT>(Bs, Kb, c_cur * BS, t);
  cp_async_commit();
  cp_async_wait<1>();
  group_sync<C::NT>(g0);
  make_frags<BS, D, MT>(frags, Bs + C::TILE, row0, lane);
  group_sync<C::NT>(g0);

  // ---- pass 1: scores into the P tiles, running maximum and denominator of the thread's own columns
  float mx[MT][2], l[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) { mx[m][h] = a.floor_v * LOG2_E; l[m][h] = 0.f; }
  bool ok = true;
  for (int k = 0; k < nblk; ++k) {
    const int col = c_cur;
    if (k + 1 < nblk) load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Kb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < nblk ? cols[k + 2] : 0;
    cp_async_wait<1>();
    group_sync<C::NT>(g0);                                              // tile k has landed
    float* tile = mine + (long long)k * rt.step;
#pragma unroll 1                                                        // unrolled, 64-wide blocks overflow the instruction cache
    for (int ks = 0; ks < BS / 32; ++ks) {
      float s[MT][4][4];
      tile_abt<BS, D, MT>(frags, Bs + (k & 1) * C::TILE, 32 * ks, lane, s);
      float pad[2][4] = {};
      if (kp) {
#pragma unroll
        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
          for (int y = 0; y < 4; ++y) pad[jj][y] = kp[col * BS + 32 * ks + 16 * jj + y] * LOG2_E;
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4 v[2];
#pragma unroll
          for (int jj = 0; jj < 2; ++jj) {
            v[jj] = quad(s[m], jj, h);
            v[jj].x = fmaf(v[jj].x, scale2, -pad[jj][0]); v[jj].y = fmaf(v[jj].y, scale2, -pad[jj][1]);
            v[jj].z = fmaf(v[jj].z, scale2, -pad[jj][2]); v[jj].w = fmaf(v[jj].w, scale2, -pad[jj][3]);
            store_vals(tile + (16 * m + 8 * h) * rt.si + 32 * ks + 16 * jj, v[jj], vec);
          }
          const float m_new = fmaxf(fmaxf(mx[m][h], fmaxf(fmaxf(v[0].x, v[0].y), fmaxf(v[0].z, v[0].w))), fmaxf(fmaxf(v[1].x, v[1].y), fmaxf(v[1].z, v[1].w)));
          const float e = ((ex2(v[0].x - m_new) + ex2(v[0].y - m_new)) + (ex2(v[0].z - m_new) + ex2(v[0].w - m_new))) +
                          ((ex2(v[1].x - m_new) + ex2(v[1].y - m_new)) + (ex2(v[1].z - m_new) + ex2(v[1].w - m_new)));
          l[m][h] = fmaf(l[m][h], ex2(mx[m][h] - m_new), e);
          mx[m][h] = m_new;
        }
    }
    group_sync<C::NT>(g0);                                              // buffer k & 1 may be refilled
  }
  c_cur = nblk > 0 ? cols[0] : 0;
  c_nxt = nblk > 1 ? cols[1] : 0;
  if (nblk > 0) load_tile<Swizzle, BS, D, C::NT>(Bs, Vb, c_cur * BS, t);
  cp_async_commit();
  float inv[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float row_m = quad_max(mx[m][h]), z = quad_sum(l[m][h] * ex2(mx[m][h] - row_m));
      inv[m][h] = 1.0f / (z + (float)(a.L - nblk * BS) * ex2(-row_m));
      mx[m][h] = inv[m][h] == 0.f ? INFINITY : row_m;                   // every P is zero then
      ok = ok && fabsf(z) <= 3.402823466e38f;                           // a score that is no number, or +infinity, makes z a NaN
    }

  // ---- pass 2: probabilities over the scores, O = P V
  float o[C::NH][MT][4][4];
#pragma unroll
  for (int h = 0; h < C::NH; ++h) clear(o[h]);
  for (int k = 0; k < nblk; ++k) {
    if (k + 1 < nblk) load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Vb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < nblk ? cols[k + 2] : 0;
    float* tile = mine + (long long)k * rt.step;
#pragma unroll 1
    for (int ks = 0; ks < BS / 32; ++ks) {
      float* part = tile + 32 * ks;
      float4 v[2][MT][2];                                               // scores; of the first 32 keys before the wait
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) v[jj][m][h] = load_vals(part + (16 * m + 8 * h) * rt.si + 16 * jj, vec);
      if (ks == 0) {
        cp_async_wait<1>();
        group_sync<C::NT>(g0);                                          // V tile k has landed
      }
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {                                  // 16 keys
        FragA f[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float4& e = v[jj][m][h];
            const float mr = mx[m][h], i = inv[m][h];
            e.x = ex2(e.x - mr) * i; e.y = ex2(e.y - mr) * i; e.z = ex2(e.z - mr) * i; e.w = ex2(e.w - mr) * i;
            store_vals(part + (16 * m + 8 * h) * rt.si + 16 * jj, e, vec);
          }
          f[m] = frag_a(v[jj][m][0], v[jj][m][1]);
        }
        tile_ab<D, MT>(f, Bs + (k & 1) * C::TILE, 32 * ks + 16 * jj, lane, o);
      }
    }
    group_sync<C::NT>(g0);                                              // buffer k & 1 may be refilled
  }
  cp_async_wait<0>();
  ok = ok && all_as_fp32<D, MT>(o);
  if (__any_sync(0xffffffffu, !ok)) {
    __syncwarp();
    redo_fwd<BS, D, MT>(a, bh, r, row0, lane);
    return;
  }
  float* Ob = a.O + (long long)bh * a.lo.bh_stride + (long long)(r * BS + row0 + g) * a.lo.sl;
  const bool ovec = a.lo.sd == 1 && (a.lo.sl & 3) == 0 && vec_ok(a.O) && (a.lo.bh_stride & 3) == 0;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) store_row<D, MT>(Ob + (16 * m + 8 * h) * a.lo.sl, a.lo.sd, ovec, o, m, h, c);
}

// ------------------------------------------------------------------------------ backward, row side
struct RowArgs {
  const float *dO, *O, *V, *K, *P;
  OperandLayout ldo, lo, lv, lk, ldq;
  ValueLayout vp, vds;
  float *dS, *dQ;
  Pattern p;
  int BH;
  float scale;
};

// O null: the row sums of dP.P in place of those of dO.O
template <int BS, int D, int MT>
__device__ __noinline__ void redo_row(const RowArgs& a, int bh, int r, int row0, int lane) {
  constexpr int WR = Cfg<BS, D, MT>::WR;
  const Operand dOb(a.dO, a.ldo, bh), Vb(a.V, a.lv, bh), Kb(a.K, a.lk, bh);
  const int rp = a.p.row_ptr[r], nblk = a.p.row_ptr[r + 1] - rp;
  const int* cols = a.p.col_idx + rp;
  const RowTiles tp = RowTiles::of<BS>(a.vp, rp, nblk), ts = RowTiles::of<BS>(a.vds, rp, nblk);
  const float* P0 = a.P + (long long)bh * a.vp.bh_stride + tp.base + row0 * tp.si;
  float* S0 = a.dS + (long long)bh * a.vds.bh_stride + ts.base + row0 * ts.si;
  plain_abt<BS, D, WR>(dOb, r * BS + row0, Vb, cols, nblk, S0, ts.si, ts.step, lane);
  for (int x = 0; x < WR; ++x) {
    const float* Pr = P0 + x * tp.si;
    float* Sr = S0 + x * ts.si;
    const int row = r * BS + row0 + x;
    float s = 0.f;
    if (a.O) {
      for (int n = lane; n < D; n += 32)
        s = fmaf(dOb.base[row * dOb.s_row + n * dOb.s_col], a.O[(long long)bh * a.lo.bh_stride + row * a.lo.sl + n * a.lo.sd], s);
    } else {
      for (int k = 0; k < nblk; ++k)
        for (int j = lane; j < BS; j += 32) s = fmaf(Sr[(long long)k * ts.step + j], Pr[(long long)k * tp.step + j], s);
    }
    s = warp_sum(s);
    for (int k = 0; k < nblk; ++k)
      for (int j = lane; j < BS; j += 32) {
        float* e = Sr + (long long)k * ts.step + j;
        const float pv = Pr[(long long)k * tp.step + j];
        *e = a.O ? pv * (*e - s) * a.scale : (*e * pv - pv * s) * a.scale;
      }
  }
  __syncwarp();
  plain_ab<BS, D, WR>(S0, ts.si, ts.step, Kb, cols, nblk, a.dQ + (long long)bh * a.ldq.bh_stride + (r * BS + row0) * a.ldq.sl, a.ldq.sl, a.ldq.sd, lane);
}

// rowsum(dP.P) = rowsum(dO.O) (delta), so dS of a tile needs nothing from the other tiles of its row and one pass suffices.  Two stages per
// block, V tile (for dP) and K tile (for dQ); the copy of one is in flight while the other is used.
template <int BS, int D, int MT>
__global__ void __launch_bounds__(128, (Cfg<BS, D, MT>::RESIDENT)) mma_bwd_row_kernel(const __grid_constant__ RowArgs a) {
  using C = Cfg<BS, D, MT>;
  extern __shared__ __align__(16) float smem[];
  const int g0 = threadIdx.x / C::NT, t = threadIdx.x % C::NT, lane = t & 31;
  const int r = blockIdx.x, bh = blockIdx.y * C::G + g0;
  if (bh >= a.BH) return;
  float* Vs = smem + g0 * (C::NT / 32 * C::FRAGS + 2 * C::TILE);
  float* Ks = Vs + C::TILE;
  float* frags = Vs + 2 * C::TILE + (t >> 5) * C::FRAGS;
  const int row0 = (t >> 5) * C::WR, g = lane >> 2, c = lane & 3;

  const int rp = a.p.row_ptr[r], nblk = a.p.row_ptr[r + 1] - rp;
  const int* cols = a.p.col_idx + rp;
  const Operand Vb(a.V, a.lv, bh), Kb(a.K, a.lk, bh);
  const RowTiles tp = RowTiles::of<BS>(a.vp, rp, nblk), ts = RowTiles::of<BS>(a.vds, rp, nblk);
  const float* Pb = a.P + (long long)bh * a.vp.bh_stride + tp.base + (row0 + g) * tp.si + 4 * c;
  float* dSb = a.dS + (long long)bh * a.vds.bh_stride + ts.base + (row0 + g) * ts.si + 4 * c;
  const bool vec_p = vec_ok(Pb), vec_s = vec_ok(dSb);

  int c_cur = nblk > 0 ? cols[0] : 0, c_nxt = nblk > 1 ? cols[1] : 0;
  load_tile<Swizzle, BS, D, C::NT>(Ks, Operand(a.dO, a.ldo, bh), r * BS, t);
  cp_async_commit();
  if (nblk > 0) load_tile<Swizzle, BS, D, C::NT>(Vs, Vb, c_cur * BS, t);
  cp_async_commit();
  cp_async_wait<1>();
  group_sync<C::NT>(g0);
  make_frags<BS, D, MT>(frags, Ks, row0, lane);
  float delta[MT][2];
  const float* Ob = a.O + (long long)bh * a.lo.bh_stride + (long long)(r * BS + row0 + g) * a.lo.sl;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float s = 0.f;
#pragma unroll
      for (int x = 0; x < C::KS; ++x) {
        const float4 q = piece(Ks + Swizzle::at<D>(row0 + 16 * m + 8 * h + g, 4 * x + c));
        const float* o = Ob + (16 * m + 8 * h) * a.lo.sl + (16 * x + 4 * c) * a.lo.sd;
        s = fmaf(q.x, o[0], s); s = fmaf(q.y, o[a.lo.sd], s); s = fmaf(q.z, o[2 * a.lo.sd], s); s = fmaf(q.w, o[3 * a.lo.sd], s);
      }
      delta[m][h] = quad_sum(s);
    }
  group_sync<C::NT>(g0);
  if (nblk > 0) load_tile<Swizzle, BS, D, C::NT>(Ks, Kb, c_cur * BS, t);
  cp_async_commit();

  float o[C::NH][MT][4][4];
#pragma unroll
  for (int h = 0; h < C::NH; ++h) clear(o[h]);
  for (int k = 0; k < nblk; ++k) {
    const float* ptile = Pb + (long long)k * tp.step;
    float* stile = dSb + (long long)k * ts.step;
    constexpr int NK = BS / 32;
    float4 v[NK][2][MT][2];                                             // probabilities, requested before the wait; then dS
#pragma unroll
    for (int ks = 0; ks < NK; ++ks)
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) v[ks][jj][m][h] = load_vals(ptile + (16 * m + 8 * h) * tp.si + 32 * ks + 16 * jj, vec_p);
    cp_async_wait<1>();
    group_sync<C::NT>(g0);                                              // V tile k has landed
#pragma unroll 1
    for (int ks = 0; ks < NK; ++ks) {
      float dp[MT][4][4];
      tile_abt<BS, D, MT>(frags, Vs, 32 * ks, lane, dp);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float4 e = NK == 1 || ks == 0 ? v[0][jj][m][h] : v[NK - 1][jj][m][h];
            const float4 x = quad(dp[m], jj, h);
            const float dl = delta[m][h];
            e.x = e.x * (x.x - dl) * a.scale; e.y = e.y * (x.y - dl) * a.scale;
            e.z = e.z * (x.z - dl) * a.scale; e.w = e.w * (x.w - dl) * a.scale;
            store_vals(stile + (16 * m + 8 * h) * ts.si + 32 * ks + 16 * jj, e, vec_s);
            if (NK == 1 || ks == 0) v[0][jj][m][h] = e;
            else v[NK - 1][jj][m][h] = e;
          }
    }
    group_sync<C::NT>(g0);                                              // V buffer free
    if (k + 1 < nblk) load_tile<Swizzle, BS, D, C::NT>(Vs, Vb, c_nxt * BS, t);
    cp_async_commit();
    cp_async_wait<1>();
    group_sync<C::NT>(g0);                                              // K tile k has landed
#pragma unroll 1
    for (int ks = 0; ks < NK; ++ks)
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        FragA f[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float4 q0 = NK == 1 || ks == 0 ? v[0][jj][m][0] : v[NK - 1][jj][m][0], q1 = NK == 1 || ks == 0 ? v[0][jj][m][1] : v[NK - 1][jj][m][1];
          f[m] = frag_a(q0, q1);
        }
        tile_ab<D, MT>(f, Ks, 32 * ks + 16 * jj, lane, o);
      }
    group_sync<C::NT>(g0);                                              // K buffer free
    if (k + 1 < nblk) load_tile<Swizzle, BS, D, C::NT>(Ks, Kb, c_nxt * BS, t);
    cp_async_commit();
    c_cur = c_nxt;
    c_nxt = k + 2 < nblk ? cols[k + 2] : 0;
  }
  cp_async_wait<0>();
  if (__any_sync(0xffffffffu, !all_as_fp32<D, MT>(o))) {               // dQ sums over dP and dS: what is amiss there shows here
    __syncwarp();
    redo_row<BS, D, MT>(a, bh, r, row0, lane);
    return;
  }
  float* Qb = a.dQ + (long long)bh * a.ldq.bh_stride + (long long)(r * BS + row0 + g) * a.ldq.sl;
  const bool ovec = a.ldq.sd == 1 && (a.ldq.sl & 3) == 0 && vec_ok(a.dQ) && (a.ldq.bh_stride & 3) == 0;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) store_row<D, MT>(Qb + (16 * m + 8 * h) * a.ldq.sl, a.ldq.sd, ovec, o, m, h, c);
}

// Without O: t = dP.P ; s = rowsum(t) ; dS = (t - P s) scale ; dQ = dS K, two passes over the blocks with dP in the dS tiles in between.
template <int BS, int D, int MT>
__global__ void __launch_bounds__(128, (Cfg<BS, D, MT>::RESIDENT)) mma_bwd_row2_kernel(const __grid_constant__ RowArgs a) {
  using C = Cfg<BS, D, MT>;
  extern __shared__ __align__(16) float smem[];
  const int g0 = threadIdx.x / C::NT, t = threadIdx.x % C::NT, lane = t & 31;
  const int r = blockIdx.x, bh = blockIdx.y * C::G + g0;
  if (bh >= a.BH) return;
  float* Bs = smem + g0 * (C::NT / 32 * C::FRAGS + 2 * C::TILE);        // two buffers: V tiles, then K tiles
  float* frags = Bs + 2 * C::TILE + (t >> 5) * C::FRAGS;
  const int row0 = (t >> 5) * C::WR, g = lane >> 2, c = lane & 3;

  const int rp = a.p.row_ptr[r], nblk = a.p.row_ptr[r + 1] - rp;
  const int* cols = a.p.col_idx + rp;
  const Operand Vb(a.V, a.lv, bh), Kb(a.K, a.lk, bh);
  const RowTiles tp = RowTiles::of<BS>(a.vp, rp, nblk), ts = RowTiles::of<BS>(a.vds, rp, nblk);
  const float* Pb = a.P + (long long)bh * a.vp.bh_stride + tp.base + (row0 + g) * tp.si + 4 * c;
  float* dSb = a.dS + (long long)bh * a.vds.bh_stride + ts.base + (row0 + g) * ts.si + 4 * c;
  const bool vec_p = vec_ok(Pb), vec_s = vec_ok(dSb);

  int c_nxt = nblk > 1 ? cols[1] : 0;
  load_tile<Swizzle, BS, D, C::NT>(Bs + C::TILE, Operand(a.dO, a.ldo, bh), r * BS, t);
  cp_async_commit();
  if (nblk > 0) load_tile<Swizzle, BS, D, C::NT>(Bs, Vb, cols[0] * BS, t);
  cp_async_commit();
  cp_async_wait<1>();
  group_sync<C::NT>(g0);
  make_frags<BS, D, MT>(frags, Bs + C::TILE, row0, lane);
  group_sync<C::NT>(g0);

  float s[MT][2] = {};
  for (int k = 0; k < nblk; ++k) {
    if (k + 1 < nblk) load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Vb, c_nxt * BS, t);
    cp_async_commit();
    c_nxt = k + 2 < nblk ? cols[k + 2] : 0;
    cp_async_wait<1>();
    group_sync<C::NT>(g0);
#pragma unroll 1
    for (int ks = 0; ks < BS / 32; ++ks) {
      float dp[MT][4][4];
      tile_abt<BS, D, MT>(frags, Bs + (k & 1) * C::TILE, 32 * ks, lane, dp);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 x = quad(dp[m], jj, h), pv = load_vals(Pb + (long long)k * tp.step + (16 * m + 8 * h) * tp.si + 32 * ks + 16 * jj, vec_p);
            s[m][h] = fmaf(x.x, pv.x, s[m][h]); s[m][h] = fmaf(x.y, pv.y, s[m][h]);
            s[m][h] = fmaf(x.z, pv.z, s[m][h]); s[m][h] = fmaf(x.w, pv.w, s[m][h]);
            store_vals(dSb + (long long)k * ts.step + (16 * m + 8 * h) * ts.si + 32 * ks + 16 * jj, x, vec_s);
          }
    }
    group_sync<C::NT>(g0);
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) s[m][h] = quad_sum(s[m][h]);

  float o[C::NH][MT][4][4];
#pragma unroll
  for (int h = 0; h < C::NH; ++h) clear(o[h]);
  c_nxt = nblk > 1 ? cols[1] : 0;
  if (nblk > 0) load_tile<Swizzle, BS, D, C::NT>(Bs, Kb, cols[0] * BS, t);
  cp_async_commit();
  for (int k = 0; k < nblk; ++k) {
    if (k + 1 < nblk) load_tile<Swizzle, BS, D, C::NT>(Bs + ((k + 1) & 1) * C::TILE, Kb, c_nxt * BS, t);
    cp_async_commit();
    c_nxt = k + 2 < nblk ? cols[k + 2] : 0;
    cp_async_wait<1>();
    group_sync<C::NT>(g0);
#pragma unroll
    for (int jj = 0; jj < BS / 16; ++jj) {
      FragA f[MT];
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        float4 ds[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float* e = dSb + (long long)k * ts.step + (16 * m + 8 * h) * ts.si + 16 * jj;
          const float4 dp = load_vals(e, vec_s), pv = load_vals(Pb + (long long)k * tp.step + (16 * m + 8 * h) * tp.si + 16 * jj, vec_p);
          const float si = s[m][h];
          ds[h] = make_float4((dp.x * pv.x - pv.x * si) * a.scale, (dp.y * pv.y - pv.y * si) * a.scale, (dp.z * pv.z - pv.z * si) * a.scale,
                              (dp.w * pv.w - pv.w * si) * a.scale);
          store_vals(e, ds[h], vec_s);
        }
        f[m] = frag_a(ds[0], ds[1]);
      }
      tile_ab<D, MT>(f, Bs + (k & 1) * C::TILE, 16 * jj, lane, o);
    }
    group_sync<C::NT>(g0);
  }
  cp_async_wait<0>();
  if (__any_sync(0xffffffffu, !all_as_fp32<D, MT>(o))) {               // dQ sums over dP and dS: what is amiss there shows here
    __syncwarp();
    redo_row<BS, D, MT>(a, bh, r, row0, lane);
    return;
  }
  float* Qb = a.dQ + (long long)bh * a.ldq.bh_stride + (long long)(r * BS + row0 + g) * a.ldq.sl;
  const bool ovec = a.ldq.sd == 1 && (a.ldq.sl & 3) == 0 && vec_ok(a.dQ) && (a.ldq.bh_stride & 3) == 0;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) store_row<D, MT>(Qb + (16 * m + 8 * h) * a.ldq.sl, a.ldq.sd, ovec, o, m, h, c);
}

// ------------------------------------------------------------------------------ backward, column side
struct ColArgs {
  const float *dS, *P, *Q, *dO;
  ValueLayout vds, vp;
  OperandLayout lq, ldo, ldk, ldv;
  float *dK, *dV;
  Pattern p;
  int BH, share_from;
};

// Keys key0 .. key0 + WR - 1 of block column c of sum_r X(r,c)^T B[r], entries e0 .. e1 - 1
template <int BS, int D, int MT>
__device__ __noinline__ void redo_col(const Pattern& p, const float* X, const ValueLayout& vl, const float* B, const OperandLayout& lb,
                                      float* out, const OperandLayout& lo, int bh, int c, int e0, int e1, int key0, int lane) {
  constexpr int WR = Cfg<BS, D, MT>::WR;
  const Operand Bb(B, lb, bh);
  const float* X0 = X + (long long)bh * vl.bh_stride + key0;
  const bool vec = vec_ok(X0);
  for (int n = lane; n < D; n += 32) {
    float s[WR] = {};
    for (int e = e0; e < e1; ++e) {
      long long base, si, sj;
      tile_address(vl, p, p.row_idx[e], c, p.csc_pos[e], base, si, sj);
      for (int i = 0; i < BS; ++i) {
        const float b = Bb.base[(p.row_idx[e] * BS + i) * Bb.s_row + n * Bb.s_col];
#pragma unroll
        for (int x = 0; x < WR; x += 4) {
          const float4 v = load_vals(X0 + base + i * si + x, vec);
          s[x] = fmaf(v.x, b, s[x]); s[x + 1] = fmaf(v.y, b, s[x + 1]); s[x + 2] = fmaf(v.z, b, s[x + 2]); s[x + 3] = fmaf(v.w, b, s[x + 3]);
        }
      }
    }
#pragma unroll
    for (int x = 0; x < WR; ++x) out[(long long)bh * lo.bh_stride + (c * BS + key0 + x) * lo.sl + n * lo.sd] = s[x];
  }
}

// sum += X^T B over the rows of a value tile; X: [bs x bs], this warp's keys from key0 on.  Row slot (m, half) of the result: key MT 2 g + 2 m + half.
template <int BS, int D, int MT>
__device__ __forceinline__ void tile_atb(const float* X, const float* B, int key0, int lane, float (&sum)[Cfg<BS, D, MT>::NH][MT][4][4]) {
  using C = Cfg<BS, D, MT>;
  const int g = lane >> 2, c = lane & 3;
#pragma unroll 1
  for (int s = 0; s < BS / 16; ++s) {
    const int row = 16 * s + 4 * c;
    FragA f[MT];
    if constexpr (MT == 2) {
      float4 q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = piece(X + Swizzle::at<BS>(row + i, (key0 >> 2) + g));
      f[0] = frag_a(make_float4(q[0].x, q[1].x, q[2].x, q[3].x), make_float4(q[0].y, q[1].y, q[2].y, q[3].y));
      f[1] = frag_a(make_float4(q[0].z, q[1].z, q[2].z, q[3].z), make_float4(q[0].w, q[1].w, q[2].w, q[3].w));
    } else {
      float2 q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float2*>(X + Swizzle::at<BS>(row + i, (key0 >> 2) + (g >> 1)) + (g & 1) * 2);
      f[0] = frag_a(make_float4(q[0].x, q[1].x, q[2].x, q[3].x), make_float4(q[0].y, q[1].y, q[2].y, q[3].y));
    }
    tile_ab<D, MT>(f, B, 16 * s, lane, sum);
  }
}

// Two stages per entry of the column, (dS, Q) for dK and (P, dO) for dV; the copy of one is in flight while the other is used.
// SHARED: the columns of at least `share_from` entries only, by a cluster of SHARE_WAYS CTAs each; the other kernel leaves them out.
// Discovered masks have columns that every row selects; one CTA would walk such a column long after the others are done.  The CTAs of the
// cluster take a share of its entries each and the first adds the others' sums, in their order, through distributed shared memory.
// The two write different columns, so the second is launched as a programmatic dependent of the first and starts as soon as all CTAs of that one
// run (each says so first thing): the few clusters of long columns leave most of the chip idle.  It reads nothing of the first; its
// last CTA waits for the first, so that what follows on the stream comes after both.  One after the other they took 66 + 66 us (15 matrices,
// L = 3008, d 64, 8 %, a full column), now 86; forward + backward with 1, 4, 12 full columns 472, 611, 1088 -> 422, 570, 1022 us.
constexpr int SHARE_WAYS = 8, SHARE_AT_ONCE = 4;                        // CTAs of a cluster; clusters along the columns

// The i-th column of at least `from` entries, or -1.  Whole CTA.
__device__ __forceinline__ int long_column(const Pattern& p, int from, int i) {
  __shared__ int found;
  if (threadIdx.x == 0) found = -1;
  __syncthreads();
  if (threadIdx.x < 32) {
    for (int c0 = 0; c0 < p.nb; c0 += 32) {
      const int c = c0 + (int)threadIdx.x;
      const bool is = c < p.nb && p.col_ptr[c + 1] - p.col_ptr[c] >= from;
      const unsigned all = __ballot_sync(0xffffffffu, is), before = all & ((1u << threadIdx.x) - 1);
      if (is && __popc(before) == i) found = c;
      i -= __popc(all);
      if (i < 0) break;
    }
  }
  __syncthreads();
  const int c = found;
  __syncthreads();                                                      // the next call writes it again
  return c;
}

// Leaves the kernel, whichever way, only after the launch before this one is complete.  Without that attribute of the launch: at once.
struct AfterLaunchBefore {
  bool on;
  __device__ ~AfterLaunchBefore() {
    if (on) wait_for_kernel_before();
  }
};

template <int BS, int D, int MT, bool SHARED>
__global__ void __launch_bounds__(128, (Cfg<BS, D, MT>::RESIDENT)) mma_bwd_col_kernel(const __grid_constant__ ColArgs a) {
  using C = Cfg<BS, D, MT>;
  extern __shared__ __align__(16) float smem[];
  const int g0 = threadIdx.x / C::NT, t = threadIdx.x % C::NT, lane = t & 31;
  const int bh_raw = blockIdx.y * C::G + g0;
  const bool active = bh_raw < a.BH;
  if (SHARED) next_may_start();
  const AfterLaunchBefore leave{!SHARED && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1};
  if (!SHARED && !active) return;
  const int bh = active ? bh_raw : a.BH - 1;                            // SHARED: the cluster barriers take every thread
  const int part = SHARED ? blockIdx.x % SHARE_WAYS : 0;
  float* dSs = smem + g0 * (2 * C::TILE + 2 * C::VALS);
  float* Qs = dSs + C::VALS;
  float* Ps = Qs + C::TILE;
  float* Os = Ps + C::VALS;
  const int key0 = (t >> 5) * C::WR;

  const float* dSb = a.dS + (long long)bh * a.vds.bh_stride;
  const float* Pb = a.P + (long long)bh * a.vp.bh_stride;
  const Operand Qb(a.Q, a.lq, bh), dOb(a.dO, a.ldo, bh);

  for (int nth = SHARED ? blockIdx.x / SHARE_WAYS : 0;; nth += SHARE_AT_ONCE) {
    const int c = SHARED ? long_column(a.p, a.share_from, nth) : blockIdx.x;
    if (SHARED && c < 0) return;                                          // the same for all CTAs of the cluster
    const int first = a.p.col_ptr[c], last = a.p.col_ptr[c + 1], n = last - first;
    if (!SHARED && n >= a.share_from) return;
    const int e0 = first + (SHARED ? n * part / SHARE_WAYS : 0), e1 = SHARED && !active ? e0 : first + (SHARED ? n * (part + 1) / SHARE_WAYS : n);
    float ak[C::NH][MT][4][4], av[C::NH][MT][4][4];
#pragma unroll
    for (int h = 0; h < C::NH; ++h) { clear(ak[h]); clear(av[h]); }

    auto fetch_k = [&](int r, int blk) {                                 // stage A: dS tile and Q rows of entry (r, blk)
      long long b1, s1, t1;
      tile_address(a.vds, a.p, r, c, blk, b1, s1, t1);
      load_tile<Swizzle, BS, BS, C::NT>(dSs, Operand(dSb + b1, (int)s1), 0, t);
      load_tile<Swizzle, BS, D, C::NT>(Qs, Qb, r * BS, t);
    };
    auto fetch_v = [&](int r, int blk) {                                 // stage B: P tile and dO rows
      long long b2, s2, t2;
      tile_address(a.vp, a.p, r, c, blk, b2, s2, t2);
      load_tile<Swizzle, BS, BS, C::NT>(Ps, Operand(Pb + b2, (int)s2), 0, t);
      load_tile<Swizzle, BS, D, C::NT>(Os, dOb, r * BS, t);
    };
    int r_cur = e0 < e1 ? a.p.row_idx[e0] : 0, b_cur = e0 < e1 ? a.p.csc_pos[e0] : 0;
    if (e0 < e1) fetch_k(r_cur, b_cur);
    cp_async_commit();
    for (int e = e0; e < e1; ++e) {
      const int r_nxt = e + 1 < e1 ? a.p.row_idx[e + 1] : 0, b_nxt = e + 1 < e1 ? a.p.csc_pos[e + 1] : 0;
      fetch_v(r_cur, b_cur);                                              // stage B was released at the end of the last iteration
      cp_async_commit();
      cp_async_wait<1>();
      group_sync<C::NT>(g0);                                              // stage A has landed
      tile_atb<BS, D, MT>(dSs, Qs, key0, lane, ak);
      group_sync<C::NT>(g0);                                              // stage A may be refilled
      if (e + 1 < e1) fetch_k(r_nxt, b_nxt);
      cp_async_commit();
      cp_async_wait<1>();
      group_sync<C::NT>(g0);                                              // stage B has landed
      tile_atb<BS, D, MT>(Ps, Os, key0, lane, av);
      group_sync<C::NT>(g0);
      r_cur = r_nxt;
      b_cur = b_nxt;
    }
    cp_async_wait<0>();
    if (SHARED) {
      auto cluster = cooperative_groups::this_cluster();
      constexpr int N = C::NH * MT * 4;                                   // float4 sums per thread and output
      group_sync<C::NT>(g0);                                              // the tiles are read: their place takes the sums
      float4* mine = reinterpret_cast<float4*>(dSs) + t;                  // sum i of thread t at i * NT + t
      static_assert(2 * N * 4 * C::NT <= 2 * (C::TILE + C::VALS), "room for the sums");
      if (part > 0) {
#pragma unroll
        for (int h = 0; h < C::NH; ++h)
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n) {
              const int i = (h * MT + m) * 4 + n;
              mine[i * C::NT] = make_float4(ak[h][m][n][0], ak[h][m][n][1], ak[h][m][n][2], ak[h][m][n][3]);
              mine[(N + i) * C::NT] = make_float4(av[h][m][n][0], av[h][m][n][1], av[h][m][n][2], av[h][m][n][3]);
            }
      }
      cluster.sync();
      if (part == 0) {
        auto add = [](float (&sum)[4], const float4& v) { sum[0] += v.x; sum[1] += v.y; sum[2] += v.z; sum[3] += v.w; };
        for (int q = 1; q < SHARE_WAYS; ++q) {
          const float4* theirs = cluster.map_shared_rank(mine, q);
#pragma unroll
          for (int h = 0; h < C::NH; ++h)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
              for (int n = 0; n < 4; ++n) {
                const int i = (h * MT + m) * 4 + n;
                add(ak[h][m][n], theirs[i * C::NT]);
                add(av[h][m][n], theirs[(N + i) * C::NT]);
              }
        }
      }
      cluster.sync();                                                     // nobody goes on while its sums are read
    }
    const int g = lane >> 2, cc = lane & 3;
    auto put = [&](const float (&sum)[C::NH][MT][4][4], float* out, const OperandLayout& lo, const float* X, const ValueLayout& vl, const float* B,
                   const OperandLayout& lb) {
      if (__any_sync(0xffffffffu, !all_as_fp32<D, MT>(sum))) {
        redo_col<BS, D, MT>(a.p, X, vl, B, lb, out, lo, bh, c, first, last, key0, lane);
        return;
      }
      const bool vec = lo.sd == 1 && (lo.sl & 3) == 0 && vec_ok(out) && (lo.bh_stride & 3) == 0;
      float* ob = out + (long long)bh * lo.bh_stride + (long long)(c * BS + key0 + 2 * MT * g) * lo.sl;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) store_row<D, MT>(ob + (2 * m + h) * lo.sl, lo.sd, vec, sum, m, h, cc);
    };
    if (part == 0 && active) {
      put(ak, a.dK, a.ldk, a.dS, a.vds, a.Q, a.lq);
      put(av, a.dV, a.ldv, a.P, a.vp, a.dO, a.ldo);
    }
    if (!SHARED) return;
  }
}

template <int BS, int D, int MT> constexpr size_t smem_row() {
  using C = Cfg<BS, D, MT>;
  return sizeof(float) * C::G * (C::NT / 32 * C::FRAGS + 2 * C::TILE);
}
template <int BS, int D, int MT> constexpr size_t smem_col() {
  using C = Cfg<BS, D, MT>;
  return sizeof(float) * C::G * (2 * C::TILE + 2 * C::VALS);
}
// Columns: as many 16-row tiles per warp as registers allow (blocks of 64, d 32: 228 us with two, 254 with one).
template <int D> constexpr int COL_MT = D == 32 ? 2 : 1;

template <int BS, int D, int MT>
int set_attrs() {
  static std::atomic<bool> done[64];
  int dev = 0;
  SPION_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return SPION_OK;
  constexpr int CM = COL_MT<D>;
  SPION_CUDA_TRY(cudaFuncSetAttribute(mma_fwd_kernel<BS, D, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_row<BS, D, MT>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(mma_bwd_row_kernel<BS, D, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_row<BS, D, MT>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(mma_bwd_row2_kernel<BS, D, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_row<BS, D, MT>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(mma_bwd_col_kernel<BS, D, CM, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_col<BS, D, CM>()));
  SPION_CUDA_TRY(cudaFuncSetAttribute(mma_bwd_col_kernel<BS, D, CM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_col<BS, D, CM>()));
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return SPION_OK;
}

template <int BS, int D, int MT>
int fwd_launch(const FwdArgs& a, cudaStream_t st) {
  using C = Cfg<BS, D, MT>;
  int rc = set_attrs<BS, D, MT>();
  if (rc) return rc;
  mma_fwd_kernel<BS, D, MT><<<dim3(a.p.nb, (a.BH + C::G - 1) / C::G), C::CTA, smem_row<BS, D, MT>(), st>>>(a);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

template <int BS, int D, int MT>
int bwd_launch(const RowArgs& ra, ColArgs& ca, int nnzb, int longest, cudaStream_t st, spion_ctx* prof) {
  using R = Cfg<BS, D, MT>;
  constexpr int CM = COL_MT<D>;
  using C = Cfg<BS, D, CM>;
  int rc = set_attrs<BS, D, MT>();
  if (rc) return rc;
  const dim3 rgrid(ra.p.nb, (ra.BH + R::G - 1) / R::G), cgrid(ra.p.nb, (ra.BH + C::G - 1) / C::G);
  if (ra.O) mma_bwd_row_kernel<BS, D, MT><<<rgrid, R::CTA, smem_row<BS, D, MT>(), st>>>(ra);
  else mma_bwd_row2_kernel<BS, D, MT><<<rgrid, R::CTA, smem_row<BS, D, MT>(), st>>>(ra);
  SPION_LAUNCH_CHECK();
  if (prof) prof_mark(prof, SPION_STAGE_BWD_ROW);
  // A column is worth sharing when it alone takes half as long as all entries of all columns do on the whole chip, and twice as long as the
  // average one.  (Blocks of 64 at d 32: the tiles leave room for two CTAs and not three.  With two here and for the registers, full columns
  // took 2 to 4 % longer: 9 matrices, 64 x 64 blocks, two full columns, forward + backward 269 -> 280 us.)
  const long long at_once = (long long)sm_count() * C::RESIDENT * C::G, entries = (long long)ca.BH * nnzb;
  long long from = entries / (2 * at_once) + 1;
  if (from < 2LL * nnzb / ca.p.nb + 1) from = 2LL * nnzb / ca.p.nb + 1;
  ca.share_from = from <= longest ? (int)from : ca.p.nb + 1;
  if (from <= longest) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SHARE_WAYS * SHARE_AT_ONCE, cgrid.y);
    cfg.blockDim = dim3(C::CTA);
    cfg.dynamicSmemBytes = smem_col<BS, D, CM>();
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = SHARE_WAYS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SPION_CUDA_TRY(cudaLaunchKernelEx(&cfg, mma_bwd_col_kernel<BS, D, CM, true>, ca));
    if (prof) prof->launches += 1;                                      // the caller counts one launch per direction
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = cgrid;
  cfg.blockDim = dim3(C::CTA);
  cfg.dynamicSmemBytes = smem_col<BS, D, CM>();
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = from <= longest ? 1 : 0;                               // never beside the row kernel, whose dS it reads
  SPION_CUDA_TRY(cudaLaunchKernelEx(&cfg, mma_bwd_col_kernel<BS, D, CM, false>, ca));
  if (prof) prof_mark(prof, SPION_STAGE_SPMM_DKDV);
  return SPION_OK;
}

}  // namespace

// Blocks of 32, d 32: one 16-row tile per warp, twice as many warps, while rows are few.  us of forward + rows with one and two, rows of 5 blocks:
// 640 rows 48, 59; 1024 61, 66; 1536 80, 84; 1792 88, 93; 2560 117, 120; 3072 135, 132; 4096 171, 165; 8192 311, 286.
#define SPION_MMA_DISPATCH(FN, ...)                                                                                      \
  do {                                                                                                                  \
    const long long rows = (long long)p.nb * BH;                                                                        \
    if (p.bs == 32 && d == 32) return rows <= 12LL * sm_count() ? FN<32, 32, 1>(__VA_ARGS__) : FN<32, 32, 2>(__VA_ARGS__); \
    if (p.bs == 32 && d == 64) return FN<32, 64, 1>(__VA_ARGS__);                                                       \
    if (p.bs == 64 && d == 32) return FN<64, 32, 1>(__VA_ARGS__);                                                       \
    if (p.bs == 64 && d == 64) return FN<64, 64, 1>(__VA_ARGS__);                                                       \
    return SPION_ERR_UNSUPPORTED;                                                                                       \
  } while (0)

int mma_fused_forward(const float* Q, OperandLayout lq, const float* K, OperandLayout lk, const float* V, OperandLayout lv, const float* keypad,
                      float floor_v, float* P, ValueLayout vl, float* O, OperandLayout lo, Pattern p, int BH, int L, int d, float scale,
                      cudaStream_t st) {
  const FwdArgs a{Q, K, V, keypad, lq, lk, lv, lo, floor_v, scale, P, O, vl, p, BH, L};
  SPION_MMA_DISPATCH(fwd_launch, a, st);
}

int mma_fused_backward(const float* Q, OperandLayout lq, const float* K, OperandLayout lk, const float* V, OperandLayout lv, const float* P,
                       ValueLayout vp, const float* O, OperandLayout lo, const float* dO, OperandLayout ldo, float* dS, ValueLayout vds, float* dQ,
                       OperandLayout ldq, float* dK, OperandLayout ldk, float* dV, OperandLayout ldv, Pattern p, int BH, int d, float scale,
                       cudaStream_t st, spion_ctx* prof, int nnzb, int longest_col) {
  const RowArgs ra{dO, O, V, K, P, ldo, lo, lv, lk, ldq, vp, vds, dS, dQ, p, BH, scale};
  ColArgs ca{dS, P, Q, dO, vds, vp, lq, ldo, ldk, ldv, dK, dV, p, BH, 0};
  SPION_MMA_DISPATCH(bwd_launch, ra, ca, nnzb, longest_col < 0 ? p.nb : longest_col, st, prof);
}
