// SIMT (CUDA-core, fp32 accumulate) kernels of the block-sparse attention path.
//
// They serve (1) the reference's fp32 layouts behind the drop-in entry points, where the
// 1e-4 max-abs parity bound rules out TF32/BF16 tensor-core inputs, and (2) every shape the
// tcgen05 engine does not cover.  Each kernel works on whole bs x bs blocks of the layer's
// mask; value tiles and dense operands are addressed through strides so that the reference's
// element-CSR layout, its transposed operands (models/attention_blockcuda.py:48,80), its
// S^T-stored dense attention (models/attention_cuda.py:36) and the native block-tile layout
// all go through the same code.
//
//   simt_sddmm        replaces cusparseSDDMM      (models/block_attn.cu:145-224, calls :459,:498)
//   simt_spmm         replaces cusparseSpMM N / T (models/block_attn.cu:236-393, calls :478,:516,:526,:536)
//   softmax_fwd_rows  replaces scale_softmax_kernel            (models/block_attn.cu:33-88, _mask.cu:88-140)
//   softmax_bwd_rows  replaces softmax_scale_backward_kernel   (models/block_attn.cu:90-130)
//   softmax_*_dense_t replace max_sum_exp_kernel[_large] / softmax_scale_backward_kernel[_large]
//                     (models/attn.cu:9-112, models/attn_mask.cu:8-122)
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int KC = 32;   // contraction chunk held in shared memory

template <typename T>
__device__ __forceinline__ float load_op(const T* base, long long idx) { return to_f32(base[idx]); }

// ------------------------------------------------------------------------------ SDDMM
// One CTA per (block, bh): vals(i,j) = sum_n A[r*bs+i, n] * B[c*bs+j, n].
template <typename TI, typename TV, int TM>
__global__ void __launch_bounds__(256) sddmm_kernel(const TI* __restrict__ A, OperandLayout la, const TI* __restrict__ B,
                                                    OperandLayout lb, TV* __restrict__ vals, ValueLayout vl, Pattern p,
                                                    int d) {
  constexpr int BS = TM * 16;
  __shared__ float As[KC][BS + 1];
  __shared__ float Bs[KC][BS + 1];
  const int blk = blockIdx.x, bh = blockIdx.y;
  const int r = p.blk_row[blk], c = p.col_idx[blk];
  const TI* Ab = A + (long long)bh * la.bh_stride + (long long)r * BS * la.sl;
  const TI* Bb = B + (long long)bh * lb.bh_stride + (long long)c * BS * lb.sl;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  float acc[TM][TM];
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TM; ++b) acc[a][b] = 0.f;

  for (int n0 = 0; n0 < d; n0 += KC) {
    for (int idx = tid; idx < BS * KC; idx += 256) {
      int i, n;
      if (la.sd == 1) { n = idx % KC; i = idx / KC; } else { i = idx % BS; n = idx / BS; }
      As[n][i] = load_op(Ab, (long long)i * la.sl + (long long)(n0 + n) * la.sd);
      if (lb.sd == 1) { n = idx % KC; i = idx / KC; } else { i = idx % BS; n = idx / BS; }
      Bs[n][i] = load_op(Bb, (long long)i * lb.sl + (long long)(n0 + n) * lb.sd);
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < KC; ++k) {
      float a[TM], b[TM];
#pragma unroll
      for (int m = 0; m < TM; ++m) a[m] = As[k][ty * TM + m];
#pragma unroll
      for (int m = 0; m < TM; ++m) b[m] = Bs[k][tx * TM + m];
#pragma unroll
      for (int x = 0; x < TM; ++x)
#pragma unroll
        for (int y = 0; y < TM; ++y) acc[x][y] = fmaf(a[x], b[y], acc[x][y]);
    }
    __syncthreads();
  }
  long long base, si, sj;
  tile_address(vl, p, r, c, blk, base, si, sj);
  TV* out = vals + (long long)bh * vl.bh_stride + base;
#pragma unroll
  for (int x = 0; x < TM; ++x)
#pragma unroll
    for (int y = 0; y < TM; ++y) out[(long long)(ty * TM + x) * si + (long long)(tx * TM + y) * sj] = from_f32<TV>(acc[x][y]);
}

// ------------------------------------------------------------------------------ SpMM
// TRANS == false: one CTA per (block row r, bh):  out[r*bs+i, :] = sum_{c in row r} vals_{r,c}(i,j) * Bop[c*bs+j, :]
// TRANS == true : one CTA per (block col c, bh):  out[c*bs+j, :] = sum_{r in col c} vals_{r,c}(i,j) * Bop[r*bs+i, :]
// Output columns are produced 32 at a time (grid.z chunks of the head dimension).
template <typename TV, typename TO, int TM, bool TRANS>
__global__ void __launch_bounds__(256) spmm_kernel(const TV* __restrict__ vals, ValueLayout vl, const TO* __restrict__ Bop,
                                                   OperandLayout lb, TO* __restrict__ out, OperandLayout lo, Pattern p) {
  constexpr int BS = TM * 16;
  constexpr int TN = 2;                 // 16 thread columns x 2 = 32 output columns per chunk
  __shared__ float As[BS][BS + 1];      // As[k][m]
  __shared__ float Bs[BS][32 + 1];      // Bs[k][n]
  const int line = blockIdx.x, bh = blockIdx.y, n0 = blockIdx.z * 32;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int beg = TRANS ? p.col_ptr[line] : p.row_ptr[line];
  const int end = TRANS ? p.col_ptr[line + 1] : p.row_ptr[line + 1];
  const TV* vb = vals + (long long)bh * vl.bh_stride;
  const TO* Bb = Bop + (long long)bh * lb.bh_stride;
  float acc[TM][TN];
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TN; ++b) acc[a][b] = 0.f;

  for (int e = beg; e < end; ++e) {
    int r, c, blk;
    if (TRANS) { c = line; r = p.row_idx[e]; blk = p.csc_pos[e]; } else { r = line; blk = e; c = p.col_idx[e]; }
    long long base, si, sj;
    tile_address(vl, p, r, c, blk, base, si, sj);
    const TV* tile = vb + base;
    for (int idx = tid; idx < BS * BS; idx += 256) {
      int i, j;
      if (sj == 1) { j = idx % BS; i = idx / BS; } else { i = idx % BS; j = idx / BS; }
      const float v = to_f32(tile[(long long)i * si + (long long)j * sj]);
      if (TRANS) As[i][j] = v; else As[j][i] = v;
    }
    const int krow0 = (TRANS ? r : c) * BS;
    for (int idx = tid; idx < BS * 32; idx += 256) {
      int k, n;
      if (lb.sd == 1) { n = idx % 32; k = idx / 32; } else { k = idx % BS; n = idx / BS; }
      Bs[k][n] = to_f32(Bb[(long long)(krow0 + k) * lb.sl + (long long)(n0 + n) * lb.sd]);
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < BS; ++k) {
      float a[TM], b[TN];
#pragma unroll
      for (int m = 0; m < TM; ++m) a[m] = As[k][ty * TM + m];
#pragma unroll
      for (int n = 0; n < TN; ++n) b[n] = Bs[k][tx * TN + n];
#pragma unroll
      for (int x = 0; x < TM; ++x)
#pragma unroll
        for (int y = 0; y < TN; ++y) acc[x][y] = fmaf(a[x], b[y], acc[x][y]);
    }
    __syncthreads();
  }
  TO* ob = out + (long long)bh * lo.bh_stride + (long long)line * BS * lo.sl;
#pragma unroll
  for (int x = 0; x < TM; ++x)
#pragma unroll
    for (int y = 0; y < TN; ++y)
      ob[(long long)(ty * TM + x) * lo.sl + (long long)(n0 + tx * TN + y) * lo.sd] = from_f32<TO>(acc[x][y]);
}

// ------------------------------------------------------------------------------ row softmax
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per element row.  Values of a row: for each block k of block row r, bs consecutive
// elements at tile base + ii*si (sj == 1 layouts only).
//   v = S*scale - keypad[col];  m = max(floor, max v);  Z = sum exp(v-m) + (L-n_i) exp(-m);  P = exp(v-m)/Z
template <typename TP>
__global__ void __launch_bounds__(256) softmax_fwd_rows_kernel(const float* S, ValueLayout vin,   // S may alias P
                                                               TP* P, ValueLayout vout, Pattern p, int BH,
                                                               int L, float scale, const float* __restrict__ keypad,
                                                               float floor_v) {
  const long long row_g = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row_g >= (long long)BH * L) return;
  const int lane = threadIdx.x & 31;
  const int bh = (int)(row_g / L), row = (int)(row_g % L);
  const int bs = p.bs, r = row / bs, ii = row % bs;
  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const float* Sb = S + (long long)bh * vin.bh_stride;
  TP* Pb = P + (long long)bh * vout.bh_stride;
  const float* kp = keypad ? keypad + (long long)bh * L : nullptr;

  float m = floor_v;
  for (int k = 0; k < nblk; ++k) {
    const int blk = rp + k, c = p.col_idx[blk];
    long long base, si, sj;
    tile_address(vin, p, r, c, blk, base, si, sj);
    const float* src = Sb + base + (long long)ii * si;
    for (int j = lane; j < bs; j += 32) {
      float v = src[j] * scale;
      if (kp) v -= kp[c * bs + j];
      m = fmaxf(m, v);
    }
  }
  m = warp_max(m);
  float sum = 0.f;
  for (int k = 0; k < nblk; ++k) {
    const int blk = rp + k, c = p.col_idx[blk];
    long long base, si, sj;
    tile_address(vin, p, r, c, blk, base, si, sj);
    const float* src = Sb + base + (long long)ii * si;
    for (int j = lane; j < bs; j += 32) {
      float v = src[j] * scale;
      if (kp) v -= kp[c * bs + j];
      sum += expf(v - m);
    }
  }
  sum = warp_sum(sum);
  sum += (float)(L - nblk * bs) * expf(-m);
  const float inv = 1.0f / sum;
  for (int k = 0; k < nblk; ++k) {
    const int blk = rp + k, c = p.col_idx[blk];
    long long base, si, sj, obase, osi, osj;
    tile_address(vin, p, r, c, blk, base, si, sj);
    tile_address(vout, p, r, c, blk, obase, osi, osj);
    const float* src = Sb + base + (long long)ii * si;
    TP* dst = Pb + obase + (long long)ii * osi;
    for (int j = lane; j < bs; j += 32) {
      float v = src[j] * scale;
      if (kp) v -= kp[c * bs + j];
      const float pv = (inv == 0.f) ? 0.f : expf(v - m) * inv;
      dst[j] = from_f32<TP>(pv);
    }
  }
}

//   t = dP*P ; s = sum_row t ; dS = (t - P*s) * scale
template <typename TP>
__global__ void __launch_bounds__(256) softmax_bwd_rows_kernel(const float* __restrict__ dP, ValueLayout vdp,
                                                               const TP* __restrict__ P, ValueLayout vp,
                                                               TP* __restrict__ dS, ValueLayout vds, Pattern p, int BH,
                                                               int L, float scale) {
  const long long row_g = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row_g >= (long long)BH * L) return;
  const int lane = threadIdx.x & 31;
  const int bh = (int)(row_g / L), row = (int)(row_g % L);
  const int bs = p.bs, r = row / bs, ii = row % bs;
  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const float* dPb = dP + (long long)bh * vdp.bh_stride;
  const TP* Pb = P + (long long)bh * vp.bh_stride;
  TP* dSb = dS + (long long)bh * vds.bh_stride;
  float s = 0.f;
  for (int k = 0; k < nblk; ++k) {
    const int blk = rp + k, c = p.col_idx[blk];
    long long b1, s1, t1, b2, s2, t2;
    tile_address(vdp, p, r, c, blk, b1, s1, t1);
    tile_address(vp, p, r, c, blk, b2, s2, t2);
    const float* a = dPb + b1 + (long long)ii * s1;
    const TP* q = Pb + b2 + (long long)ii * s2;
    for (int j = lane; j < bs; j += 32) s += a[j] * to_f32(q[j]);
  }
  s = warp_sum(s);
  for (int k = 0; k < nblk; ++k) {
    const int blk = rp + k, c = p.col_idx[blk];
    long long b1, s1, t1, b2, s2, t2, b3, s3, t3;
    tile_address(vdp, p, r, c, blk, b1, s1, t1);
    tile_address(vp, p, r, c, blk, b2, s2, t2);
    tile_address(vds, p, r, c, blk, b3, s3, t3);
    const float* a = dPb + b1 + (long long)ii * s1;
    const TP* q = Pb + b2 + (long long)ii * s2;
    TP* o = dSb + b3 + (long long)ii * s3;
    for (int j = lane; j < bs; j += 32) {
      const float pv = to_f32(q[j]);
      o[j] = from_f32<TP>((a[j] * pv - pv * s) * scale);
    }
  }
}

// ---- rows of 32- or 64-wide blocks in 16-byte pieces: sixteen lanes per element row
// Lane hl of a row's sixteen owns four consecutive values of one block per step: step `it` covers block it (64-wide)
// or blocks 2 it and 2 it + 1 (32-wide).  Rows of at most 16 * 4 * ROW_STEPS_* values are read once into registers, all
// loads of a lane issued before the first use, and written once; longer rows make two passes.  Needs 16-byte
// aligned value arrays (8 bytes for bf16), which the launchers check; same formulas as the kernels above, other
// summation order.
constexpr int ROW_STEPS_FWD = 8, ROW_STEPS_BWD = 4;   // measured: deeper caches cost occupancy in the backward

template <int BS>
struct RowPiece {
  const int nblk, hl;
  __device__ __forceinline__ RowPiece(int nblk_, int hl_) : nblk(nblk_), hl(hl_) {}
  __device__ __forceinline__ int steps() const { return BS == 64 ? nblk : (nblk + 1) >> 1; }
  __device__ __forceinline__ int block(int it) const { return BS == 64 ? it : 2 * it + (hl >> 3); }
  __device__ __forceinline__ bool valid(int it) const { return block(it) < nblk; }
  __device__ __forceinline__ int col() const { return BS == 64 ? hl * 4 : (hl & 7) * 4; }
};

// Start of element row ii's values inside one (b,h) matrix and the distance between its slices of consecutive blocks.
__device__ __forceinline__ void row_base(const ValueLayout& vl, int bs, int rp, int nblk, int ii, long long& base,
                                         int& kstride) {
  if (vl.mode == VAL_ELEMCSR) {
    base = (long long)rp * bs * bs + (long long)ii * nblk * bs;
    kstride = bs;
  } else {
    base = (long long)rp * bs * bs + (long long)ii * bs;
    kstride = bs * bs;
  }
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&w.x);
  const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&w.y);
  const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  uint2 w;
  w.x = *reinterpret_cast<const unsigned*>(&lo);
  w.y = *reinterpret_cast<const unsigned*>(&hi);
  *reinterpret_cast<uint2*>(p) = w;
}
__device__ __forceinline__ float half_max(unsigned mask, float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(mask, v, o));
  return v;
}
__device__ __forceinline__ float half_sum(unsigned mask, float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}
// The forward works in base-2 units (one multiply and one ex2 per value instead of a full-range expf; the issue
// slots were the kernel's second limit after the bytes in flight): v2 = S * (scale * log2 e) - keypad * log2 e.
constexpr float ROW_LOG2E = 1.4426950408889634f;
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float4 scaled(float4 v, float scale2, const float* kp) {
  v.x *= scale2, v.y *= scale2, v.z *= scale2, v.w *= scale2;
  if (kp) {
    const float4 k = load4(kp);
    v.x = fmaf(-k.x, ROW_LOG2E, v.x), v.y = fmaf(-k.y, ROW_LOG2E, v.y);
    v.z = fmaf(-k.z, ROW_LOG2E, v.z), v.w = fmaf(-k.w, ROW_LOG2E, v.w);
  }
  return v;
}
__device__ __forceinline__ float max4(float m, float4 v) { return fmaxf(fmaxf(m, fmaxf(v.x, v.y)), fmaxf(v.z, v.w)); }
__device__ __forceinline__ float4 exp4(float4 v, float m) {
  return make_float4(ex2f(v.x - m), ex2f(v.y - m), ex2f(v.z - m), ex2f(v.w - m));
}

template <typename TP, int BS>
__global__ void __launch_bounds__(256, 4) softmax_fwd_rows16_kernel(const float* S, ValueLayout vin,   // S may alias P
                                                                    TP* P, ValueLayout vout, Pattern p, int BH, int L,
                                                                    float scale, const float* __restrict__ keypad,
                                                                    float floor_v) {
  const unsigned ctas_per_bh = (unsigned)L >> 4;   // L is a multiple of the block size
  const int bh = (int)(blockIdx.x / ctas_per_bh), row = (int)(blockIdx.x % ctas_per_bh) * 16 + (threadIdx.x >> 4);
  const unsigned hmask = 0xffffu << (threadIdx.x & 16);
  const int r = row / BS, ii = row % BS;
  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const RowPiece<BS> pc(nblk, threadIdx.x & 15);
  long long ibase, obase;
  int iks, oks;
  row_base(vin, BS, rp, nblk, ii, ibase, iks);
  row_base(vout, BS, rp, nblk, ii, obase, oks);
  const float* src = S + (long long)bh * vin.bh_stride + ibase + pc.col();
  TP* dst = P + (long long)bh * vout.bh_stride + obase + pc.col();
  const float* kp = keypad ? keypad + (long long)bh * L + pc.col() : nullptr;
  const int nsteps = pc.steps(), nvals = nblk * BS;
  const float scale2 = scale * ROW_LOG2E, floor2 = floor_v * ROW_LOG2E;

  if (nsteps <= ROW_STEPS_FWD) {
    float4 v[ROW_STEPS_FWD];
#pragma unroll
    for (int it = 0; it < ROW_STEPS_FWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it)) v[it] = load4(src + pc.block(it) * iks);
    }
    float m = floor2;
#pragma unroll
    for (int it = 0; it < ROW_STEPS_FWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it)) {
        v[it] = scaled(v[it], scale2, kp ? kp + p.col_idx[rp + pc.block(it)] * BS : nullptr);
        m = max4(m, v[it]);
      }
    }
    m = half_max(hmask, m);
    float sum = 0.f;
#pragma unroll
    for (int it = 0; it < ROW_STEPS_FWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it)) {
        v[it] = exp4(v[it], m);
        sum += (v[it].x + v[it].y) + (v[it].z + v[it].w);
      }
    }
    sum = half_sum(hmask, sum) + (float)(L - nvals) * ex2f(-m);
    const float inv = 1.0f / sum;
#pragma unroll
    for (int it = 0; it < ROW_STEPS_FWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it)) {
        const float4 o = (inv == 0.f) ? make_float4(0.f, 0.f, 0.f, 0.f)
                                      : make_float4(v[it].x * inv, v[it].y * inv, v[it].z * inv, v[it].w * inv);
        store4(dst + pc.block(it) * oks, o);
      }
    }
    return;
  }

  // Longer rows, two passes with the loads of four steps in flight: (1) per lane the running maximum and the sum of
  // exponentials relative to it (rescaled when the maximum rises), joined over the sixteen lanes; (2) P.
  auto value = [&](int it) {
    return scaled(load4(src + pc.block(it) * iks), scale2, kp ? kp + p.col_idx[rp + pc.block(it)] * BS : nullptr);
  };
  float m = floor2, sum = 0.f;
  for (int it0 = 0; it0 < nsteps; it0 += 4) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (it0 + u < nsteps && pc.valid(it0 + u)) v[u] = value(it0 + u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (it0 + u < nsteps && pc.valid(it0 + u)) {
        const float vm = max4(m, v[u]);
        if (vm > m) {
          sum *= ex2f(m - vm);
          m = vm;
        }
        const float4 e = exp4(v[u], m);
        sum += (e.x + e.y) + (e.z + e.w);
      }
  }
  const float mrow = half_max(hmask, m);
  sum = half_sum(hmask, sum * ex2f(m - mrow)) + (float)(L - nvals) * ex2f(-mrow);
  const float inv = 1.0f / sum;
  for (int it0 = 0; it0 < nsteps; it0 += 4) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (it0 + u < nsteps && pc.valid(it0 + u)) v[u] = value(it0 + u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (it0 + u < nsteps && pc.valid(it0 + u)) {
        const float4 e = exp4(v[u], mrow);
        store4(dst + pc.block(it0 + u) * oks, (inv == 0.f) ? make_float4(0.f, 0.f, 0.f, 0.f)
                                                             : make_float4(e.x * inv, e.y * inv, e.z * inv, e.w * inv));
      }
  }
}

template <typename TP, int BS>
__global__ void __launch_bounds__(256, 4) softmax_bwd_rows16_kernel(const float* __restrict__ dP, ValueLayout vdp,
                                                                    const TP* __restrict__ P, ValueLayout vp,
                                                                    TP* __restrict__ dS, ValueLayout vds, Pattern p,
                                                                    int BH, int L, float scale) {
  const unsigned ctas_per_bh = (unsigned)L >> 4;   // L is a multiple of the block size
  const int bh = (int)(blockIdx.x / ctas_per_bh), row = (int)(blockIdx.x % ctas_per_bh) * 16 + (threadIdx.x >> 4);
  const unsigned hmask = 0xffffu << (threadIdx.x & 16);
  const int r = row / BS, ii = row % BS;
  const int rp = p.row_ptr[r], nblk = p.row_ptr[r + 1] - rp;
  const RowPiece<BS> pc(nblk, threadIdx.x & 15);
  long long b1, b2, b3;
  int k1, k2, k3;
  row_base(vdp, BS, rp, nblk, ii, b1, k1);
  row_base(vp, BS, rp, nblk, ii, b2, k2);
  row_base(vds, BS, rp, nblk, ii, b3, k3);
  const float* pa = dP + (long long)bh * vdp.bh_stride + b1 + pc.col();
  const TP* pq = P + (long long)bh * vp.bh_stride + b2 + pc.col();
  TP* po = dS + (long long)bh * vds.bh_stride + b3 + pc.col();
  const int nsteps = pc.steps();

  if (nsteps <= ROW_STEPS_BWD) {
    float4 a[ROW_STEPS_BWD], q[ROW_STEPS_BWD];
#pragma unroll
    for (int it = 0; it < ROW_STEPS_BWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it)) {
        a[it] = load4(pa + pc.block(it) * k1);
        q[it] = load4(pq + pc.block(it) * k2);
      }
    }
    float s = 0.f;
#pragma unroll
    for (int it = 0; it < ROW_STEPS_BWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it)) {
        a[it].x *= q[it].x, a[it].y *= q[it].y, a[it].z *= q[it].z, a[it].w *= q[it].w;
        s += (a[it].x + a[it].y) + (a[it].z + a[it].w);
      }
    }
    s = half_sum(hmask, s);
#pragma unroll
    for (int it = 0; it < ROW_STEPS_BWD; ++it) {
      if (it >= nsteps) break;
      if (pc.valid(it))
        store4(po + pc.block(it) * k3,
               make_float4((a[it].x - q[it].x * s) * scale, (a[it].y - q[it].y * s) * scale,
                           (a[it].z - q[it].z * s) * scale, (a[it].w - q[it].w * s) * scale));
    }
    return;
  }

  float s = 0.f;
  for (int it = 0; it < nsteps; ++it)
    if (pc.valid(it)) {
      const float4 a = load4(pa + pc.block(it) * k1), q = load4(pq + pc.block(it) * k2);
      s += (a.x * q.x + a.y * q.y) + (a.z * q.z + a.w * q.w);
    }
  s = half_sum(hmask, s);
  for (int it = 0; it < nsteps; ++it)
    if (pc.valid(it)) {
      const float4 a = load4(pa + pc.block(it) * k1), q = load4(pq + pc.block(it) * k2);
      store4(po + pc.block(it) * k3,
             make_float4((a.x * q.x - q.x * s) * scale, (a.y * q.y - q.y * s) * scale, (a.z * q.z - q.z * s) * scale,
                         (a.w * q.w - q.w * s) * scale));
    }
}

// Dense attention stored transposed (value(i,j) at j*L + i).  A CTA owns 32 consecutive query rows (lane = row, so
// that a warp touches 128 consecutive bytes per key) and its DENSE_WARPS warps split the keys; the row statistics
// of the slices meet in shared memory.  Three passes over the CTA's [L x 32] strip (maximum, sum, write), which
// stays in L2 between them.  Semantics as softmax_fwd_rows_kernel at full density (models/attn.cu:9-36).
constexpr int DENSE_WARPS = 8;

__global__ void __launch_bounds__(DENSE_WARPS * 32) softmax_fwd_dense_t_kernel(float* __restrict__ S, int L, float scale,
                                                                               const float* __restrict__ keypad,
                                                                               float floor_v) {
  __shared__ float s_red[DENSE_WARPS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  const int bh = blockIdx.y;
  const bool live = i < L;
  float* Sb = S + (long long)bh * L * L + (live ? i : 0);
  const float* kp = keypad ? keypad + (long long)bh * L : nullptr;
  const int per = (L + DENSE_WARPS - 1) / DENSE_WARPS, j0 = w * per, j1 = min(L, j0 + per);
  float m = floor_v;
  if (live) {
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      float v = Sb[(long long)j * L] * scale;
      if (kp) v -= kp[j];
      m = fmaxf(m, v);
    }
  }
  s_red[w][lane] = m;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k) m = fmaxf(m, s_red[k][lane]);
  __syncthreads();
  float sum = 0.f;
  if (live) {
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      float v = Sb[(long long)j * L] * scale;
      if (kp) v -= kp[j];
      sum += expf(v - m);
    }
  }
  s_red[w][lane] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k) sum += s_red[k][lane];      // slices added in slice order
  const float inv = 1.0f / sum;
  if (live) {
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      float v = Sb[(long long)j * L] * scale;
      if (kp) v -= kp[j];
      Sb[(long long)j * L] = expf(v - m) * inv;
    }
  }
}

// dS = (dP . P - P rowsum(dP . P)) scale (models/attn.cu:67-87), same decomposition.
__global__ void __launch_bounds__(DENSE_WARPS * 32) softmax_bwd_dense_t_kernel(const float* __restrict__ dP,
                                                                               const float* __restrict__ P,
                                                                               float* __restrict__ dS, int L, float scale) {
  __shared__ float s_red[DENSE_WARPS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  const int bh = blockIdx.y;
  const bool live = i < L;
  const long long o = (long long)bh * L * L + (live ? i : 0);
  const int per = (L + DENSE_WARPS - 1) / DENSE_WARPS, j0 = w * per, j1 = min(L, j0 + per);
  float s = 0.f;
  if (live) {
#pragma unroll 4
    for (int j = j0; j < j1; ++j) s += dP[o + (long long)j * L] * P[o + (long long)j * L];
  }
  s_red[w][lane] = s;
  __syncthreads();
  s = 0.f;
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k) s += s_red[k][lane];
  if (live) {
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      const float pv = P[o + (long long)j * L];
      dS[o + (long long)j * L] = (dP[o + (long long)j * L] * pv - pv * s) * scale;
    }
  }
}

// The same with the slab on chip: sixteen columns per CTA, their values in shared memory (backward: P there, dP in registers), so
// that they are read once instead of three times (twice) and all loads of a CTA are in flight together; two or three
// CTAs per SM overlap one's loads with another's arithmetic.  Slices, expressions and order of additions are those above.
// 16 matrices, L = 1024 (64 MB each way): 65 -> 30 us, backward 80 -> 68.
constexpr int SLAB = 16;
__host__ __device__ inline int slab_per(int L) { return (L + DENSE_WARPS - 1) / DENSE_WARPS; }
__host__ __device__ inline int slab_slice(int L) { return slab_per(L) * SLAB + SLAB; }   // floats; the pad keeps a warp's two slices on different banks
__device__ __forceinline__ void load_slab(float* slab, const float* src, int L) {        // src: row 0 of the CTA's columns
  const int per = slab_per(L);
  for (int e = threadIdx.x; e < L * (SLAB / 4); e += DENSE_WARPS * SLAB) {
    const int j = e / (SLAB / 4), c4 = e % (SLAB / 4), w = j / per;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(slab + w * slab_slice(L) + (j - w * per) * SLAB + c4 * 4)),
                 "l"(src + (long long)j * L + c4 * 4) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(DENSE_WARPS * SLAB) softmax_fwd_dense_t_slab(float* __restrict__ S, int L, float scale,
                                                                               const float* __restrict__ keypad, float floor_v) {
  extern __shared__ __align__(16) float s_slab[];
  __shared__ float s_red[DENSE_WARPS][SLAB];
  const int col = threadIdx.x % SLAB, w = threadIdx.x / SLAB;
  const int per = slab_per(L), j0 = w * per, n = max(0, min(L, j0 + per) - j0);
  float* Sb = S + (long long)blockIdx.y * L * L + blockIdx.x * SLAB;
  const float* kp = keypad ? keypad + (long long)blockIdx.y * L + j0 : nullptr;
  const float* x = s_slab + w * slab_slice(L) + col;
  load_slab(s_slab, Sb, L);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  Sb += (long long)j0 * L + col;
  float m = floor_v;
#pragma unroll 8
  for (int u = 0; u < n; ++u) {
    float v = x[u * SLAB] * scale;
    if (kp) v -= kp[u];
    m = fmaxf(m, v);
  }
  s_red[w][col] = m;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k) m = fmaxf(m, s_red[k][col]);
  __syncthreads();
  float sum = 0.f;
#pragma unroll 8
  for (int u = 0; u < n; ++u) {
    float v = x[u * SLAB] * scale;
    if (kp) v -= kp[u];
    sum += expf(v - m);
  }
  s_red[w][col] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k) sum += s_red[k][col];       // slices added in slice order
  const float inv = 1.0f / sum;
#pragma unroll 8
  for (int u = 0; u < n; ++u) {
    float v = x[u * SLAB] * scale;
    if (kp) v -= kp[u];
    Sb[(long long)u * L] = expf(v - m) * inv;
  }
}

template <int PER>
__global__ void __launch_bounds__(DENSE_WARPS * SLAB) softmax_bwd_dense_t_slab(const float* __restrict__ dP, const float* __restrict__ P,
                                                                               float* __restrict__ dS, int L, float scale) {
  extern __shared__ __align__(16) float s_slab[];
  __shared__ float s_red[DENSE_WARPS][SLAB];
  const int col = threadIdx.x % SLAB, w = threadIdx.x / SLAB;
  const int per = slab_per(L), j0 = w * per, n = max(0, min(L, j0 + per) - j0);
  const long long base = (long long)blockIdx.y * L * L + blockIdx.x * SLAB, o = base + (long long)j0 * L + col;
  const float* p = s_slab + w * slab_slice(L) + col;
  load_slab(s_slab, P + base, L);
  float x[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (u < n) x[u] = dP[o + (long long)u * L];
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (u < n) s += x[u] * p[u * SLAB];
  s_red[w][col] = s;
  __syncthreads();
  s = 0.f;
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k) s += s_red[k][col];
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (u < n) {
      const float pv = p[u * SLAB];
      dS[o + (long long)u * L] = (x[u] * pv - pv * s) * scale;
    }
}

// ------------------------------------------------------------------------------ full masks, fp32, S^T-stored values
// The reference-layout dense path: every value tile is selected, value(i, j) at j*L + i.  The block kernels above spend a scalar
// shared-memory read on every other multiply-add and hold one tile in flight; these keep the order of additions of
// every output (n, or k, ascending into one fp32 sum), so the results are the same bit for bit, with packed pairs of
// multiply-adds, 16-byte reads and cp.async.  16 matrices, L = 1024, d 32: S, dP 81 -> 31 us
// each, P V and dS K 102 -> 34, dS^T Q and P^T dO 118 -> 38; in one kernel with what follows them, or with one another, below.
__device__ __forceinline__ uint32_t dense_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void dense_cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dense_smem(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void dense_cp4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dense_smem(dst)), "l"(src) : "memory");
}
using pair_t = unsigned long long;
__device__ __forceinline__ pair_t twice(float x) {
  pair_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void fma2(pair_t& acc, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ float4 as_float4(pair_t lo, pair_t hi) {
  float4 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(lo));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(hi));
  return v;
}

// S^T[j][i] = sum_n A[i][n] B[j][n]: a 64 x 64 tile by 64 threads, rows j = ty + 8 y, columns i = 4 tx .. and 32 + 4 tx ..
constexpr int DT = 64;
__global__ void __launch_bounds__(64) sddmm_dense_kernel(const float* __restrict__ A, OperandLayout la, const float* __restrict__ B,
                                                         OperandLayout lb, float* __restrict__ vals, int L, int d) {
  __shared__ __align__(16) float As[KC][DT];           // [n][i], pieces of four i exchanged by n / 4: written along n, read along i
  __shared__ __align__(16) float Bs[DT][KC + 4];       // [j][n]
  const int t = threadIdx.x, ty = t >> 3, tx = t & 7;
  const int i0 = blockIdx.x * DT, j0 = blockIdx.y * DT, bh = blockIdx.z;
  const float* Ab = A + (long long)bh * la.bh_stride + (long long)i0 * la.sl;
  const float* Bb = B + (long long)bh * lb.bh_stride + (long long)j0 * lb.sl;
  pair_t acc[8][4];
#pragma unroll
  for (int y = 0; y < 8; ++y)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[y][x] = 0ull;
  for (int n0 = 0; n0 < d; n0 += KC) {
    if (la.sl == 1 && (la.sd & 3) == 0 && (reinterpret_cast<uintptr_t>(Ab) & 15) == 0) {
#pragma unroll
      for (int e = t; e < KC * DT / 4; e += 64) dense_cp16(&As[e >> 4][((e & 15) ^ (e >> 6)) * 4], Ab + (long long)(n0 + (e >> 4)) * la.sd + (e & 15) * 4);
    } else if (la.sd == 1 && (la.sl & 3) == 0 && (reinterpret_cast<uintptr_t>(Ab) & 15) == 0) {
#pragma unroll
      for (int e = t; e < KC * DT / 4; e += 64) {
        const int i = e >> 3, n4 = e & 7;
        const float4 v = *reinterpret_cast<const float4*>(Ab + (long long)i * la.sl + n0 + 4 * n4);
        float* to = &As[4 * n4][i ^ (4 * n4)];
        to[0] = v.x, to[DT] = v.y, to[2 * DT] = v.z, to[3 * DT] = v.w;
      }
    } else {
      for (int n = 0; n < KC; ++n) As[n][t ^ (n & ~3)] = Ab[(long long)t * la.sl + (long long)(n0 + n) * la.sd];
    }
    if (lb.sd == 1 && (lb.sl & 3) == 0 && (reinterpret_cast<uintptr_t>(Bb) & 15) == 0) {
#pragma unroll
      for (int e = t; e < DT * KC / 4; e += 64) dense_cp16(&Bs[e >> 3][(e & 7) * 4], Bb + (long long)(e >> 3) * lb.sl + n0 + (e & 7) * 4);
    } else {
      for (int e = t; e < DT * KC; e += 64) dense_cp4(&Bs[e & 63][e >> 6], Bb + (long long)(e & 63) * lb.sl + (long long)(n0 + (e >> 6)) * lb.sd);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll 2
    for (int n = 0; n < KC; n += 4) {
      float b[8][4];
#pragma unroll
      for (int y = 0; y < 8; ++y) {
        const float4 v = *reinterpret_cast<const float4*>(&Bs[ty + 8 * y][n]);
        b[y][0] = v.x, b[y][1] = v.y, b[y][2] = v.z, b[y][3] = v.w;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(&As[n + k][(4 * tx) ^ n]), hi = *reinterpret_cast<const ulonglong2*>(&As[n + k][32 + ((4 * tx) ^ n)]);
#pragma unroll
        for (int y = 0; y < 8; ++y) {
          const pair_t bb = twice(b[y][k]);
          fma2(acc[y][0], lo.x, bb), fma2(acc[y][1], lo.y, bb), fma2(acc[y][2], hi.x, bb), fma2(acc[y][3], hi.y, bb);
        }
      }
    }
    __syncthreads();
  }
  float* out = vals + (long long)bh * L * L + (long long)j0 * L + i0 + 4 * tx;
#pragma unroll
  for (int y = 0; y < 8; ++y) {
    float* row = out + (long long)(ty + 8 * y) * L;
    *reinterpret_cast<float4*>(row) = as_float4(acc[y][0], acc[y][1]);
    *reinterpret_cast<float4*>(row + 32) = as_float4(acc[y][2], acc[y][3]);
  }
}

// TRANS == false: out[i] = sum_j value(i, j) Bop[j];  true: out[j] = sum_i value(i, j) Bop[i].  Tiles of 64 rows x 32 columns, the sum over L in
// steps of 16 through two stages of T threads (a warp of its own, or both warps of a tile).  A lane has U rows by eight columns: a
// shared-memory read returns one register per lane and cycle, so eight rows take 16 such cycles for 32 packed multiply-adds, four by eight, as
// before, 12 for 16.  The sum of an output stays one chain where its bits are kept (dK), ascending.
constexpr int DK = 16;
constexpr int SPMM_STAGE = DT * (DK + 4) + DK * 36;              // floats of a stage: value tile, operand tile [k][32 + 4]
template <bool TRANS, int U, int T>
struct Spmm {
  pair_t acc[U][4];
  int row0, tx;                                                  // this lane's rows: TRANS row0 + 8 u, else row0 + u; columns 4 tx .., 16 + 4 tx ..
  __device__ __forceinline__ void run(float* smem, int t, int warp_row, int bh, int r0, int n0, int c0, int chunks, const float* vals, const float* Bop,
                                      const OperandLayout& lb, int L) {
    constexpr int VR = TRANS ? DT : DK, VC = TRANS ? DK : DT, VP = TRANS ? DK + 4 : DT;   // value tile as in memory: rows j, columns i
    const int lane = threadIdx.x & 31, ty = lane >> 2;
    tx = lane & 3;
    row0 = warp_row + (TRANS ? ty : U * ty);
    const float* vb = vals + (long long)bh * L * L + (TRANS ? (long long)r0 * L : (long long)r0);
    const float* Bb = Bop + (long long)bh * lb.bh_stride + (long long)n0 * lb.sd;
    const bool rows = lb.sd == 1 && (lb.sl & 3) == 0 && (reinterpret_cast<uintptr_t>(Bb) & 15) == 0;
    auto load = [&](int c) {
      const int k0 = (c0 + c) * DK;
      float* V = smem + (c & 1) * SPMM_STAGE;
      float* B = V + DT * (DK + 4);
      const float* v = vb + (TRANS ? (long long)k0 : (long long)k0 * L);
#pragma unroll
      for (int e = t; e < VR * VC / 4; e += T) dense_cp16(V + e / (VC / 4) * VP + e % (VC / 4) * 4, v + (long long)(e / (VC / 4)) * L + e % (VC / 4) * 4);
      if (rows) {
#pragma unroll
        for (int e = t; e < DK * 32 / 4; e += T) dense_cp16(B + (e >> 3) * 36 + (e & 7) * 4, Bb + (long long)(k0 + (e >> 3)) * lb.sl + (e & 7) * 4);
      } else {
#pragma unroll 4
        for (int e = t; e < DK * 32; e += T) dense_cp4(B + e % DK * 36 + e / DK, Bb + (long long)(k0 + e % DK) * lb.sl + (long long)(e / DK) * lb.sd);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int x = 0; x < U; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) acc[x][y] = 0ull;
    if (chunks > 0) load(0);
    for (int c = 0; c < chunks; ++c) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      if (T > 32) __syncthreads(); else __syncwarp();  // chunk c has landed; the stage of chunk c - 1 is free
      if (c + 1 < chunks) load(c + 1);
      const float* Vs = smem + (c & 1) * SPMM_STAGE;
      const float* Bs = Vs + DT * (DK + 4) + 4 * tx;
#pragma unroll
      for (int k = 0; k < DK; k += 4) {
        float a[TRANS ? U : 1][4];
        if (TRANS) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float4 v = *reinterpret_cast<const float4*>(Vs + (row0 + 8 * u) * VP + k);
            a[u][0] = v.x, a[u][1] = v.y, a[u][2] = v.z, a[u][3] = v.w;
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float r[U];
          if (!TRANS) {
#pragma unroll
            for (int u = 0; u < U; u += 4) {
              const float4 v = *reinterpret_cast<const float4*>(Vs + (k + i) * VP + row0 + u);
              r[u] = v.x, r[u + 1] = v.y, r[u + 2] = v.z, r[u + 3] = v.w;
            }
          }
          const ulonglong2 lo2 = *reinterpret_cast<const ulonglong2*>(Bs + (k + i) * 36), hi2 = *reinterpret_cast<const ulonglong2*>(Bs + (k + i) * 36 + 16);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const pair_t aa = twice(TRANS ? a[TRANS ? u : 0][i] : r[u]);
            fma2(acc[u][0], aa, lo2.x), fma2(acc[u][1], aa, lo2.y), fma2(acc[u][2], aa, hi2.x), fma2(acc[u][3], aa, hi2.y);
          }
        }
      }
    }
  }
  // parts of a sum in PARTS warps: in the first one's accumulators, added in order.  All of them call it.
  template <int PARTS> __device__ __forceinline__ void join(float* smem) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float2* part = reinterpret_cast<float2*>(smem);
    __syncthreads();
    if (w > 0) {
#pragma unroll
      for (int e = 0; e < 4 * U; ++e) {
        float2 v;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(acc[e >> 2][e & 3]));
        part[((w - 1) * 4 * U + e) * 32 + lane] = v;
      }
    }
    __syncthreads();
    if (w > 0) return;
#pragma unroll
    for (int e = 0; e < 4 * U; ++e) {
      float2 v;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(acc[e >> 2][e & 3]));
#pragma unroll
      for (int o = 0; o < PARTS - 1; ++o) {
        const float2 y = part[(o * 4 * U + e) * 32 + lane];
        v.x += y.x;
        v.y += y.y;
      }
      asm("mov.b64 %0, {%1, %2};" : "=l"(acc[e >> 2][e & 3]) : "f"(v.x), "f"(v.y));
    }
  }
  __device__ __forceinline__ void write(int bh, int r0, int n0, float* out, const OperandLayout& lo) {
    float* ob = out + (long long)bh * lo.bh_stride;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int row = r0 + row0 + (TRANS ? 8 * u : u);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = as_float4(acc[u][2 * h], acc[u][2 * h + 1]);
        float* o = ob + (long long)row * lo.sl + (long long)(n0 + 16 * h + 4 * tx) * lo.sd;
        if (lo.sd == 1 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) *reinterpret_cast<float4*>(o) = v;
        else o[0] = v.x, o[lo.sd] = v.y, o[2 * lo.sd] = v.z, o[3 * lo.sd] = v.w;
      }
    }
  }
};

// O = P V.  Its bits are nobody's: four warps take a quarter of the keys each.  16 matrices, L = 1024, d 32: 34 us with one chain of 64 threads a
// tile, 31 with four of them, 28 so; 60 matrices 121, 122, 96.
constexpr int OPARTS = 4;
__global__ void __launch_bounds__(32 * OPARTS) spmm_dense_split(const float* __restrict__ vals, const float* __restrict__ Bop, OperandLayout lb,
                                                                float* __restrict__ out, OperandLayout lo, int L) {
  extern __shared__ __align__(16) float s_spmm[];
  const int w = threadIdx.x >> 5, r0 = blockIdx.x * DT, bh = blockIdx.y, n0 = blockIdx.z * 32;
  const int chunks = L / DK, per = (chunks + OPARTS - 1) / OPARTS, c0 = min(chunks, w * per), c1 = min(chunks, c0 + per);
  Spmm<false, 8, 32> x;
  x.run(s_spmm + w * 2 * SPMM_STAGE, threadIdx.x & 31, 0, bh, r0, n0, c0, c1 - c0, vals, Bop, lb, L);
  x.join<OPARTS>(s_spmm);
  if (w == 0) x.write(bh, r0, n0, out, lo);
}

// dK = dS^T Q, dV = P^T dO and dQ = dS K of a backward in one launch, so that every SM has ten warps or more; dK by two warps of 32 rows each, the others
// by two warps of half of the sum each.  16 matrices, L = 1024, d 32: 107 us in three launches, 94 in one with four by eight outputs a lane,
// 88 so; 60 matrices 376, 333, 314 (4 matrices, L = 512, d 64: 57, 26, 27).
struct DenseGrads {
  const float *P, *dS, *Q, *K, *dO;
  float *dQ, *dK, *dV;
  OperandLayout lo;
  int L, halves;                                       // head_dim / 32
};
__global__ void __launch_bounds__(64) spmm_dense_grads(const DenseGrads a) {
  extern __shared__ __align__(16) float s_spmm[];
  const int what = blockIdx.z / a.halves, n0 = (blockIdx.z - what * a.halves) * 32, r0 = blockIdx.x * DT, bh = blockIdx.y, w = threadIdx.x >> 5;
  const int chunks = a.L / DK, half = chunks / 2;      // L is a multiple of 64
  float* own = s_spmm + w * 2 * SPMM_STAGE;
  const int lane = threadIdx.x & 31;
  if (what == 0) {
    Spmm<true, 4, 64> x;
    x.run(s_spmm, threadIdx.x, 32 * w, bh, r0, n0, 0, chunks, a.dS, a.Q, a.lo, a.L);
    x.write(bh, r0, n0, a.dK, a.lo);
  } else if (what == 1) {
    Spmm<true, 8, 32> x;
    x.run(own, lane, 0, bh, r0, n0, w * half, w ? chunks - half : half, a.P, a.dO, a.lo, a.L);
    x.join<2>(s_spmm);
    if (w == 0) x.write(bh, r0, n0, a.dV, a.lo);
  } else {
    Spmm<false, 8, 32> x;
    x.run(own, lane, 0, bh, r0, n0, w * half, w ? chunks - half : half, a.dS, a.K, a.lo, a.L);
    x.join<2>(s_spmm);
    if (w == 0) x.write(bh, r0, n0, a.dQ, a.lo);
  }
}

// Scores and their softmax (forward), dP and dS (backward) of sixteen query rows and all keys by one CTA: what the product leaves stays in
// registers, so that S and dP never reach memory.  A warp has one of the DENSE_WARPS slices of the keys, a lane KPL keys by eight queries of
// it (packed multiply-adds over pairs of queries: a shared-memory read returns one register per lane and cycle, which eight by eight tiles
// balance with the multiply-adds; four by four took 62 us forward); sums along the keys go through shared memory, one lane per query and
// slice.  Slices, expressions and order of additions are those of sddmm_dense_kernel and the slab kernels: the results are the same bits.
// Up to 2048 keys (8 KPL accumulators for slices of 16 KPL).
// Which calls take them and what that gives: simt_dense_joint.
// keys kg + 16 r, queries 4 ig + (0 .. 3) and 8 + 4 ig + (0 .. 3), in pairs
template <int KPL>
struct Slice {
  pair_t acc[KPL][4];
  __device__ __forceinline__ float4 at(int r, int h) const { return as_float4(acc[r][2 * h], acc[r][2 * h + 1]); }
};
// Products of the keys B[0 .. n) of a slice with As [d][16], eight columns of B at a time (NB buffers).
template <int KPL, int NB, class BEFORE>
__device__ __forceinline__ void slice_products(Slice<KPL>& x, const float* __restrict__ B, int ld, int n, int d, const float* As, float* stage, BEFORE before) {
  const int lane = threadIdx.x & 31, kg = lane >> 1, ig = lane & 1;
#pragma unroll
  for (int r = 0; r < KPL; ++r)
#pragma unroll
    for (int y = 0; y < 4; ++y) x.acc[r][y] = 0ull;
  auto load = [&](int n0, float* to) {
#pragma unroll
    for (int e = 0; e < KPL; ++e) {
      const int row = e * 16 + (lane >> 1), q = lane & 1;
      if (row < n) dense_cp16(to + row * 8 + 4 * q, B + (long long)row * ld + n0 + 4 * q);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0, stage);
  before();                                            // copies of the caller's, one group
  for (int n0 = 0; n0 < d; n0 += 8) {
    const float* st = stage;
    if (NB == 2) {
      if (n0 + 8 < d) load(n0 + 8, stage + ((n0 >> 3) + 1 & 1) * 128 * KPL);
      else asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      st += ((n0 >> 3) & 1) * 128 * KPL;
    } else if (n0 == 0) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      load(n0, stage);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      float2 b[KPL];
#pragma unroll
      for (int r = 0; r < KPL; ++r) b[r] = *reinterpret_cast<const float2*>(st + (kg + 16 * r) * 8 + k);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float* a = As + (n0 + k + u) * 16 + 4 * ig;
        const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(a), hi = *reinterpret_cast<const ulonglong2*>(a + 8);
#pragma unroll
        for (int r = 0; r < KPL; ++r) {
          const pair_t bb = twice(u ? b[r].y : b[r].x);
          fma2(x.acc[r][0], lo.x, bb); fma2(x.acc[r][1], lo.y, bb); fma2(x.acc[r][2], hi.x, bb); fma2(x.acc[r][3], hi.y, bb);
        }
      }
    }
    __syncwarp();                                      // the buffer may be filled again
  }
}
__device__ __forceinline__ void load_queries(float* As, const float* A, const OperandLayout& la, int bh, int i0, int d) {     // As [d][16]
  const float* src = A + (long long)bh * la.bh_stride + (long long)i0 * la.sl;
  for (int e = threadIdx.x; e < 16 * d; e += DENSE_WARPS * 32) {
    const int i = la.sl == 1 ? e & 15 : e / d, n = la.sl == 1 ? e >> 4 : e % d;
    As[n * 16 + i] = src[(long long)i * la.sl + (long long)n * la.sd];
  }
}
__device__ __forceinline__ float4 operator+(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
constexpr int SLICE_MAX_L = 2048;

template <int KPL>
__global__ void __launch_bounds__(DENSE_WARPS * 32, KPL <= 8 ? 2 : 1) dense_scores_kernel(const float* __restrict__ Q, OperandLayout lq, const float* __restrict__ K,
                                                                                     float* __restrict__ P, int L, int d, float scale,
                                                                                     const float* __restrict__ keypad, float floor_v) {
  extern __shared__ __align__(16) float s_dyn[];
  __shared__ __align__(16) float As[64 * 16];
  __shared__ __align__(16) float s_red[2][DENSE_WARPS][SLAB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, kg = lane >> 1, ig = lane & 1;
  const int bh = blockIdx.y, i0 = blockIdx.x * SLAB;
  const int per = slab_per(L), j0 = w * per, n = max(0, min(L, j0 + per) - j0);
  float* mine = s_dyn + w * 256 * KPL;                 // two operand stages, then the slice's exponentials [key][16]
  load_queries(As, Q, lq, bh, i0, d);
  __syncthreads();
  Slice<KPL> x;
  slice_products<KPL, 2>(x, K + ((long long)bh * L + j0) * d, d, n, d, As, mine, [] {});
  const float* kp = keypad ? keypad + (long long)bh * L + j0 : nullptr;
  // s scale - penalty, each rounded once together, and, without penalties, the maximum taken off in the same step: as the compiler contracts
  // the expressions of the kernels above
  float4 m[2] = {make_float4(floor_v, floor_v, floor_v, floor_v), make_float4(floor_v, floor_v, floor_v, floor_v)};
#pragma unroll
  for (int r = 0; r < KPL; ++r) {
    const int j = kg + 16 * r;
    if (j >= n) continue;
    const float k = kp ? kp[j] : 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 s = x.at(r, h);
      m[h].x = fmaxf(m[h].x, fmaf(s.x, scale, -k)); m[h].y = fmaxf(m[h].y, fmaf(s.y, scale, -k));
      m[h].z = fmaxf(m[h].z, fmaf(s.z, scale, -k)); m[h].w = fmaxf(m[h].w, fmaf(s.w, scale, -k));
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int o = 2; o < 32; o <<= 1) {
      m[h].x = fmaxf(m[h].x, __shfl_xor_sync(0xffffffffu, m[h].x, o)); m[h].y = fmaxf(m[h].y, __shfl_xor_sync(0xffffffffu, m[h].y, o));
      m[h].z = fmaxf(m[h].z, __shfl_xor_sync(0xffffffffu, m[h].z, o)); m[h].w = fmaxf(m[h].w, __shfl_xor_sync(0xffffffffu, m[h].w, o));
    }
  if (kg == 0) {
    *reinterpret_cast<float4*>(&s_red[0][w][4 * ig]) = m[0];
    *reinterpret_cast<float4*>(&s_red[0][w][8 + 4 * ig]) = m[1];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < DENSE_WARPS; ++k)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 o = *reinterpret_cast<const float4*>(&s_red[0][k][8 * h + 4 * ig]);
      m[h].x = fmaxf(m[h].x, o.x); m[h].y = fmaxf(m[h].y, o.y); m[h].z = fmaxf(m[h].z, o.z); m[h].w = fmaxf(m[h].w, o.w);
    }
#pragma unroll
  for (int r = 0; r < KPL; ++r) {
    const int j = kg + 16 * r;
    if (j >= n) continue;
    const float k = kp ? kp[j] : 0.f;
    auto ex = [&](float s, float most) { return expf(kp ? __fsub_rn(fmaf(s, scale, -k), most) : fmaf(s, scale, -most)); };
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 s = x.at(r, h), e = make_float4(ex(s.x, m[h].x), ex(s.y, m[h].y), ex(s.z, m[h].z), ex(s.w, m[h].w));
      *reinterpret_cast<float4*>(mine + j * SLAB + 8 * h + 4 * ig) = e;
      asm("mov.b64 %0, {%1, %2};" : "=l"(x.acc[r][2 * h]) : "f"(e.x), "f"(e.y));
      asm("mov.b64 %0, {%1, %2};" : "=l"(x.acc[r][2 * h + 1]) : "f"(e.z), "f"(e.w));
    }
  }
  __syncwarp();
  if (lane < SLAB) {
    float sum = 0.f;
#pragma unroll 8
    for (int u = 0; u < n; ++u) sum += mine[u * SLAB + lane];
    s_red[1][w][lane] = sum;
  }
  __syncthreads();
  float* out = P + (long long)bh * L * L + (long long)j0 * L + i0 + 4 * ig;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < DENSE_WARPS; ++k) t = t + *reinterpret_cast<const float4*>(&s_red[1][k][8 * h + 4 * ig]);      // slices added in slice order
    const float4 inv = make_float4(1.0f / t.x, 1.0f / t.y, 1.0f / t.z, 1.0f / t.w);
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int j = kg + 16 * r;
      const float4 e = x.at(r, h);
      if (j < n) *reinterpret_cast<float4*>(out + (long long)j * L + 8 * h) = make_float4(e.x * inv.x, e.y * inv.y, e.z * inv.z, e.w * inv.w);
    }
  }
}

template <int KPL>
__global__ void __launch_bounds__(DENSE_WARPS * 32, KPL <= 8 ? 2 : 1) dense_dscores_kernel(const float* __restrict__ dO, OperandLayout ldo, const float* __restrict__ V,
                                                                                      const float* __restrict__ P, float* __restrict__ dS, int L, int d,
                                                                                      float scale) {
  extern __shared__ __align__(16) float s_dyn[];
  __shared__ __align__(16) float As[64 * 16];
  __shared__ __align__(16) float s_red[DENSE_WARPS][SLAB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, kg = lane >> 1, ig = lane & 1;
  const int bh = blockIdx.y, i0 = blockIdx.x * SLAB;
  const int per = slab_per(L), j0 = w * per, n = max(0, min(L, j0 + per) - j0);
  float* mine = s_dyn + w * (per * SLAB + 128 * KPL);  // P of the slice [key][16], then a stage
  float* stage = mine + per * SLAB;
  const long long at = (long long)bh * L * L + (long long)j0 * L + i0;
  load_queries(As, dO, ldo, bh, i0, d);
  __syncthreads();
  Slice<KPL> x;
  slice_products<KPL, 1>(x, V + ((long long)bh * L + j0) * d, d, n, d, As, stage, [&] {
    for (int e = lane; e < 4 * n; e += 32) dense_cp16(mine + e * 4, P + at + (long long)(e >> 2) * L + 4 * (e & 3));
    asm volatile("cp.async.commit_group;" ::: "memory");
  });
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < KPL / 2; ++c) {                  // 32 keys of dP at a time through the stage
    if (c * 32 >= n) break;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) *reinterpret_cast<float4*>(stage + (kg + 16 * u) * SLAB + 8 * h + 4 * ig) = x.at(2 * c + u, h);
    __syncwarp();
    if (lane < SLAB) {
      const float* p = mine + c * 32 * SLAB + lane;
      const int most = min(32, n - c * 32);
#pragma unroll 8
      for (int u = 0; u < most; ++u) s += stage[u * SLAB + lane] * p[u * SLAB];
    }
    __syncwarp();
  }
  if (lane < SLAB) s_red[w][lane] = s;
  __syncthreads();
  float* out = dS + at + 4 * ig;
  auto ds = [&](float dp, float pv, float sum) { return (dp * pv - pv * sum) * scale; };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < DENSE_WARPS; ++k) t = t + *reinterpret_cast<const float4*>(&s_red[k][8 * h + 4 * ig]);
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int j = kg + 16 * r;
      if (j >= n) continue;
      const float4 g = x.at(r, h), p = *reinterpret_cast<const float4*>(mine + j * SLAB + 8 * h + 4 * ig);
      *reinterpret_cast<float4*>(out + (long long)j * L + 8 * h) = make_float4(ds(g.x, p.x, t.x), ds(g.y, p.y, t.y), ds(g.z, p.z, t.z), ds(g.w, p.w, t.w));
    }
  }
}

// Only the dense context stores values this way, and its mask is always full; blocks of 64 stand for L being a multiple of 64.
bool full_dense(const ValueLayout& vl, const Pattern& p, const void* vals) {
  return vl.mode == VAL_DENSE_T && p.bs == DT && (reinterpret_cast<uintptr_t>(vals) & 15) == 0;
}

}  // namespace

// ================================================================================ launchers
template <typename TI, typename TV>
static int sddmm_dispatch(const void* A, OperandLayout la, const void* B, OperandLayout lb, void* vals, ValueLayout vl,
                          Pattern p, int nnzb, int BH, int d, cudaStream_t st) {
  dim3 grid(nnzb, BH);
  if (p.bs == 64)
    sddmm_kernel<TI, TV, 4><<<grid, 256, 0, st>>>((const TI*)A, la, (const TI*)B, lb, (TV*)vals, vl, p, d);
  else if (p.bs == 32)
    sddmm_kernel<TI, TV, 2><<<grid, 256, 0, st>>>((const TI*)A, la, (const TI*)B, lb, (TV*)vals, vl, p, d);
  else
    return SPION_ERR_UNSUPPORTED;
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

int simt_sddmm(int dtype_in, int dtype_val, const void* A, OperandLayout la, const void* B, OperandLayout lb, void* vals,
               ValueLayout vl, Pattern p, int nnzb, int BH, int d, cudaStream_t st) {
  if (d % KC != 0 || BH > 65535) return SPION_ERR_UNSUPPORTED;
  if (nnzb == 0) return SPION_OK;
  if (dtype_in == SPION_F32 && dtype_val == SPION_F32 && full_dense(vl, p, vals)) {
    sddmm_dense_kernel<<<dim3(p.nb, p.nb, BH), 64, 0, st>>>((const float*)A, la, (const float*)B, lb, (float*)vals, vl.L, d);
    SPION_LAUNCH_CHECK();
    return SPION_OK;
  }
  if (dtype_in == SPION_F32 && dtype_val == SPION_F32)
    return sddmm_dispatch<float, float>(A, la, B, lb, vals, vl, p, nnzb, BH, d, st);
  if (dtype_in == SPION_BF16 && dtype_val == SPION_F32)
    return sddmm_dispatch<__nv_bfloat16, float>(A, la, B, lb, vals, vl, p, nnzb, BH, d, st);
  return SPION_ERR_UNSUPPORTED;
}

template <typename TV, typename TO>
static int spmm_dispatch(bool trans, const void* vals, ValueLayout vl, const void* Bop, OperandLayout lb, void* out,
                         OperandLayout lo, Pattern p, int BH, int d, cudaStream_t st) {
  dim3 grid(p.nb, BH, d / 32);
#define SPION_SPMM(TMv, TR) \
  spmm_kernel<TV, TO, TMv, TR><<<grid, 256, 0, st>>>((const TV*)vals, vl, (const TO*)Bop, lb, (TO*)out, lo, p)
  if (p.bs == 64) { if (trans) SPION_SPMM(4, true); else SPION_SPMM(4, false); }
  else if (p.bs == 32) { if (trans) SPION_SPMM(2, true); else SPION_SPMM(2, false); }
  else return SPION_ERR_UNSUPPORTED;
#undef SPION_SPMM
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

int simt_spmm(int dtype_val, int dtype_op, bool trans, const void* vals, ValueLayout vl, const void* Bop,
              OperandLayout lb, void* out, OperandLayout lo, Pattern p, int BH, int d, cudaStream_t st) {
  if (d % 32 != 0 || BH > 65535) return SPION_ERR_UNSUPPORTED;
  if (!trans && dtype_val == SPION_F32 && dtype_op == SPION_F32 && full_dense(vl, p, vals)) {       // trans: simt_dense_grads
    constexpr int smem = OPARTS * 2 * SPMM_STAGE * (int)sizeof(float);
    SPION_CUDA_TRY(cudaFuncSetAttribute(spmm_dense_split, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    spmm_dense_split<<<dim3(p.nb, BH, d / 32), 32 * OPARTS, smem, st>>>((const float*)vals, (const float*)Bop, lb, (float*)out, lo, vl.L);
    SPION_LAUNCH_CHECK();
    return SPION_OK;
  }
  if (dtype_val == SPION_F32 && dtype_op == SPION_F32)
    return spmm_dispatch<float, float>(trans, vals, vl, Bop, lb, out, lo, p, BH, d, st);
  if (dtype_val == SPION_BF16 && dtype_op == SPION_BF16)
    return spmm_dispatch<__nv_bfloat16, __nv_bfloat16>(trans, vals, vl, Bop, lb, out, lo, p, BH, d, st);
  return SPION_ERR_UNSUPPORTED;
}

static bool aligned_to(const void* ptr, size_t n) { return ((uintptr_t)ptr & (n - 1)) == 0; }
static bool piece_layout(const ValueLayout& vl) { return vl.mode != VAL_DENSE_T && vl.bh_stride % 4 == 0; }

template <int BS>
static void softmax_fwd_rows16_launch(int dtype_out, const float* S, ValueLayout vin, void* P, ValueLayout vout, Pattern p,
                                      int BH, int L, float scale, const float* keypad, float floor_v, cudaStream_t st) {
  const unsigned grid = (unsigned)BH * (unsigned)(L / 16);
  if (dtype_out == SPION_F32)
    softmax_fwd_rows16_kernel<float, BS><<<grid, 256, 0, st>>>(S, vin, (float*)P, vout, p, BH, L, scale, keypad,
                                                               floor_v);
  else
    softmax_fwd_rows16_kernel<__nv_bfloat16, BS><<<grid, 256, 0, st>>>(S, vin, (__nv_bfloat16*)P, vout, p, BH, L,
                                                                       scale, keypad, floor_v);
}

int softmax_fwd_rows(int dtype_out, const float* S, ValueLayout vin, void* P, ValueLayout vout, Pattern p, int BH, int L,
                     float scale, const float* keypad, float floor_v, cudaStream_t st) {
  const long long rows = (long long)BH * L;
  const bool pieces = (p.bs == 32 || p.bs == 64) && piece_layout(vin) && piece_layout(vout) && aligned_to(S, 16) &&
                      aligned_to(P, dtype_out == SPION_F32 ? 16 : 8) && (!keypad || aligned_to(keypad, 16));
  if (pieces && p.bs == 64) {
    softmax_fwd_rows16_launch<64>(dtype_out, S, vin, P, vout, p, BH, L, scale, keypad, floor_v, st);
  } else if (pieces) {
    softmax_fwd_rows16_launch<32>(dtype_out, S, vin, P, vout, p, BH, L, scale, keypad, floor_v, st);
  } else {
    const unsigned grid = (unsigned)((rows + 7) / 8);
    if (dtype_out == SPION_F32)
      softmax_fwd_rows_kernel<float><<<grid, 256, 0, st>>>(S, vin, (float*)P, vout, p, BH, L, scale, keypad, floor_v);
    else
      softmax_fwd_rows_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(S, vin, (__nv_bfloat16*)P, vout, p, BH, L, scale,
                                                                   keypad, floor_v);
  }
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

template <int BS>
static void softmax_bwd_rows16_launch(int dtype_p, const float* dP, ValueLayout vdp, const void* P, ValueLayout vp,
                                      void* dS, ValueLayout vds, Pattern p, int BH, int L, float scale, cudaStream_t st) {
  const unsigned grid = (unsigned)BH * (unsigned)(L / 16);
  if (dtype_p == SPION_F32)
    softmax_bwd_rows16_kernel<float, BS><<<grid, 256, 0, st>>>(dP, vdp, (const float*)P, vp, (float*)dS, vds, p, BH, L,
                                                               scale);
  else
    softmax_bwd_rows16_kernel<__nv_bfloat16, BS><<<grid, 256, 0, st>>>(dP, vdp, (const __nv_bfloat16*)P, vp,
                                                                       (__nv_bfloat16*)dS, vds, p, BH, L, scale);
}

int softmax_bwd_rows(int dtype_p, const float* dP, ValueLayout vdp, const void* P, ValueLayout vp, void* dS,
                     ValueLayout vds, Pattern p, int BH, int L, float scale, cudaStream_t st) {
  const long long rows = (long long)BH * L;
  const size_t pal = dtype_p == SPION_F32 ? 16 : 8;
  const bool pieces = (p.bs == 32 || p.bs == 64) && piece_layout(vdp) && piece_layout(vp) && piece_layout(vds) &&
                      aligned_to(dP, 16) && aligned_to(P, pal) && aligned_to(dS, pal);
  if (pieces && p.bs == 64) {
    softmax_bwd_rows16_launch<64>(dtype_p, dP, vdp, P, vp, dS, vds, p, BH, L, scale, st);
  } else if (pieces) {
    softmax_bwd_rows16_launch<32>(dtype_p, dP, vdp, P, vp, dS, vds, p, BH, L, scale, st);
  } else {
    const unsigned grid = (unsigned)((rows + 7) / 8);
    if (dtype_p == SPION_F32)
      softmax_bwd_rows_kernel<float><<<grid, 256, 0, st>>>(dP, vdp, (const float*)P, vp, (float*)dS, vds, p, BH, L,
                                                           scale);
    else
      softmax_bwd_rows_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(dP, vdp, (const __nv_bfloat16*)P, vp,
                                                                   (__nv_bfloat16*)dS, vds, p, BH, L, scale);
  }
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

constexpr int SLAB_SMEM = 112 * 1024;
int softmax_fwd_dense_t(float* S, int BH, int L, float scale, const float* keypad, float floor_v, cudaStream_t st) {
  if (BH > 65535) return SPION_ERR_UNSUPPORTED;
  // the slab kernel while at least two CTAs of it fit an SM
  const int smem = DENSE_WARPS * slab_slice(L) * (int)sizeof(float);
  if (L % SLAB == 0 && ((uintptr_t)S & 15) == 0 && smem <= SLAB_SMEM) {
    SPION_CUDA_TRY(cudaFuncSetAttribute(softmax_fwd_dense_t_slab, cudaFuncAttributeMaxDynamicSharedMemorySize, SLAB_SMEM));
    softmax_fwd_dense_t_slab<<<dim3(L / SLAB, BH), DENSE_WARPS * SLAB, smem, st>>>(S, L, scale, keypad, floor_v);
  } else {
    softmax_fwd_dense_t_kernel<<<dim3((L + 31) / 32, BH), DENSE_WARPS * 32, 0, st>>>(S, L, scale, keypad, floor_v);
  }
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

int softmax_bwd_dense_t(const float* dP, const float* P, float* dS, int BH, int L, float scale, cudaStream_t st) {
  if (BH > 65535) return SPION_ERR_UNSUPPORTED;
  // the slab kernel while a slice of dP fits a thread's registers
  const int smem = DENSE_WARPS * slab_slice(L) * (int)sizeof(float), per = slab_per(L);
  auto slab = [&](auto kernel) -> int {
    SPION_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SLAB_SMEM));
    kernel<<<dim3(L / SLAB, BH), DENSE_WARPS * SLAB, smem, st>>>(dP, P, dS, L, scale);
    return SPION_OK;
  };
  int rc = SPION_OK;
  if (L % SLAB == 0 && ((uintptr_t)P & 15) == 0 && per <= 128) rc = per <= 64 ? slab(softmax_bwd_dense_t_slab<64>) : slab(softmax_bwd_dense_t_slab<128>);
  else softmax_bwd_dense_t_kernel<<<dim3((L + 31) / 32, BH), DENSE_WARPS * 32, 0, st>>>(dP, P, dS, L, scale);
  if (rc) return rc;
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

// ------------------------------------------------------------------------------ dense phase, several stages per launch
template <class F>
static int with_slices(int L, F f) {
  const int keys = (slab_per(L) + 15) / 16;            // of a lane; an even number, four at least
  switch (keys <= 4 ? 4 : (keys + 1) & ~1) {
    case 4: return f(std::integral_constant<int, 4>());
    case 6: return f(std::integral_constant<int, 6>());
    case 8: return f(std::integral_constant<int, 8>());
    case 10: return f(std::integral_constant<int, 10>());
    case 12: return f(std::integral_constant<int, 12>());
    case 14: return f(std::integral_constant<int, 14>());
    default: return f(std::integral_constant<int, 16>());
  }
}
// 64-wide tiles in the S^T layout, operand rows of K (V) and values that are read in 16-byte pieces, up to SLICE_MAX_L keys.
// Measured, us in two launches and in one (matrices x L, d): backward 4 x 1024, 32 24, 20; 8 x 1024, 64 58, 51; 12 x 1024, 32 74, 52; 8 x 1472, 32 136,
// 78; 20 x 512, 32 23.5, 23.3; 4 x 512, 64 14, 9; 96 x 256, 32 34, 36; 64 x 256, 64 31, 35: from 512 keys on, and where one wave of CTAs holds all.
// Forward 4 x 512, 64 12, 9; 4 x 1024, 32 20, 20; 8 x 1024, 64 46, 52; 60 x 1024, 32 212, 228; 1 x 2048, 64 131, 31 (rows that the slab kernel does not
// take): one wave or such rows, else S is faster with a kernel of its own (sixteen warps per SM hide the latencies of all stages at once badly).
bool simt_dense_joint(bool backward, int L, int d, int BH, const void* rows, const void* values, const void* values2) {
  if (L % DT != 0 || L > SLICE_MAX_L || d % KC != 0 || d > 64 || BH > 65535 || !aligned_to(rows, 16) || !aligned_to(values, 16) || !aligned_to(values2, 16))
    return false;
  const bool one_wave = (long long)BH * (L / SLAB) <= 2LL * sm_count();
  return one_wave || (backward ? L >= 512 : DENSE_WARPS * slab_slice(L) * (int)sizeof(float) > SLAB_SMEM);
}
int simt_dense_scores(const float* Q, OperandLayout lq, const float* K, float* P, int BH, int L, int d, float scale, const float* keypad, float floor_v, cudaStream_t st) {
  const int rc = with_slices(L, [&](auto kpl) -> int {
    constexpr int KPL = decltype(kpl)::value, smem = DENSE_WARPS * 256 * KPL * (int)sizeof(float);
    auto k = dense_scores_kernel<KPL>;
    SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k<<<dim3(L / SLAB, BH), DENSE_WARPS * 32, smem, st>>>(Q, lq, K, P, L, d, scale, keypad, floor_v);
    return SPION_OK;
  });
  if (rc) return rc;
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}
int simt_dense_dscores(const float* dO, OperandLayout ldo, const float* V, const float* P, float* dS, int BH, int L, int d, float scale, cudaStream_t st) {
  const int rc = with_slices(L, [&](auto kpl) -> int {
    constexpr int KPL = decltype(kpl)::value;
    const int smem = DENSE_WARPS * (slab_per(L) * SLAB + 128 * KPL) * (int)sizeof(float);
    auto k = dense_dscores_kernel<KPL>;
    SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k<<<dim3(L / SLAB, BH), DENSE_WARPS * 32, smem, st>>>(dO, ldo, V, P, dS, L, d, scale);
    return SPION_OK;
  });
  if (rc) return rc;
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}
// whole tiles of 64 x 64 values (any L): all three products of the backward.  SPION_ERR_UNSUPPORTED: one by one (simt_spmm)
int simt_dense_grads(const float* P, const float* dS, const float* Q, const float* K, const float* dO, OperandLayout lo, float* dQ, float* dK, float* dV,
                     Pattern p, int BH, int L, int d, cudaStream_t st) {
  const ValueLayout vl{VAL_DENSE_T, L, (long long)L * L};
  if (d % 32 != 0 || BH > 65535 || !full_dense(vl, p, P) || !full_dense(vl, p, dS)) return SPION_ERR_UNSUPPORTED;
  constexpr int smem = 2 * 2 * SPMM_STAGE * (int)sizeof(float);
  spmm_dense_grads<<<dim3(p.nb, BH, 3 * (d / 32)), 64, smem, st>>>(DenseGrads{P, dS, Q, K, dO, dQ, dK, dV, lo, L, d / 32});
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}
