// The mean attention map of the warm-up phase without a stored P (sm_100a, bf16, 64x64 blocks): rebuilt from Q, K and the
// forward's log-sum-exp, lse2_i = m_i log2(e) + log2(Z_i), where Z_i includes the reference's term for the non-selected keys
// (models/block_attn.cu:65-71):
//     P_ij = exp2(s_ij scale log2(e) - pad_j log2(e) - lse2_i)                      (:72-87)
// The backward from the same quantities is in tc_bwd_stream.cu.
#include <cuda.h>

#include "common.cuh"
#include "tc_tiles.cuh"

using namespace tc;

#ifdef SPION_TRACE
SPION_TRACE_SETTER(spion_debug_trace_rc)
#endif

namespace {

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr size_t MM_SMEM(int tile_bytes) { return 1024 + (size_t)2 * 2 * 2 * tile_bytes + 128; }

// =====================================================================================
// Head / batch mean of the attention probabilities without a stored P (models/model_transformer.py:137):
//     A[i, j] = (1 / BH) sum_bh exp2(s_ij(bh) scale log2(e) - pad_j log2(e) - lse2_i(bh))   on the selected blocks.
// One CTA per selected block (r, c); the (b,h) matrices are taken two at a time (first in lanes 0-15 of
// every TMEM quadrant, second in lanes 16-31) through two stages: while the probabilities of one pair are
// summed in registers, the S tiles of the next pair are already being computed and the tiles of the pair
// after that are on their way.  Every thread keeps the 64 running sums of its row.
// The log-sum-exp and the penalties of a pair (one key per thread, handed round through shared memory) are requested when the pair before
// has been summed, ahead of the barrier that ends it: the log-sum-exp has the wait for S to arrive, a penalty is waited for as soon as the
// pair begins.  Asked for where they were used, two loads in a row were most of a pair's time, and a block with padded keys took 64 more
// per thread.  18 matrices, L = 1984, d 32, padded keys: 46 -> 40 us.
template <int D, bool SUB>
__global__ void __launch_bounds__(128) k_mean_map_rc(const __grid_constant__ CUtensorMap tmQ,
                                                     const __grid_constant__ CUtensorMap tmK,
                                                     const float* __restrict__ lse_in, const float* __restrict__ keypad,
                                                     float* __restrict__ A, const int* __restrict__ blk_row,
                                                     const int* __restrict__ col_idx, const uint8_t* __restrict__ submask,
                                                     int L, int BH, int heads, float scale, int* status) {
  using T = OpTile<D>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  // stage st: Q tiles of the pair at sbase + st*4*T + {0, T}, K tiles at + {2T, 3T}
  const uint32_t bars = sbase + 8 * T::BYTES;
  const uint32_t bar_full = bars, bar_s = bars + 16, slot = bars + 32;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - raw));
  __shared__ int s_abort;
  __shared__ __align__(16) float s_pen[2][128];                  // per parity of the pair: penalties of the block's keys in both matrices
  __shared__ int s_any[2][4];                                    // ... and, per 32 of them, whether any is not zero

  const int tid = threadIdx.x, q = warp_uniform(tid >> 5), lane = tid & 31;
  const int hf = lane >> 4, row = q * 16 + (lane & 15);
  const int blk = blockIdx.x;
  const int r = blk_row[blk], c = col_idx[blk];
  const int npair = (BH + 1) >> 1;

  auto issue = [&](int it) {                                     // warp 0, all lanes
    const int st = it & 1;
    const int cnt = min(2, BH - 2 * it);
    const uint32_t base = sbase + st * 4 * T::BYTES;
    if (lane == 0) mbar_expect_tx(bar_full + 8 * st, cnt * 2 * T::BYTES);
    __syncwarp();
    if (lane < 2 * cnt) {
      const int hb = lane >> 1;
      const OpPos pos = op_pos(2 * it + hb, L, heads, D);
      if (lane & 1) tma_load_2d(base + (2 + hb) * T::BYTES, &tmK, bar_full + 8 * st, pos.x0, pos.row0 + c * BS);
      else tma_load_2d(base + hb * T::BYTES, &tmQ, bar_full + 8 * st, pos.x0, pos.row0 + r * BS);
    }
  };

  if (q == 0) {
    if (lane == 0) {
      s_abort = *reinterpret_cast<volatile int*>(status);
      for (int i = 0; i < 4; ++i) mbar_init(bar_full + 8 * i, 1);     // bar_full[2], bar_s[2]
      fence_barrier_init();
    }
    __syncwarp();
    if (s_abort == 0) {
      issue(0);
      if (npair > 1) issue(1);
    }
  }
  __syncthreads();
  if (s_abort != 0) return;
  if (q == 0) {
    tmem_alloc(slot, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16);
  constexpr uint32_t IDESC_S = make_idesc_bf16(64, 64, 0, 0);
  const float sc2 = scale * LOG2E;
  bool ok = true;

  // warp 0: S tiles of pair `it` into columns 64 (it & 1)
  auto issue_s = [&](int it) -> bool {
    const int st = it & 1;
    const int cnt = min(2, BH - 2 * it);
    if (!warp_wait(bar_full + 8 * st, (uint32_t)(it >> 1) & 1u, status, ERR_LOAD_WAIT)) return false;
    if (elect_one()) {
      tc_fence_after();
      const uint64_t base = T::kmajor(sbase + st * 4 * T::BYTES, 0);
      for (int hb = 0; hb < cnt; ++hb) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_bf16(tmem + ((uint32_t)(hb * 16) << 16) + (uint32_t)st * 64u, desc_advance(base, hb * T::BYTES + kk * T::K_STEP),
                   desc_advance(base, (2 + hb) * T::BYTES + kk * T::K_STEP), IDESC_S, kk > 0);
      }
      mma_commit(bar_s + 8 * st);
    }
    __syncwarp();
    return true;
  };

  float acc[64];
#pragma unroll
  for (int j = 0; j < 64; ++j) acc[j] = 0.f;
  const bool live0 = !SUB || ((submask[blk] >> ((q >> 1) * 2 + 0)) & 1);
  const bool live1 = !SUB || ((submask[blk] >> ((q >> 1) * 2 + 1)) & 1);

  float lse = 0.f, pen = 0.f;                                    // of the next pair, as they were loaded
  auto request = [&](int it) {                                   // (a matrix past the end: the last one's, not used)
    lse = lse_in[(size_t)min(2 * it + hf, BH - 1) * L + r * BS + row];
    if (keypad) pen = keypad[(size_t)min(2 * it + (tid >> 6), BH - 1) * L + c * BS + (tid & 63)];
  };
  request(0);
  if (q == 0) issue_s(0);
  for (int it = 0; it < npair && ok; ++it) {
    const int st = it & 1;
    if (keypad) {                                                // read before the last barrier of pair it - 1 by all that read pair it - 2
      s_pen[st][tid] = pen;
      const int any = __any_sync(0xffffffffu, pen != 0.f);
      if (lane == 0) s_any[st][q] = any;
    }
    if (q == 0 && it + 1 < npair) issue_s(it + 1);
    if (!__syncthreads_and(mbar_wait(bar_s + 8 * st, (uint32_t)(it >> 1) & 1u))) {
      if (tid == 0) report(status, ERR_MMA_WAIT);
      ok = false;
      break;
    }
    tc_fence_after();
    if (q == 0 && it + 2 < npair) issue(it + 2);                  // the MMAs have consumed this stage's tiles
    const int bh = 2 * it + hf;
    const bool mine = bh < BH;
    const bool padded = keypad && (s_any[st][2 * hf] | s_any[st][2 * hf + 1]);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t v[32];
      tmem_ld32(t_lane + (uint32_t)st * 64u + half * 32, v);
      tmem_ld_wait();
      if (mine && (half ? live1 : live0)) {
        if (padded) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(&s_pen[st][hf * 64 + half * 32 + j]);
            acc[half * 32 + j] += ex2f(fmaf(__uint_as_float(v[j]), sc2, -fmaf(k4.x, LOG2E, lse)));
            acc[half * 32 + j + 1] += ex2f(fmaf(__uint_as_float(v[j + 1]), sc2, -fmaf(k4.y, LOG2E, lse)));
            acc[half * 32 + j + 2] += ex2f(fmaf(__uint_as_float(v[j + 2]), sc2, -fmaf(k4.z, LOG2E, lse)));
            acc[half * 32 + j + 3] += ex2f(fmaf(__uint_as_float(v[j + 3]), sc2, -fmaf(k4.w, LOG2E, lse)));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[half * 32 + j] += ex2f(fmaf(__uint_as_float(v[j]), sc2, -lse));
        }
      }
    }
    if (it + 1 < npair) request(it + 1);
    tc_fence_before();
    __syncthreads();                                               // pair it + 2 overwrites these columns
    tc_fence_after();
  }
  if (ok) {
    const float inv = 1.0f / (float)BH;
    float* dst = A + (size_t)(r * BS + row) * L + c * BS;
#pragma unroll
    for (int j = 0; j < 64; j += 4) {
      float4 o;
      o.x = (acc[j] + __shfl_xor_sync(0xffffffffu, acc[j], 16)) * inv;
      o.y = (acc[j + 1] + __shfl_xor_sync(0xffffffffu, acc[j + 1], 16)) * inv;
      o.z = (acc[j + 2] + __shfl_xor_sync(0xffffffffu, acc[j + 2], 16)) * inv;
      o.w = (acc[j + 3] + __shfl_xor_sync(0xffffffffu, acc[j + 3], 16)) * inv;
      if (hf == 0) *reinterpret_cast<float4*>(dst + j) = o;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (q == 0) tmem_dealloc(tmem, 128);
}

}  // namespace

namespace tc {

template <int D>
static int rc_attrs() {
  SPION_CUDA_TRY(cudaFuncSetAttribute(k_mean_map_rc<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MM_SMEM(OpTile<D>::BYTES)));
  SPION_CUDA_TRY(cudaFuncSetAttribute(k_mean_map_rc<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MM_SMEM(OpTile<D>::BYTES)));
  return SPION_OK;
}

int mean_map_set_attrs(int d) { return d == 64 ? rc_attrs<64>() : rc_attrs<32>(); }

template <int D>
static int rc_mean_map(spion_ctx* c, TcState* s, const void* Q, const void* K, const float* lse, const float* keypad,
                       float* A) {
  const TcView vw = tc_view(c, s);
  CUtensorMap mq, mk;
  int rc;
  if ((rc = make_operand_map(c, s, &mq, Q, D)) || (rc = make_operand_map(c, s, &mk, K, D))) return rc;
  if (c->nnzb != c->nb * c->nb)                                   // the full mask writes every element
    SPION_CUDA_TRY(cudaMemsetAsync(A, 0, (size_t)c->L * c->L * sizeof(float), c->stream));
  const int32_t* blk_row = s->super ? s->blk_row64 : c->blk_row;
  if (vw.submask)
    k_mean_map_rc<D, true><<<vw.nnzb, 128, MM_SMEM(OpTile<D>::BYTES), c->stream>>>(
        mq, mk, lse, keypad, A, blk_row, vw.col_idx, vw.submask, c->L, c->BH, c->heads, c->scale, c->status_dev);
  else
    k_mean_map_rc<D, false><<<vw.nnzb, 128, MM_SMEM(OpTile<D>::BYTES), c->stream>>>(
        mq, mk, lse, keypad, A, blk_row, vw.col_idx, vw.submask, c->L, c->BH, c->heads, c->scale, c->status_dev);
  SPION_LAUNCH_CHECK();
  c->launches += 1;
  return SPION_OK;
}

int recompute_mean_map(spion_ctx* c, TcState* s, const void* Q, const void* K, const float* lse, const float* keypad,
                       float* A) {
  return c->d == 64 ? rc_mean_map<64>(c, s, Q, K, lse, keypad, A) : rc_mean_map<32>(c, s, Q, K, lse, keypad, A);
}

}  // namespace tc
