// Block CSR / CSC of a 0/1 block mask, by one CTA (any whole number of warps).
#pragma once
#include "common.cuh"

// mat [nb*nb] uint8 -> CSR (row_ptr, col_idx, blk_row), CSC (col_ptr, row_idx, csc_pos) and the block count.  work [nb*nb] receives
// the CSR block id of every set cell, longest_col (if given) the entries of the longest column.  A warp per line, 32 cells per step: the rows' bits and starts are kept in shared
// memory, positions are ballot prefixes, nothing is read back from global memory.  Loops stay rolled (see pattern.cu).  (One thread per line took 13 us at nb = 64: 256 dependent byte loads.)
static __device__ void build_structure(const uint8_t* mat, int nb, int32_t* nnzb, int32_t* row_ptr, int32_t* col_idx, int32_t* blk_row,
                                       int32_t* col_ptr, int32_t* row_idx, int32_t* csc_pos, int32_t* work,
                                       int32_t* longest_col = nullptr) {
  __shared__ uint32_t s_bits[SPION_MAX_NB * (SPION_MAX_NB / 32)];
  __shared__ int s_ptr[SPION_MAX_NB + 1];
  __shared__ int s_row[SPION_MAX_NB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int W = (nb + 31) >> 5;
  const uint32_t below = (1u << lane) - 1u;
  // s_ptr[0 .. nb) holds counts: exclusive scan in place, the total in s_ptr[nb]
  auto scan = [&]() {
    if (warp == 0) {
      int carry = 0;
#pragma unroll 1
      for (int i0 = 0; i0 < nb; i0 += 32) {
        const int i = i0 + lane, n = i < nb ? s_ptr[i] : 0;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += y;
        }
        if (i < nb) s_ptr[i] = carry + upto - n;
        carry += __shfl_sync(0xffffffffu, upto, 31);
      }
      if (lane == 0) s_ptr[nb] = carry;
    }
    __syncthreads();
  };
  // ---- rows
#pragma unroll 1
  for (int r = warp; r < nb; r += nwarps) {
    int n = 0;
#pragma unroll 1
    for (int w = 0; w < W; ++w) {
      const int c = 32 * w + lane;
      const uint32_t b = __ballot_sync(0xffffffffu, c < nb && mat[(size_t)r * nb + c] != 0);
      if (lane == 0) s_bits[r * W + w] = b;
      n += __popc(b);
    }
    if (lane == 0) s_ptr[r] = n;
  }
  __syncthreads();
  scan();
  if (threadIdx.x == 0) *nnzb = s_ptr[nb];
#pragma unroll 1
  for (int r = threadIdx.x; r <= nb; r += blockDim.x) {
    row_ptr[r] = s_ptr[r];
    if (r < nb) s_row[r] = s_ptr[r];
  }
#pragma unroll 1
  for (int r = warp; r < nb; r += nwarps) {
    int pos = s_ptr[r];
#pragma unroll 1
    for (int w = 0; w < W; ++w) {
      const uint32_t b = s_bits[r * W + w];
      if ((b >> lane) & 1u) {
        const int c = 32 * w + lane, x = pos + __popc(b & below);
        col_idx[x] = c;
        blk_row[x] = r;
        work[(size_t)r * nb + c] = x;
      }
      pos += __popc(b);
    }
  }
  __syncthreads();
  // ---- columns
#pragma unroll 1
  for (int c = warp; c < nb; c += nwarps) {
    int n = 0;
#pragma unroll 1
    for (int r0 = 0; r0 < nb; r0 += 32) {
      const int r = r0 + lane;
      n += __popc(__ballot_sync(0xffffffffu, r < nb && ((s_bits[r * W + (c >> 5)] >> (c & 31)) & 1u)));
    }
    if (lane == 0) s_ptr[c] = n;
  }
  __syncthreads();
  if (longest_col && warp == 0) {
    int most = 0;
#pragma unroll 1
    for (int c = lane; c < nb; c += 32) most = max(most, s_ptr[c]);
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) *longest_col = most;
    __syncwarp();
  }
  scan();
#pragma unroll 1
  for (int c = threadIdx.x; c <= nb; c += blockDim.x) col_ptr[c] = s_ptr[c];
#pragma unroll 1
  for (int c = warp; c < nb; c += nwarps) {
    int pos = s_ptr[c];
#pragma unroll 1
    for (int r0 = 0; r0 < nb; r0 += 32) {
      const int r = r0 + lane;
      const bool on = r < nb && ((s_bits[r * W + (c >> 5)] >> (c & 31)) & 1u);
      const uint32_t b = __ballot_sync(0xffffffffu, on);
      if (on) {
        const int x = pos + __popc(b & below);
        row_idx[x] = r;
        int id = s_row[r];                             // the set cells before c in row r
#pragma unroll 1
        for (int w = 0; w < (c >> 5); ++w) id += __popc(s_bits[r * W + w]);
        csc_pos[x] = id + __popc(s_bits[r * W + (c >> 5)] & ((1u << (c & 31)) - 1u));
      }
      pos += __popc(b);
    }
  }
}
