// What the fp32 attention kernels share (simt_fused.cu, mma_fused.cu): operand tiles by cp.async, the value tiles of a block row.
#pragma once
#include "common.cuh"

namespace fp32 {

// the threads of problem g
template <int NT>
__device__ __forceinline__ void group_sync(int g) {
  if (NT == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(NT) : "memory");
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A [L x d] operand of one (b,h) matrix, or a value tile: element (i, n) at base + i*s_row + n*s_col.
struct Operand {
  const float* base;
  long long s_row, s_col;
  bool pieces;                                       // rows in 16-byte pieces
  __device__ __forceinline__ Operand(const float* p, const OperandLayout& l, int bh)
      : base(p + (long long)bh * l.bh_stride), s_row(l.sl), s_col(l.sd) {
    pieces = s_col == 1 && (s_row & 3) == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0;
  }
  __device__ __forceinline__ Operand(const float* p, int stride)
      : base(p), s_row(stride), s_col(1), pieces((reinterpret_cast<uintptr_t>(p) & 15) == 0) {}
};

// Start the asynchronous copy of rows row0 .. row0 + ROWS - 1 into shared memory by the NT threads of one problem.  The caller commits the
// group, waits for it and synchronises before the tile is read.  Place::template at<COLS>(row, piece): float offset of a 16-byte piece of a row.
template <class Place, int ROWS, int COLS, int NT>
__device__ __forceinline__ void load_tile(float* dst, const Operand& o, int row0, int t) {
  const float* src = o.base + row0 * o.s_row;
  if (o.pieces) {
    constexpr int STEP = NT / (COLS / 4);            // rows per round
    const int row = t / (COLS / 4), c4 = t % (COLS / 4);
    src += row * o.s_row + c4 * 4;
    const long long step = STEP * o.s_row;
#pragma unroll
    for (int i = 0; i < ROWS / STEP; ++i) {
      cp_async16(dst + Place::template at<COLS>(row + i * STEP, c4), src);
      src += step;
    }
  } else if (o.s_col == 1) {
    for (int idx = t; idx < ROWS * COLS; idx += NT) {
      const int row = idx / COLS, col = idx % COLS;
      cp_async4(dst + Place::template at<COLS>(row, col >> 2) + (col & 3), src + row * o.s_row + col);
    }
  } else {
#pragma unroll 4
    for (int idx = t; idx < ROWS * COLS; idx += NT) {
      const int row = idx % ROWS, col = idx / ROWS;
      cp_async4(dst + Place::template at<COLS>(row, col >> 2) + (col & 3), src + row * o.s_row + col * o.s_col);
    }
  }
}

// The value tiles of one block row: element (i, j) of its k-th tile at base + k * step + i * si + j.
struct RowTiles {
  long long base;
  int si, step;
  template <int BS>
  static __device__ __forceinline__ RowTiles of(const ValueLayout& vl, int rp, int nblk) {
    const long long base = (long long)rp * BS * BS;
    return vl.mode == VAL_ELEMCSR ? RowTiles{base, nblk * BS, BS} : RowTiles{base, BS, BS * BS};
  }
};
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float LOG2_E = 1.4426950408889634f;

// Four consecutive values of a value tile (tile rows are contiguous; `vec`: 16-byte aligned).
__device__ __forceinline__ float4 load_vals(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ void store_vals(float* p, float4 v, bool vec) {
  if (vec) *reinterpret_cast<float4*>(p) = v;
  else p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
}
__device__ __forceinline__ bool vec_ok(const float* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace fp32
