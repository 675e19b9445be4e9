// Pattern discovery on the GPU: convolution + block average pooling of the mean attention
// map, quantile threshold, the reference's greedy walkers, forced diagonal, block CSR/CSC.
//
// Replaces the CPU/Python block of the reference driver, main_conv_ff.py:255-279, and its
// recursive flood_fill (main_conv_ff.py:35-62); the top-k selection of main_conv.py:246-251;
// F == 1 gives main_ff.py:255 (no convolution).
//
// Integer outputs equal those of oracle/pattern.py: the float stages are fp64 sums rounded to fp32 once (conv_pool_kernel's in the
// oracle's order of additions, documented at each loop; diag_parts_kernel's in another), and the lerp is fused as there.
//
// The loops of the selection and of the structure (structure.cuh) are kept rolled: one CTA walks most of them a few times, and what it waits
// for is its instructions.  Unrolled as the compiler would, a call of 90 us takes 3 - 4 us more.
#include <atomic>

#include "common.cuh"
#include "structure.cuh"

namespace {

// ---------------------------------------------------------------- conv + pool (one CTA per cell)
// smem: tile[(bs+F-1)^2] fp32 (zero padded halo) | c[bs*bs] fp64 | rsum[bs] fp64
__global__ void __launch_bounds__(256) conv_pool_kernel(const float* __restrict__ A, int L, int bs, int kind, int F,
                                                        float* __restrict__ pooled) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int h = F / 2;
  const int T = bs + 2 * h;
  float* tile = reinterpret_cast<float*>(smem_raw);
  size_t off = ((size_t)T * T * sizeof(float) + 15) & ~(size_t)15;
  double* cval = reinterpret_cast<double*>(smem_raw + off);
  double* rsum = cval + (size_t)bs * bs;
  const int bi = blockIdx.y, bj = blockIdx.x, nb = gridDim.x;
  const int i0 = bi * bs - h, j0 = bj * bs - h;
  for (int t = threadIdx.x; t < T * T; t += blockDim.x) {
    const int ti = t / T, tj = t % T;
    const int gi = i0 + ti, gj = j0 + tj;
    tile[t] = (gi >= 0 && gi < L && gj >= 0 && gj < L) ? A[(size_t)gi * L + gj] : 0.0f;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < bs * bs; e += blockDim.x) {
    const int i = e / bs, j = e % bs;
    double c = 0.0;
    if (kind == SPION_CONV_DIAG) {
      // c = sum_{t=-h..h} A[i+t, j+t], added for t ascending (oracle: conv_fixed_order)
      for (int t = 0; t < F; ++t) c = c + (double)tile[(i + t) * T + (j + t)];
    } else {
      // box mean: u outer, v inner, ascending; one fp64 division
      for (int u = 0; u < F; ++u)
        for (int v = 0; v < F; ++v) c = c + (double)tile[(i + u) * T + (j + v)];
      c = c / (double)(F * F);
    }
    cval[e] = c;
  }
  __syncthreads();
  // r[i] = sum_jj c[i, jj]  (jj ascending), then p = sum_ii r[ii] (ii ascending): pool_fixed_order
  for (int i = threadIdx.x; i < bs; i += blockDim.x) {
    double r = 0.0;
    for (int jj = 0; jj < bs; ++jj) r = r + cval[i * bs + jj];
    rsum[i] = r;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double p = 0.0;
    for (int ii = 0; ii < bs; ++ii) p = p + rsum[ii];
    pooled[(size_t)bi * nb + bj] = (float)(p / (double)(bs * bs));
  }
}

// Diagonal filter of 31 taps, blocks of 32 or 64 (the reference's settings: main_conv_ff.py:258).  Filter and pooling are one weighted sum:
// an element counts in a cell as often as the diagonal through it has taps whose output lies in the cell's block.  With h = 15 an element
// (a, b) of its own block reaches that block's cell and, from the outer 16 rows and columns, the six cells above / left / below / right / on
// the diagonal:
//   own cell      min(15, min(a, b)) - max(-15, max(a, b) - BS + 1) + 1
//   above (-1,0)  min(15, b) - a        left (0,-1)  min(15, a) - b           (-1,-1)  15 - max(a, b)
//   below (+1,0)  min(a', a - b)        right (0,+1) min(b', b - a)           (+1,+1)  min(a', b')         a' = a - BS + 16, b' likewise
// where these are positive.  So every element is read once, converted once, and no filtered map is formed: the kernel writes seven
// partial sums per block, diag_combine_kernel adds the seven that belong to a cell.  All sums are fp64 with weights that are whole
// numbers (formed as sums of running sums, nothing is subtracted), rounded to fp32 once: the error is that of the ordered sums of conv_pool_kernel, some
// 1e-16, before the rounding.  An element whose weight is zero is left out, not multiplied: infinities stay where the filter has them.
//
// A lane owns a row of a block: one warp takes the 16 rows at the top and the 16 at the bottom, a second one the 32 between them (BS = 64);
// two buffers per block filled by cp.async, rows padded by 16 bytes (conflict-free 16-byte reads of one row per lane).  In the corners of a
// block the weights bend at the diagonal: running sums from both ends, added to one of two totals on either side of it.
// Bound by the pass over the map: two L = 4096 maps 125 us with the 31 ordered additions per element, 28 now, 4.8 TB/s (33 with one warp per block).
struct MapList { const float* A[16]; };
constexpr int DIAG_GROUPS = 6, DIAG_PARTS = 10;
template <int BS>
__global__ void __launch_bounds__(BS * DIAG_GROUPS) diag_parts_kernel(const __grid_constant__ MapList maps, int layers, int L, double* part) {
  static_assert(BS == 32 || BS == 64, "16 outer rows on either side, 0 or 32 between them");
  constexpr int TP = BS + 4, PIECES = BS / 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, gt = threadIdx.x % BS, group = threadIdx.x / BS;      // BS threads per block
  const bool outer = gt < 32;
  float* buf = reinterpret_cast<float*>(smem_raw) + (size_t)group * 2 * BS * TP;
  const int nb = L / BS, per = nb * nb;
  const int total = layers * per, step = (int)gridDim.x * DIAG_GROUPS;
  auto meet = [&]() {
    if constexpr (BS == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(BS) : "memory");
  };
  next_may_start();
  auto load = [&](int cell, float* to) {
    const int m = cell / per, rest = cell - m * per;
    const float* src = maps.A[m] + (size_t)(rest / nb) * BS * L + (rest % nb) * BS;
#pragma unroll 8
    for (int e = gt; e < BS * PIECES; e += BS) {
      const int r = e / PIECES, c = 4 * (e % PIECES);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to + r * TP + c)),
                   "l"(src + (size_t)r * L + c) : "memory");
    }
  };
  auto read16 = [](const float* p, double* x) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(p + 4 * i);
      x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
    }
  };
  int cell = blockIdx.x * DIAG_GROUPS + group;
  if (cell < total) load(cell, buf);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int n = 0; cell < total; cell += step, n ^= 1) {
    const float* t = buf + n * BS * TP;
    if (cell + step < total) load(cell + step, buf + (n ^ 1) * BS * TP);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    meet();
    double own = 0.0, left = 0.0, right = 0.0, vert = 0.0, diag = 0.0;      // vert, diag: upwards in lanes 0-15, downwards in 16-31
    double x[16];
    if (outer) {
      const bool low = lane < 16;
      const int a = lane & 15, w = low ? 15 - a : a;                        // w: weight of the row in the cell above / below
      const float* row = t + (low ? a : BS - 16 + a) * TP;
      // the 16 columns at the same end: weights bend at b = a
      read16(row + (low ? 0 : BS - 16), x);
      double up = 0.0, from0 = 0.0, from1 = 0.0;                            // up = x[0] + .. + x[b]; sums of it for b < a, a <= b < 15
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        up += x[b];
        if (b < a) from0 += up;                                             // in all: sum of (a - b)+ x
        else if (b < 15) from1 += up;                                       // sum of (15 - max(a, b)) x
      }
      double down = 0.0, to0 = 0.0, to1 = 0.0;                              // down = x[15] + .. + x[b]
#pragma unroll
      for (int b = 15; b > 0; --b) {
        down += x[b];
        if (b > a) to1 += down;                                             // sum of (b - a)+ x
        else to0 += down;                                                   // sum of min(a, b) x
      }
      own = fma(16.0, up, low ? to0 : from1);
      diag = low ? from1 : to0;
      vert = low ? to1 : from0;
      left = low ? from0 : 0.0;
      right = low ? 0.0 : to1;
      // the 16 columns at the other end
      read16(row + (low ? BS - 16 : 0), x);
      double s0 = 0.0, rise = 0.0, fall = 0.0;
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        s0 += x[b];
        if (b > 0) rise = fma((double)b, x[b], rise);
        if (b < 15) fall = fma((double)(15 - b), x[b], fall);
      }
      own += fma((double)(16 - w), s0, low ? fall : rise);
      if (low) right = rise; else left = fall;
      if constexpr (BS > 32) {                                              // the columns between
        double m0 = 0.0, m1 = 0.0;
        read16(row + 16, x);
#pragma unroll
        for (int b = 0; b < 16; ++b) m0 += x[b];
        read16(row + 32, x);
#pragma unroll
        for (int b = 0; b < 16; ++b) m1 += x[b];
        m0 += m1;
        own = fma((double)(31 - w), m0, own);
        s0 += m0;
      }
      if (w > 0) vert = fma((double)w, s0, vert);
    }
    if (!outer) {                                                           // the rows between: weights follow the column
      const float* row = t + (16 + lane) * TP;
      double o0 = 0.0, o1 = 0.0, l = 0.0, r = 0.0;
      read16(row, x);
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        o0 = fma((double)(16 + b), x[b], o0);
        if (b < 15) l = fma((double)(15 - b), x[b], l);
      }
      read16(row + 48, x);
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        o1 = fma((double)(31 - b), x[b], o1);
        if (b > 0) r = fma((double)b, x[b], r);
      }
      double m0 = 0.0, m1 = 0.0;
      read16(row + 16, x);
#pragma unroll
      for (int b = 0; b < 16; ++b) m0 += x[b];
      read16(row + 32, x);
#pragma unroll
      for (int b = 0; b < 16; ++b) m1 += x[b];
      own = fma(31.0, m0 + m1, o0 + o1);
      left = l;
      right = r;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      own += __shfl_xor_sync(0xffffffffu, own, o);
      left += __shfl_xor_sync(0xffffffffu, left, o);
      right += __shfl_xor_sync(0xffffffffu, right, o);
      if (!outer) continue;
      vert += __shfl_xor_sync(0xffffffffu, vert, o);
      diag += __shfl_xor_sync(0xffffffffu, diag, o);
    }
    own += __shfl_xor_sync(0xffffffffu, own, 16);
    left += __shfl_xor_sync(0xffffffffu, left, 16);
    right += __shfl_xor_sync(0xffffffffu, right, 16);
    // own | left | right | above | above left | below | below right | own, left, right of the rows between
    double* dst = part + (size_t)cell * DIAG_PARTS;
    if (lane == 0) { double* d3 = dst + (outer ? 0 : 7); d3[0] = own; d3[1] = left; d3[2] = right; }
    if (outer && lane == 0) { dst[3] = vert; dst[4] = diag; }
    if (outer && lane == 16) { dst[5] = vert; dst[6] = diag; }
    meet();                                                                 // the buffer is refilled from here on
  }
}

// A cell: its own block's sum and what the blocks around it have for it, added in a fixed order.  between: blocks of 64.
__device__ __forceinline__ float combine_cell(const double* part, int cell, int nb, bool between, double area) {
  const int rest = cell % (nb * nb), r = rest / nb, c = rest - r * nb;
  const bool up = r > 0, down = r + 1 < nb, lt = c > 0, rt = c + 1 < nb;
  const double* p = part + (size_t)cell * DIAG_PARTS;
  const int line = nb * DIAG_PARTS;
  double s = p[0];
  s += rt ? p[DIAG_PARTS + 1] : 0.0;
  s += lt ? p[-DIAG_PARTS + 2] : 0.0;
  if (between) {
    s += p[7];
    s += rt ? p[DIAG_PARTS + 8] : 0.0;
    s += lt ? p[-DIAG_PARTS + 9] : 0.0;
  }
  s += down ? p[line + 3] : 0.0;
  s += down && rt ? p[line + DIAG_PARTS + 4] : 0.0;
  s += up ? p[-line + 5] : 0.0;
  s += up && lt ? p[-line - DIAG_PARTS + 6] : 0.0;
  return (float)(s / area);
}
__global__ void __launch_bounds__(256) diag_combine_kernel(const double* part, int nb, int total, bool between, double area, float* __restrict__ pooled) {
  next_may_start();
  wait_for_kernel_before();
  const int cell = blockIdx.x * 256 + threadIdx.x;
  if (cell < total) pooled[cell] = combine_cell(part, cell, nb, between, area);
}

// Lets kernel K use `bytes` (always the same) of shared memory on the current device, once: the call is a microsecond or two of a small
// discovery's 20 on the host.
template <auto K>
int allow_smem(int bytes) {
  static std::atomic<bool> done[64];
  int dev = 0;
  SPION_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return SPION_OK;
  SPION_CUDA_TRY(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return SPION_OK;
}

template <int BS>
int launch_diag(const MapList& maps, int layers, int L, int nb, double* part, float* pooled, bool combine, cudaStream_t st) {
  const int smem = DIAG_GROUPS * 2 * BS * (BS + 4) * (int)sizeof(float), total = layers * nb * nb;
  const int sms = sm_count();
  if (sms < 1) return SPION_ERR_CUDA;
  const int rc = allow_smem<diag_parts_kernel<BS>>(smem);
  if (rc) return rc;
  const int ctas = (total + DIAG_GROUPS - 1) / DIAG_GROUPS, cap = (BS == 64 ? 1 : 4) * sms;      // 209 KB or 55 KB each
  diag_parts_kernel<BS><<<ctas < cap ? ctas : cap, BS * DIAG_GROUPS, smem, st>>>(maps, layers, L, part);
  SPION_LAUNCH_CHECK();
  if (combine)
    SPION_CUDA_TRY(launch_after(diag_combine_kernel, dim3((total + 255) / 256), dim3(256), 0, st, (const double*)part, nb, total, BS == 64, (double)(BS * BS), pooled));
  return SPION_OK;
}

// ---------------------------------------------------------------- order statistics (one CTA)
__device__ __forceinline__ uint32_t order_key(float x) {
  uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

// k-th smallest (0-based) of vals[0..n), by a block of 1024 threads: the range of the keys is cut into 1024 bins, then the bin that holds the
// k-th key, until a bin is one key (values of a map share their leading bits: three rounds, the second and third over the few keys of a
// bin; four rounds of 8-bit digits from the top, most atomics of the first two on the same counters, took 5 us of this kernel's 23).
// A warp whose keys fall into one bin counts them in one go.  All threads call it; s_sel: 4 words, s_hist: 1024.
__device__ __forceinline__ float select_kth(const float* vals, int n, int k, int* s_hist, uint32_t* s_sel) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t least = 0xffffffffu, most = 0;
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += 1024) {
    const uint32_t key = order_key(vals[i]);
    least = min(least, key);
    most = max(most, key);
  }
  least = __reduce_min_sync(0xffffffffu, least);
  most = __reduce_max_sync(0xffffffffu, most);
  if (threadIdx.x == 0) { s_sel[0] = 0xffffffffu; s_sel[1] = 0; }
  __syncthreads();
  if (lane == 0) { atomicMin(&s_sel[0], least); atomicMax(&s_sel[1], most); }
  __syncthreads();
  uint32_t base = s_sel[0], range = s_sel[1] - base;               // keys base .. base + range
#pragma unroll 1
  while (range > 0) {
    const int shift = max(0, 22 - __clz(range));                   // 32 - clz bits, ten of them for the bins
    s_hist[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 1024) {
      const int i = i0 + threadIdx.x;
      const uint32_t key = i < n ? order_key(vals[i]) : 0u, off = key - base;
      const bool in = i < n && key >= base && off <= range;
      const int bin = in ? (int)(off >> shift) : -1;
      const bool all = __all_sync(0xffffffffu, bin == __shfl_sync(0xffffffffu, bin, 0));
      if (in && (!all || lane == 0)) atomicAdd(&s_hist[bin], all ? 32 : 1);
    }
    __syncthreads();
    // inclusive sums of the bins: a warp scans its 32, every warp the sums of the warps before it
    const int mine = s_hist[threadIdx.x];
    int upto = mine;
#pragma unroll 1
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    __syncthreads();
    if (lane == 31) s_hist[warp] = upto;
    __syncthreads();
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? s_hist[lane] : 0);
    upto += before;
    if (k >= upto - mine && k < upto) { s_sel[2] = threadIdx.x; s_sel[3] = (uint32_t)(k - (upto - mine)); }
    __syncthreads();
    base += s_sel[2] << shift;
    range = (1u << shift) - 1u;
    k = (int)s_sel[3];
  }
  return key_to_float(base);
}

// ---------------------------------------------------------------- selection (one CTA)
// select == PATHS: thresh = torch.quantile(pooled, q) (linear), then 2*nb greedy walkers.
// select == TOPK : the kcount largest cells (ties: lower flat index first).
// One CTA per map; its block structure follows in the same kernel: a chain of latencies, 17 us for two 64 x 64 maps (21 with the walkers
// step by step and the mask in global memory; 36 us of selection and 13 us of structure for each of them with one launch per map and
// step).  copies: how many times the 0/1 float mask is written, `mats_step` floats apart (the driver's stacked list, main_conv_ff.py:298-299).
constexpr int SELECT_SMEM_CELLS = 128 * 128;           // maps up to this size are kept in shared memory
// Up to this size select_kernel adds the parts of the cells itself: a launch between the two kernels is 3 us of the host, which is what a
// small call waits for, but one SM reads the parts slowly, 32 sectors a load.  Time by the selection ÷ by a launch of their own, 1, 2, 6 maps:
//   cells             1024              1600              1936              2304              3136              4096
//   blocks of 32  0.96 0.96 0.98   0.97 0.98 0.98   0.97 0.97 0.97   0.96 0.96 0.98   1.00 1.02 1.03   1.10 1.09 1.09
//   blocks of 64  0.96 0.98 0.99   0.96 1.07 1.06   1.00 1.16 1.12   1.03 1.16 1.12   1.13 1.26 1.17   1.20 1.27 1.19
constexpr int COMBINE_CELLS = 1536;
constexpr int SELECT_SMEM_BYTES = 7;                   // per cell: value, where a walker goes from it, mask
struct SelectOut {
  uint8_t* mat;
  float *thresh, *mats;
  int32_t *nnzb, *row_ptr, *col_idx, *blk_row, *col_ptr, *row_idx, *csc_pos, *work;
  int copies;
  long long mats_step;
};
template <bool SMALL>                                  // up to SELECT_SMEM_CELLS
__global__ void __launch_bounds__(1024) select_kernel(float* pooled_all, const double* part, bool between, double area, int nb, int select, float q,
                                                      int kcount, const __grid_constant__ SelectOut out) {
  extern __shared__ float s_val[];
  __shared__ int hist[1024];
  __shared__ uint32_t s_sel[4];
  __shared__ float s_thresh;
  __shared__ int s_warp[32];
  __shared__ int s_running;
  const size_t cells = (size_t)nb * nb;
  const int n = nb * nb;
  uint16_t* s_to = reinterpret_cast<uint16_t*>(s_val + n);
  uint8_t* mat_out = out.mat + blockIdx.x * cells;
  uint8_t* mat = SMALL ? reinterpret_cast<uint8_t*>(s_to + n) : mat_out;
  float* thresh_out = out.thresh ? out.thresh + blockIdx.x : nullptr;
  const float* pooled = SMALL ? s_val : pooled_all + blockIdx.x * cells;
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += 1024) mat[i] = 0;
  wait_for_kernel_before();
  if (SMALL) {
    float* from = pooled_all + blockIdx.x * cells;
    if (part) {
#pragma unroll 2
      for (int i = threadIdx.x; i < n; i += 1024) from[i] = s_val[i] = combine_cell(part, blockIdx.x * n + i, nb, between, area);
    } else {
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += 1024) s_val[i] = from[i];
    }
  }
  __syncthreads();

  if (select == SPION_SELECT_PATHS) {
    // torch.quantile: rank = fp32(q) * fp32(n-1); lerp(lo, hi, w) as torch's fused CPU kernel
    const float rank = __fmul_rn(q, (float)(n - 1));
    const float fl = floorf(rank);
    const int lo_i = (int)fl;
    const int hi_i = (int)ceilf(rank);
    const float w = __fsub_rn(rank, fl);
    const float lo = select_kth(pooled, n, lo_i, hist, s_sel);
    // the next order statistic: lo again if it occurs often enough, else the smallest value above it
    float hi = lo;
    if (hi_i != lo_i) {
      const uint32_t klo = order_key(lo);
      int le = 0;
      uint32_t above = 0xffffffffu;
#pragma unroll 1
      for (int i = threadIdx.x; i < n; i += 1024) {
        const uint32_t key = order_key(pooled[i]);
        if (key <= klo) ++le; else above = min(above, key);
      }
      le = __reduce_add_sync(0xffffffffu, le);
      above = __reduce_min_sync(0xffffffffu, above);
      if (threadIdx.x == 0) { hist[0] = 0; hist[1] = -1; }
      __syncthreads();
      if ((threadIdx.x & 31) == 0) {
        atomicAdd(&hist[0], le);
        atomicMin(reinterpret_cast<unsigned int*>(&hist[1]), above);
      }
      __syncthreads();
      if (hist[0] <= hi_i) hi = key_to_float((uint32_t)hist[1]);
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      const float d = __fsub_rn(hi, lo);
      float t;
      if (fabsf(w) < 0.5f) t = __fmaf_rn(w, d, lo);
      else t = __fmaf_rn(-d, __fsub_rn(1.0f, w), hi);
      s_thresh = t;
      if (thresh_out) *thresh_out = t;
    }
    __syncthreads();
    const float thresh = s_thresh;
    // walkers: seeds (0,k) then (k,0); main_conv_ff.py:271-274.  Order-free: marks are idempotent.  Stops on the zero guard row /
    // column (:37).  step(): where a walker goes from (x, y), and whether the cell it reaches is marked.
    auto step = [&](int x, int y) -> int {
      const float D = (x + 1 < nb) ? pooled[(size_t)(x + 1) * nb + y] : 0.0f;
      const float R = (y + 1 < nb) ? pooled[(size_t)x * nb + y + 1] : 0.0f;
      const float G = (x + 1 < nb && y + 1 < nb) ? pooled[(size_t)(x + 1) * nb + y + 1] : 0.0f;
      const float first = D > R ? D : R;
      const int to = first > G ? (D > R ? 1 : 2) : 3;
      const float v = first > G ? first : G;
      return to | (v > thresh && v > 0.0f ? 4 : 0);
    };
    if (SMALL) {
      // all steps first, in parallel, so that a walker's chain is one load per cell: the next cell, whether it is marked, or the end.  (All
      // walkers at once, cells passing on what is 2^k steps ahead in round k: 7 us for 64 x 64 cells on one SM, twice what these chains take.)
#pragma unroll 1
      for (int i = threadIdx.x; i < n; i += 1024) {
        const int x = i / nb, y = i - x * nb, t = step(x, y);
        s_to[i] = x + (t & 1) < nb && y + ((t >> 1) & 1) < nb ? (uint16_t)((i + (t & 1) * nb + ((t >> 1) & 1)) | (t & 4 ? 0x4000 : 0)) : (uint16_t)0x8000;
      }
      __syncthreads();
      if (threadIdx.x < 2 * nb) {
        uint32_t t = s_to[threadIdx.x < nb ? threadIdx.x : (threadIdx.x - nb) * nb];
#pragma unroll 1
        while (t < 0x8000) {
          const uint32_t at = t & 0x3fff;
          if (t & 0x4000) mat[at] = 1;
          t = s_to[at];
        }
      }
    } else {
#pragma unroll 1
      for (int s = threadIdx.x; s < 2 * nb; s += 1024) {
        int x = (s < nb) ? 0 : s - nb;
        int y = (s < nb) ? s : 0;
        while (x < nb && y < nb) {
          const int t = step(x, y);
          x += t & 1;
          y += (t >> 1) & 1;
          if ((t & 4) && x < nb && y < nb) mat[(size_t)x * nb + y] = 1;
        }
      }
    }
  } else {
    if (thresh_out && threadIdx.x == 0) *thresh_out = 0.0f;
    if (kcount > 0) {
      const int kk = kcount > n ? n : kcount;
      const float v = select_kth(pooled, n, n - kk, hist, s_sel);   // kk-th largest
      // count strictly greater
      if (threadIdx.x == 0) s_running = 0;
      __syncthreads();
      int local = 0;
#pragma unroll 1
      for (int i = threadIdx.x; i < n; i += 1024) {
        if (pooled[i] > v) { mat[i] = 1; ++local; }
      }
      atomicAdd(&s_running, local);
      __syncthreads();
      const int need = kk - s_running;                 // how many cells equal to v to take
      __syncthreads();
      if (threadIdx.x == 0) s_running = 0;
      __syncthreads();
      const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = 32;
#pragma unroll 1
      for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const int flag = (i < n && pooled[i] == v) ? 1 : 0;
        const unsigned bal = __ballot_sync(0xffffffffu, flag);
        const int in_warp = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) s_warp[wid] = __popc(bal);
        __syncthreads();
        int before = s_running;
#pragma unroll 1
        for (int w2 = 0; w2 < wid; ++w2) before += s_warp[w2];
        if (flag && before + in_warp < need) mat[i] = 1;
        __syncthreads();
        if (threadIdx.x == 0) {
          int tot = 0;
#pragma unroll 1
          for (int w2 = 0; w2 < nwarps; ++w2) tot += s_warp[w2];
          s_running += tot;
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int i = threadIdx.x; i < nb; i += 1024) mat[(size_t)i * nb + i] = 1;   // main_conv_ff.py:277-278
  __syncthreads();
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += 1024) {
    const uint8_t on = mat[i];
    if (SMALL) mat_out[i] = on;
    float* m = out.mats + blockIdx.x * cells + i;
#pragma unroll 4
    for (int c = 0; c < out.copies; ++c) m[c * out.mats_step] = (float)on;
  }
  build_structure(mat, nb, out.nnzb + blockIdx.x, out.row_ptr + (size_t)blockIdx.x * (nb + 1), out.col_idx + blockIdx.x * cells,
                  out.blk_row + blockIdx.x * cells, out.col_ptr + (size_t)blockIdx.x * (nb + 1), out.row_idx + blockIdx.x * cells,
                  out.csc_pos + blockIdx.x * cells, out.work + blockIdx.x * cells);
}

// ---------------------------------------------------------------- mean over (b,h) of the dense map
// out[i*L + j] = (1/H) sum_h ( (1/B) sum_b in[b*H + h][...] ), b and h ascending.
// A thread owns four consecutive memory columns of one row (16-byte loads, 512 contiguous bytes per warp and
// matrix) and keeps eight matrices' loads in flight; the additions stay in the order above.  L % 128 == 0.
__global__ void __launch_bounds__(256) mean_map_kernel(const float* __restrict__ attn, int B, int H, int L, int transposed,
                                                       float* __restrict__ A) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
  const size_t LL = (size_t)L * L;
  const int row = blockIdx.y * 8 + ty, col = blockIdx.x * 128 + 4 * tx;        // memory coordinates
  const size_t m = (size_t)row * L + col;
  float4 acc_h = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int hh = 0; hh < H; ++hh) {
    float4 acc_b = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int b = 0; b < B; ++b) {
      const float4 v = *reinterpret_cast<const float4*>(attn + (size_t)(b * H + hh) * LL + m);
      acc_b.x += v.x; acc_b.y += v.y; acc_b.z += v.z; acc_b.w += v.w;
    }
    acc_h.x += acc_b.x / (float)B; acc_h.y += acc_b.y / (float)B;
    acc_h.z += acc_b.z / (float)B; acc_h.w += acc_b.w / (float)B;
  }
  const float4 r = make_float4(acc_h.x / (float)H, acc_h.y / (float)H, acc_h.z / (float)H, acc_h.w / (float)H);
  if (transposed) {                                          // memory (row = j, col = i) -> A[i][j]
    A[(size_t)(col + 0) * L + row] = r.x;
    A[(size_t)(col + 1) * L + row] = r.y;
    A[(size_t)(col + 2) * L + row] = r.z;
    A[(size_t)(col + 3) * L + row] = r.w;
  } else {
    *reinterpret_cast<float4*>(A + m) = r;
  }
}

// The same for any L that is a multiple of 32 (one value per thread, 32 x 32 tiles through shared memory).
__global__ void mean_map_kernel32(const float* __restrict__ attn, int B, int H, int L, int transposed,
                                  float* __restrict__ A) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x, ty = threadIdx.y;             // 32 x 8
  const size_t LL = (size_t)L * L;
  for (int rr = ty; rr < 32; rr += 8) {
    // memory coordinates: row = blockIdx.y*32 + rr, col = blockIdx.x*32 + tx
    const size_t m = (size_t)(blockIdx.y * 32 + rr) * L + blockIdx.x * 32 + tx;
    float acc_h = 0.0f;
    for (int hh = 0; hh < H; ++hh) {
      float acc_b = 0.0f;
#pragma unroll 8
      for (int b = 0; b < B; ++b) acc_b += attn[(size_t)(b * H + hh) * LL + m];   // loads of eight matrices in flight; sum in order
      acc_h += acc_b / (float)B;
    }
    tile[rr][tx] = acc_h / (float)H;
  }
  __syncthreads();
  for (int rr = ty; rr < 32; rr += 8) {
    if (transposed) {
      // memory (row=j, col=i) -> A[i][j]
      const int i = blockIdx.x * 32 + rr, j = blockIdx.y * 32 + tx;
      A[(size_t)i * L + j] = tile[tx][rr];
    } else {
      const int i = blockIdx.y * 32 + rr, j = blockIdx.x * 32 + tx;
      A[(size_t)i * L + j] = tile[rr][tx];
    }
  }
}

// Mean over the (b,h) matrices of block-tile probabilities: one CTA per selected block.
// A[i, j] = (1 / BH) * sum_bh P[bh][blk][i % bs][j % bs]; cells of unselected blocks stay 0.
template <typename T>
__global__ void __launch_bounds__(256) mean_map_tiles_kernel(const T* __restrict__ P, const int32_t* __restrict__ blk_row,
                                                             const int32_t* __restrict__ col_idx, int bs, int nnzb,
                                                             int BH, int L, float* __restrict__ A) {
  const int blk = blockIdx.x;
  const int r = blk_row[blk], c = col_idx[blk];
  const int n = bs * bs;
  const float inv = 1.0f / (float)BH;
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    float acc = 0.f;
    const T* src = P + (size_t)blk * n + e;
#pragma unroll 8
    for (int bh = 0; bh < BH; ++bh) acc += to_f32(src[(size_t)bh * nnzb * n]);   // eight loads in flight; sum in order
    A[(size_t)(r * bs + e / bs) * L + c * bs + e % bs] = acc * inv;
  }
}

}  // namespace

extern "C" int spion_mean_map_tiles(const void* P, int dtype, const int32_t* blk_row, const int32_t* col_idx,
                                    int block_size, int nnzb, int num_batches, int L, float* A, void* cuda_stream) {
  if (!P || !blk_row || !col_idx || !A) return SPION_ERR_ARG;
  if (block_size < 1 || nnzb < 0 || num_batches < 1 || L < 1 || L % block_size != 0) return SPION_ERR_SHAPE;
  if (dtype != SPION_F32 && dtype != SPION_BF16) return SPION_ERR_ARG;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  SPION_CUDA_TRY(cudaMemsetAsync(A, 0, (size_t)L * L * sizeof(float), st));
  if (nnzb == 0) return SPION_OK;
  if (dtype == SPION_F32)
    mean_map_tiles_kernel<float><<<nnzb, 256, 0, st>>>((const float*)P, blk_row, col_idx, block_size, nnzb,
                                                       num_batches, L, A);
  else
    mean_map_tiles_kernel<__nv_bfloat16><<<nnzb, 256, 0, st>>>((const __nv_bfloat16*)P, blk_row, col_idx, block_size,
                                                               nnzb, num_batches, L, A);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

namespace {
struct Scratch {                                                  // of a call, from the library's pool: given back whichever way the call ends
  void* p = nullptr;
  cudaStream_t st;
  explicit Scratch(cudaStream_t s) : st(s) {}
  bool take(size_t bytes) { return scratch_alloc(&p, bytes, st) == SPION_OK; }
  void give_back() { if (p) scratch_free(p, st); p = nullptr; }
  ~Scratch() { give_back(); }
};
}  // namespace

// Bytes of scratch that spion_discover_patterns_in can be given (per call of `layers` maps).
extern "C" long long spion_discover_scratch_bytes(int layers, int L, int block_size) {
  if (layers < 1 || L < 1 || block_size < 1) return 0;
  const long long nb = L / block_size;
  return layers * nb * nb * DIAG_PARTS * (long long)sizeof(double);
}

extern "C" int spion_discover_patterns(const float* const* host_A, int layers, int L, int block_size, int conv_kind, int F, int select,
                                       double param, uint8_t* mat, float* pooled, float* thresh, int32_t* nnzb,
                                       int32_t* row_ptr, int32_t* col_idx, int32_t* blk_row, int32_t* col_ptr,
                                       int32_t* row_idx, int32_t* csc_pos, int32_t* work, float* mats, int copies,
                                       int32_t* host_nnzb, void* cuda_stream) {
  return spion_discover_patterns_in(host_A, layers, L, block_size, conv_kind, F, select, param, mat, pooled, thresh, nnzb, row_ptr, col_idx,
                                    blk_row, col_ptr, row_idx, csc_pos, work, mats, copies, host_nnzb, nullptr, cuda_stream);
}

// ... with the partial sums of the filter in memory of the caller (8-byte aligned, spion_discover_scratch_bytes; NULL: the library's pool)
extern "C" int spion_discover_patterns_in(const float* const* host_A, int layers, int L, int block_size, int conv_kind, int F, int select,
                                          double param, uint8_t* mat, float* pooled, float* thresh, int32_t* nnzb,
                                          int32_t* row_ptr, int32_t* col_idx, int32_t* blk_row, int32_t* col_ptr,
                                          int32_t* row_idx, int32_t* csc_pos, int32_t* work, float* mats, int copies,
                                          int32_t* host_nnzb, double* scratch, void* cuda_stream) {
  if (!host_A || layers < 1 || layers > 16 || copies < 0 || (copies > 0 && !mats)) return SPION_ERR_ARG;
  MapList maps = {};
  for (int i = 0; i < layers; ++i) { maps.A[i] = host_A[i]; if (!host_A[i]) return SPION_ERR_ARG; }
  if (!mat || !pooled || !nnzb || !row_ptr || !col_idx || !blk_row || !col_ptr || !row_idx || !csc_pos || !work)
    return SPION_ERR_ARG;
  if (L < 1 || block_size < 1 || L % block_size != 0) return SPION_ERR_SHAPE;
  const int bs = block_size, nb = L / bs;
  if (nb > SPION_MAX_NB || bs > 128) return SPION_ERR_SHAPE;
  if (F < 1 || F % 2 == 0 || F > 65) return SPION_ERR_ARG;
  if (conv_kind != SPION_CONV_DIAG && conv_kind != SPION_CONV_BOX) return SPION_ERR_ARG;
  if (select != SPION_SELECT_PATHS && select != SPION_SELECT_TOPK) return SPION_ERR_ARG;
  if (select == SPION_SELECT_PATHS && !(param >= 0.0 && param <= 1.0)) return SPION_ERR_ARG;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  const size_t cells = (size_t)nb * nb;

  const int T = bs + F - 1;
  size_t smem = (((size_t)T * T * sizeof(float) + 15) & ~(size_t)15) + ((size_t)bs * bs + bs) * sizeof(double);
  // The opt-in above 48 KB belongs to the current device only (a process may drive several), and the
  // call is cheap: make it on every launch that needs it instead of remembering one process-wide size.
  bool aligned = true;
  for (int i = 0; i < layers; ++i) aligned = aligned && ((uintptr_t)host_A[i] & 15u) == 0;
  // the reference's filter takes the kernel above; without memory for its partial sums the general one answers
  double* part = nullptr;
  const bool fits = conv_kind == SPION_CONV_DIAG && F == 31 && (bs == 64 || bs == 32) && aligned;
  const bool given = fits && scratch && ((uintptr_t)scratch & 7) == 0;
  Scratch own(st);
  const bool diag = fits && (given || own.take(layers * cells * DIAG_PARTS * sizeof(double)));
  if (diag) part = given ? scratch : (double*)own.p;
  const bool alone = diag && cells > COMBINE_CELLS;                 // the parts of a cell by a kernel of their own
  if (diag) {
    const int rc = bs == 64 ? launch_diag<64>(maps, layers, L, nb, part, pooled, alone, st) : launch_diag<32>(maps, layers, L, nb, part, pooled, alone, st);
    if (rc) return rc;
  } else {
    if (smem > 48 * 1024)
      SPION_CUDA_TRY(cudaFuncSetAttribute(conv_pool_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int i = 0; i < layers; ++i) {
      conv_pool_kernel<<<dim3(nb, nb), 256, smem, st>>>(host_A[i], L, bs, conv_kind, F, pooled + i * cells);
      SPION_LAUNCH_CHECK();
    }
  }

  int kcount = 0;
  if (select == SPION_SELECT_TOPK) kcount = (int)((double)(nb * nb) * param - (double)nb);   // main_conv.py:247
  const bool small = cells <= SELECT_SMEM_CELLS;
  auto kernel = small ? select_kernel<true> : select_kernel<false>;
  const size_t dyn = small ? cells * SELECT_SMEM_BYTES : 0;
  if (small) {
    const int rc = allow_smem<select_kernel<true>>(SELECT_SMEM_CELLS * SELECT_SMEM_BYTES);
    if (rc) return rc;
  }
  const SelectOut out{mat, thresh, mats, nnzb, row_ptr, col_idx, blk_row, col_ptr, row_idx, csc_pos, work, copies, (long long)(layers * cells)};
  SPION_CUDA_TRY(launch_after(kernel, dim3(layers), dim3(1024), dyn, st, pooled, (const double*)(diag && !alone ? part : nullptr), bs == 64, (double)(bs * bs), nb, select, (float)param, kcount, out));
  own.give_back();                                               // behind the last kernel: between two of them it would keep the second waiting
  if (host_nnzb) {
    SPION_CUDA_TRY(cudaMemcpyAsync(host_nnzb, nnzb, layers * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    SPION_CUDA_TRY(cudaStreamSynchronize(st));
  }
  return SPION_OK;
}

extern "C" int spion_discover_pattern(const float* A, int L, int block_size, int conv_kind, int F, int select,
                                      double param, uint8_t* mat, float* pooled, float* thresh, int32_t* nnzb,
                                      int32_t* row_ptr, int32_t* col_idx, int32_t* blk_row, int32_t* col_ptr,
                                      int32_t* row_idx, int32_t* csc_pos, int32_t* work, int32_t* host_nnzb,
                                      void* cuda_stream) {
  return spion_discover_patterns(&A, 1, L, block_size, conv_kind, F, select, param, mat, pooled, thresh, nnzb, row_ptr, col_idx, blk_row,
                                 col_ptr, row_idx, csc_pos, work, nullptr, 0, host_nnzb, cuda_stream);
}

extern "C" int spion_mean_attention_map(const float* attn, int batch, int heads, int L, int transposed, float* A,
                                        void* cuda_stream) {
  if (!attn || !A) return SPION_ERR_ARG;
  if (batch < 1 || heads < 1 || L < 32 || L % 32 != 0) return SPION_ERR_SHAPE;
  const bool aligned = (((uintptr_t)attn | (uintptr_t)A) & 15u) == 0;          // 16-byte loads and stores
  if (L % 128 == 0 && aligned)
    mean_map_kernel<<<dim3(L / 128, L / 8), 256, 0, (cudaStream_t)cuda_stream>>>(attn, batch, heads, L, transposed, A);
  else
    mean_map_kernel32<<<dim3(L / 32, L / 32), dim3(32, 8), 0, (cudaStream_t)cuda_stream>>>(attn, batch, heads, L,
                                                                                            transposed, A);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}
