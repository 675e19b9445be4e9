// The narrow linear layers around the attention call (torch.nn.Linear in the reference: models/attention.py:55-57,102 and the
// feed-forward block of models/model_transformer.py) as two tensor-core kernels:
//
//   k_lin_gemm    Y[T, N] = A[T, K] B + bias     A: tokens x features; B = W^T (forward) or W (gradient of the input)
//   k_lin_wgrad   dW[N, K] = dY^T X, db = column sums of dY, partial sums per CTA, then k_lin_reduce
//
// With K, N of 32 .. a few hundred and T of 10^3 .. 10^6 tokens the work is bound by the passes over the token matrices, so
// the kernels read every token matrix once, in the form its producer left it (fp32 or bf16, row-major or split into heads,
// up to three matrices side by side), convert on the way into shared memory, add the bias and write the form the consumer
// reads: no casts, no head-split copies, no concatenation, no separate bias or bias-gradient pass.
//
// Precision.  bf16 mode: operands rounded to bf16, fp32 accumulation (what mixed precision asks for).  fp32 mode: every fp32
// operand is split into three bf16 parts (8 + 8 + 8 significant bits: the split is exact) and the six partial products of
// weight 2^0, 2^-8 and 2^-16 are accumulated in fp32; the dropped ones are below 2^-25 of the product, i.e. below the rounding
// of an fp32 multiplication.  A sum in tensor memory is truncated at every step, which adds up to a bias of half a unit in the last
// place per step.  In the weight gradient, where a sum runs over all tokens, the leading products therefore go round as many
// accumulators as tensor memory holds, the small ones to one of their own, and a CTA takes no more tokens than leave CHAIN
// steps to each; what the accumulators and the CTAs hold is added in fp32.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"
#include "tc_tiles.cuh"

using namespace tc;

namespace {

// Set by a bounded wait that gave up.  The linear layers have no context of their own: one word per device; launches after it
// leave at once, as those of the attention kernels do, until spion_check_device_status or spion_linear_status has reported it.
__device__ int g_lin_status;

// Tokens x features, up to three equally wide matrices side by side, row-major or split into heads [T / L, heads, L, d].
// Row-major is the same with one head of width `per` and one sequence of all tokens.
struct TokMat {
  void* p[3];
  int per, d, dsh, L;       // features per matrix; head width, its log2 (31: one head); tokens per sequence
  long long hstride, bstride;
};
// Row and column parts of an element's offset are kept apart: rows advance by a constant step, columns hardly change, so the
// loops below compute no division.
struct RowIt {
  int b, l;                 // sequence, position
  __device__ __forceinline__ void init(const TokMat& m, int t) { b = t / m.L; l = t - b * m.L; }
  __device__ __forceinline__ long long off(const TokMat& m) const { return (long long)b * m.bstride + (long long)l * m.d; }
  __device__ __forceinline__ void add(const TokMat& m, int db, int dl) {      // step = db sequences + dl positions, dl < L
    b += db; l += dl;
    if (l >= m.L) { l -= m.L; ++b; }
  }
};
template <typename E> __device__ __forceinline__ E* tok_col(const TokMat& m, int c) {       // column c of the stack, token 0
  const int i = (c >= m.per) + (c >= 2 * m.per);
  c -= i * m.per;
  const int h = c >> m.dsh;
  return reinterpret_cast<E*>(i == 0 ? m.p[0] : (i == 1 ? m.p[1] : m.p[2])) + (h * m.hstride + (c - h * m.d));
}

__device__ __forceinline__ void ld_v8(const void* p, uint32_t (&r)[8]) {     // 32 bytes, 32-byte aligned
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "l"(p));
}
// ... or zeros.  One predicated load: with a branch around it the compiler joins the two values through register copies, which
// wait for the load where it is issued instead of where it is used.
__device__ __forceinline__ void ld_v8_if(bool in, const void* p, uint32_t (&r)[8]) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %9, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "mov.b32 %4, 0;\n\tmov.b32 %5, 0;\n\tmov.b32 %6, 0;\n\tmov.b32 %7, 0;\n\t"
      "@q ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
      : "l"(p), "r"((int)in));
}
__device__ __forceinline__ void st_v8(void* p, const uint32_t (&r)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void st_shared16(uint32_t a, const uint32_t (&w)[4]) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// bf16 operands need no conversion: sixteen bytes straight into their place in shared memory (zeros when !in), asynchronously
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// bf16 tokens through tensor maps (the GEMM's A), up to three matrices.  Row-major: boxes of 64 features, in the swizzle of the images.
// Split into heads: boxes of 64 tokens of one head; heads of 32 make a chunk of two images with 64-byte rows (32 features each).  A box
// whose rows are narrower than the swizzle is spread to its width, so that two heads cannot share 128-byte rows.
// Copied piece by piece, 16 bytes per thread, the loaders' address arithmetic was the limit: 1080 cycles per chunk of 16 KB, no time
// waited for memory.  524288 tokens, heads of 32, before and now: gradient of the input from three gradients of 64 features 103 -> 63 us,
// output projection 39 -> 27, its gradient (row-major) 39 -> 25.  Other widths, sequences that are no multiple of 64 and calls of one tile
// per CTA keep the copies; so do the weight gradients, where boxes of 64-byte rows were slower (two of them 136 us, 143 through maps).
enum : int { MAP_NONE = 0, MAP_ROWS = 1, MAP_HEADS = 2 };
struct LinMaps {
  CUtensorMap m[3];         // bf16 A
  CUtensorMap y[3], g, h;   // staged: Y, activation, pre-activation
};
__device__ __forceinline__ int which_matrix(const TokMat& t, int c) { return (c >= t.per) + (c >= 2 * t.per); }
// One thread: features c .. c + 63 of 64 tokens from t on of a head-split operand; the images of a chunk of heads of 32 are `image` bytes apart
__device__ __forceinline__ void load_heads(const TokMat& t, const CUtensorMap* m, uint32_t dst, uint32_t image, uint32_t bar, int c, int tok) {
  const int i = which_matrix(t, c), b = tok / t.L, heads = t.per >> t.dsh;
  c -= i * t.per;
  for (int f = 0; f < 64; f += t.d, dst += image)
    tma_load_2d(dst, m + i, bar, 0, (b * heads + ((c + f) >> t.dsh)) * t.L + (tok - b * t.L));
}

// Eight features of one token in registers: 8 fp32 words, or 4 words of bf16 pairs.
template <bool BF16> struct Raw { uint32_t w[BF16 ? 4 : 8]; };
// ... into the shared-memory images: SPLIT == 1 one bf16 image, SPLIT == 3 three (leading, middle, last 8 bits), `part` bytes apart
template <int SPLIT, bool BF16> __device__ __forceinline__ void raw_store(const Raw<BF16>& r, uint32_t addr, uint32_t part) {
  if constexpr (BF16) {
    st_shared16(addr, r.w);
  } else {
    uint32_t w[4];
    float f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r.w[i]);
#pragma unroll
    for (int s = 0; s < SPLIT; ++s) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w[i] = pack_bf16(f[2 * i], f[2 * i + 1]);
        if (s + 1 < SPLIT) { f[2 * i] -= bf16_lo(w[i]); f[2 * i + 1] -= bf16_hi(w[i]); }
      }
      st_shared16(addr + s * part, w);
    }
  }
}

// the partial products of the split operands, smallest first: (part of A, part of B)
template <int SPLIT> struct Prod { static constexpr int N = 1; __device__ static int a(int) { return 0; } __device__ static int b(int) { return 0; } };
template <> struct Prod<3> {
  static constexpr int N = 6;
  __device__ static constexpr int a(int i) { return i == 0 ? 0 : i == 1 ? 1 : i == 2 ? 2 : i == 3 ? 0 : i == 4 ? 1 : 0; }
  __device__ static constexpr int b(int i) { return i == 0 ? 2 : i == 1 ? 1 : i == 2 ? 0 : i == 3 ? 1 : i == 4 ? 0 : 0; }
};

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) { return tc::warp_wait(bar, parity, &g_lin_status, ERR_MMA_WAIT); }

// ------------------------------------------------------------------------------------------------ GEMM over tokens
enum { EPI_NONE = 0, EPI_GELU = 1, EPI_DGELU = 2 };

struct GemmArgs {
  TokMat A, Y;
  const float* W[3];        // stacked along their rows, each [wper, wld]
  const float* bias[3];     // [wper] each, or null (forward only)
  int wper, wld;
  int T, K, N;              // tokens, contraction length of this launch, output features
  int k0;                   // first contraction index of this launch
  int accum;                // add to Y (fp32) instead of overwriting it: a contraction split over several launches
  int nc, nstages;          // output features per CTA (blockIdx.y), stages of the A ring
  int nacc;                 // accumulators per tile (fp32 mode): the leading products rotate over nacc - 1 of them by chunk
  int parts;                // bf16 gradient of three stacked layers: chunks per layer (0: one accumulator for the whole contraction)
  int tma;                  // bf16 A through maps.m[0 .. 2] (MAP_*)
  int staged;               // outputs (and h) through shared memory and the other maps
  int table;                // GELU or its derivative by table (which kernel: the host's choice)
  const __nv_bfloat16* h;   // EPI_DGELU: pre-activation [T, N]
  __nv_bfloat16* g;         // EPI_GELU: activation [T, N] (Y receives the pre-activation)
  // What a backward reads in place of the caller's tensors.  262144 tokens of 64 fp32 features: 33 MB written here, 33 MB less read by
  // the weight gradient; the layer of 128 x 2 matrices, L = 4096 went from 1432 to 1458 us.
  __nv_bfloat16* x_copy;    // or null: A as the products use it, [T, K] (fp32 tokens in bf16 mode)
  float* w_copy;            // or null: the stacked W
  const float* mask;        // pen not null: key-padding mask [T / pen_L, pen_L] -> penalties of pen_heads matrices each
  float* pen;
  int pen_heads, pen_L;
};

// The three parts of an infinity (or of a value that rounds to one in bf16) are not finite themselves, and their products are NaN
// where an fp32 product may be an infinity or a number.  A finite result has no such operand; the others are formed again as an
// fp32 sum in ascending order.  They are rare, and a NaN ends the sum.
__device__ __forceinline__ bool all_finite(float probe) { return probe == 0.f; }      // probe: a sum of 0 * value
__device__ __noinline__ void redo_outputs(const GemmArgs& a, bool transb, int t, int c, float* dst) {       // token t, outputs c .. c + 31
  RowIt row;
  row.init(a.A, t);
  for (int i = 0; i < 32; ++i) {
    if (fabsf(dst[i]) <= 3.402823466e38f) continue;
    const int n = c + i;
    float s = 0.f;
    for (int k = 0; k < a.k0 + a.K && s == s; ++k) {
      const int r = transb ? k : n, m = r / a.wper;      // row of the stacked W
      const float* w = (m == 0 ? a.W[0] : m == 1 ? a.W[1] : a.W[2]) + (size_t)(r - m * a.wper) * a.wld;
      s = fmaf(tok_col<const float>(a.A, k)[row.off(a.A)], w[transb ? n : k], s);
    }
    if (a.bias[0]) {
      const int m = n / a.wper;
      s += (m == 0 ? a.bias[0] : m == 1 ? a.bias[1] : a.bias[2])[n - m * a.wper];
    }
    dst[i] = s;
  }
}

constexpr int LG_LOADERS = 8;
constexpr int LG_DEPTH = 4;                              // bf16 operands: stages whose copies are in flight
constexpr int LG_THREADS = 32 * (LG_LOADERS + 1 + 8);
constexpr uint32_t CHUNK = 128 * 128;                    // [128 tokens x 64 features] bf16

// Gauss error linear unit, exact form (torch.nn.GELU's default)
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float dgelu(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// Both are functions of a bf16 number here, the pre-activation: x / 2 times 1 + erf, and the slope.  A CTA forms the factor, or the slope, of every
// number of a range of octaves once, with the functions above, and looks them up (83 instructions a value before): the outputs are the same bits.
// Outside of the range they are constants.  GELU: below 2^-9 x / 2 is what the activation rounds to (1 + erf is 0.8 2^-9 beside 1 at most, half a step
// of bf16 2^-9 at least), from 8 on erf is 1 to fp32.  Slope: from 16 on the exponential is zero; numbers below 2^-14, where erf is the first term of its series
// and the exponential 1, take a branch with the infinities and NaN.  65536 tokens, 64 x 64, functions, table: GELU 14.4 us, 12.4 for pre-activations of
// deviation 8, 1 and 0; its derivative 18.5, 16.4, of deviations 2^-17 and 0 too (with a call of the functions for every number outside of a table of
// 2^-14 to 8: 26.7, 14.0, 25.6; 36.9, 16.4, 34.9).
template <int EPI> struct Tab {
  static constexpr bool SLOPE = EPI == EPI_DGELU;
  static constexpr uint32_t FROM = SLOPE ? 0x3880u : 0x3b00u - 1u, END = SLOPE ? 0x4180u : 0x4100u;          // first and last, bits of a number without its sign
  static constexpr uint32_t LEN = END - FROM + 1, BYTES = 2 * LEN * 4;
  __device__ static __forceinline__ float entry(uint32_t i) {
    const uint32_t k = i < LEN ? i : i - LEN;
    const float x = __uint_as_float(((i < LEN ? 0u : 0x8000u) | (FROM + k)) << 16);
    return SLOPE ? dgelu(x) : k == 0 ? 1.0f : 1.0f + erff(x * 0.70710678118654752f);
  }
};
template <int EPI> __device__ __forceinline__ void look_up(const float* tab, const uint32_t (&w)[8], float (&v)[16]) {
  using T = Tab<EPI>;
  bool some = false;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const uint32_t bits = e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu, size = bits & 0x7fffu;
    if (T::SLOPE) {
      v[e] = tab[min(size - T::FROM, T::LEN - 1) + (bits >> 15) * T::LEN];
      some |= ((size + 0x80u) & 0x7fffu) < T::FROM + 0x80u;
    } else {
      v[e] = 0.5f * (e & 1 ? bf16_hi(w[e >> 1]) : bf16_lo(w[e >> 1])) * tab[min(max(size, T::FROM), T::END) - T::FROM + (bits >> 15) * T::LEN];
    }
  }
  if (T::SLOPE && some) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float x = e & 1 ? bf16_hi(w[e >> 1]) : bf16_lo(w[e >> 1]), c = 0.39894228040143268f;         // 1 / sqrt(2 pi): each summand's slope at 0
      v[e] = fabsf(x) < 0x1p-14f ? fmaf(c, x, fmaf(c, x, 0.5f)) : fmaf(x, 0.f, v[e]);
    }
  }
}
// From the table, or, where wide weights leave no room for it, from the functions
template <int EPI, bool TAB> __device__ __forceinline__ void activate(const float* tab, const uint32_t (&w)[8], float (&v)[16]) {
  if (TAB) {
    look_up<EPI>(tab, w, v);
    return;
  }
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const float x = e & 1 ? bf16_hi(w[e >> 1]) : bf16_lo(w[e >> 1]);
    v[e] = EPI == EPI_GELU ? gelu(x) : dgelu(x);
  }
}

// One persistent CTA per SM over tiles of 128 tokens: warps 0-7 bring 64-feature chunks of A through registers (a chunk of
// loads in flight while the previous one is converted) into a ring of shared-memory stages, warp 8 issues the MMAs
// (M = 128, two accumulator buffers in tensor memory), warps 9-16 write finished tiles.  W sits in shared memory for the
// whole run.  Bound by the HBM passes over A and Y.
// A lane has 32 features of a token: written from registers, an instruction touches 32 lines for 32 bytes each, 14 bytes a cycle and SM
// whatever the form of Y.  Calls of more tiles than CTAs write them to a tile of 32 x 32 in shared memory that a bulk store takes to
// its place, and fetch the pre-activations the same way; sequences that are no multiple of 32, and outputs that are added to, keep
// the stores from registers.  Us, before, with the table above, and with the tiles too: 65536 tokens, 64 x 128, GELU 20.6, 19.2, 17.6; its derivative
// 31.3, 25.9, 24.6; 524288 tokens 107, 94, 81 and 179, 141, 111; fp32, 262144 tokens, 64 x 192 67, -, 50; 64 x 64 37, -, 30.
template <int SPLIT, bool A_BF16, bool TRANSB, int EPI, bool Y_BF16, bool STAGED, bool TAB>
__global__ void __launch_bounds__(LG_THREADS, 1) k_lin_gemm(const __grid_constant__ GemmArgs a, const __grid_constant__ LinMaps maps) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int nchunks = (a.K + 63) >> 6;
  const int n0 = blockIdx.y * a.nc;
  const int nc = min(a.nc, a.N - n0);
  const int G = (a.nc + 63) >> 6;
  // bytes of one part of B: [nc rows x 64] per chunk (K-major), or G tiles [64 x 64] per chunk (contraction rows)
  const uint32_t bchunk = TRANSB ? (uint32_t)G * 8192u : (uint32_t)a.nc * 128u;
  const uint32_t bpart = ((uint32_t)nchunks * bchunk + 1023u) & ~1023u;
  const uint32_t sA = sbase + SPLIT * bpart;
  const uint32_t sBias = sA + a.nstages * SPLIT * CHUNK;
  const uint32_t bars = sBias + 1024u;
  const uint32_t full = bars, empty = bars + 64, acc_full = bars + 128, acc_empty = bars + 144, slot = bars + 160;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  float* bias_ptr = reinterpret_cast<float*>(smem_raw + (sBias - sbase));
  float* tab = reinterpret_cast<float*>(smem_raw + (bars + 256u - sbase));
  // staged: a tile of 32 x 32 outputs per writing warp, with GELU two, with its derivative one and one of pre-activations
  constexpr uint32_t OTILE = Y_BF16 ? 2048u : 4096u, OWARP = (EPI == EPI_NONE ? 1u : 2u) * OTILE;
  const uint32_t outs = (bars + 256u + (TAB ? Tab<EPI>::BYTES : 0u) + 1023u) & ~1023u, hbars = bars + 168;

  const int ntiles = (a.T + 127) >> 7;
  const int G_x = (int)gridDim.x;
  __shared__ int s_abort;
  const bool tma = A_BF16 && a.tma;
  const int my_chunks = ((ntiles - (int)blockIdx.x + G_x - 1) / G_x) * nchunks;
  auto tma_chunk = [&](int n) {                          // one thread
    const int c = (n % nchunks) * 64, st = n % a.nstages, t = ((int)blockIdx.x + n / nchunks * G_x) * 128;
    const uint32_t dst = sA + st * CHUNK;
    if (a.tma == MAP_ROWS) {
      const int i = which_matrix(a.A, c);
      mbar_expect_tx(full + 8 * st, CHUNK);
      tma_load_2d(dst, &maps.m[i], full + 8 * st, c - i * a.A.per, t);
    } else {                                             // 64 tokens each; rows past the end keep what is there, their results are dropped
      const uint32_t image = CHUNK / 2, rows = a.A.d == 32 ? 64 * 64 : 64 * 128;
      mbar_expect_tx(full + 8 * st, t + 64 < a.T ? CHUNK : CHUNK / 2);
      load_heads(a.A, maps.m, dst, image, full + 8 * st, c, t);
      if (t + 64 < a.T) load_heads(a.A, maps.m, dst + rows, image, full + 8 * st, c, t + 64);
    }
  };

  if (warp == LG_LOADERS) {
    if (lane == 0) {
      s_abort = *reinterpret_cast<volatile int*>(&g_lin_status);
      for (int i = 0; i < a.nstages; ++i) { mbar_init(full + 8 * i, tma ? 1 : LG_LOADERS); mbar_init(empty + 8 * i, 1); }
      for (int i = 0; i < 2; ++i) { mbar_init(acc_full + 8 * i, 1); mbar_init(acc_empty + 8 * i, 8); }
      for (int i = 0; i < 8; ++i) mbar_init(hbars + 8 * i, 1);
      fence_barrier_init();
      if (tma && s_abort == 0) {                         // the first chunks are on their way before the weights are converted
        fence_proxy_async();
        for (int n = 0; n < a.nstages && n < my_chunks; ++n) tma_chunk(n);
      }
    }
    __syncwarp();
    tmem_alloc(slot, 512u);
    tmem_relinquish();
  }
  // first chunk of the first tile is requested before the weights are converted
  constexpr int R = 4;
  const int lrow = tid >> 3, lc8 = tid & 7;
  using AE = typename std::conditional<A_BF16, __nv_bfloat16, float>::type;
  auto a_col = [&](int ch) -> const AE* {                // this thread's eight features of chunk ch, null past the end
    const int c = ch * 64 + lc8 * 8;
    return c < a.K ? tok_col<const AE>(a.A, c + a.k0) : nullptr;
  };
  RowIt row[R];                                          // rows of the tile whose loads are issued next
  const int step = G_x * 128, step_b = step / a.A.L, step_l = step - step_b * a.A.L;
  if (warp < LG_LOADERS) {
#pragma unroll
    for (int i = 0; i < R; ++i) row[i].init(a.A, min(a.T - 1, (int)blockIdx.x * 128 + lrow + 32 * i));
  }
  auto load_row = [&](const AE* col, int tile, int i) {
    Raw<false> r;
    ld_v8_if(col && tile * 128 + lrow + 32 * i < a.T, col + row[i].off(a.A), r.w);
    return r;
  };
  Raw<false> cur[R];
  if (!A_BF16 && warp < LG_LOADERS) {
    const AE* col = a_col(0);
#pragma unroll
    for (int i = 0; i < R; ++i) cur[i] = load_row(col, blockIdx.x, i);
  }

  // bf16: the first LG_DEPTH chunks are on their way before the weights are converted (their stages are free)
  int ld_n = 0, ld_tile = blockIdx.x, ld_ch = 0;
  auto copy_chunk = [&]() {
    const uint32_t dst = sA + (ld_n % a.nstages) * CHUNK;
    const AE* col = a_col(ld_ch);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = lrow + 32 * i;
      const bool in = col && ld_tile * 128 + r < a.T;
      cp_async16(dst + r * 128 + ((lc8 ^ (r & 7)) << 4), in ? col + row[i].off(a.A) : reinterpret_cast<const AE*>(a.A.p[0]), in);
    }
    cp_async_commit();
    ++ld_n;
    if (++ld_ch == nchunks) {
      ld_ch = 0; ld_tile += G_x;
#pragma unroll
      for (int i = 0; i < R; ++i) row[i].add(a.A, step_b, step_l);
    }
  };
  if constexpr (A_BF16) {
    if (warp < LG_LOADERS && !tma)
      while (ld_n < LG_DEPTH && ld_tile < ntiles) copy_chunk();
  }

  {                                                      // weights -> shared memory
    const int per_row = TRANSB ? nc >> 3 : a.K >> 3;
    const int rows = TRANSB ? a.K : nc;
    for (int idx = tid; idx < rows * per_row; idx += LG_THREADS) {
      const int r = idx / per_row, c8 = idx - r * per_row;
      const int gr = TRANSB ? a.k0 + r : n0 + r;         // row of the stacked W
      const int m = gr / a.wper;
      const float* src = (m == 0 ? a.W[0] : m == 1 ? a.W[1] : a.W[2]) + (size_t)(gr - m * a.wper) * a.wld + (TRANSB ? n0 : a.k0) + c8 * 8;
      Raw<false> v;
      const uint4 x = *reinterpret_cast<const uint4*>(src), y = *reinterpret_cast<const uint4*>(src + 4);
      v.w[0] = x.x; v.w[1] = x.y; v.w[2] = x.z; v.w[3] = x.w; v.w[4] = y.x; v.w[5] = y.y; v.w[6] = y.z; v.w[7] = y.w;
      const uint32_t dst = TRANSB ? ((uint32_t)((r >> 6) * G + (c8 >> 3)) * 8192u + (r & 63) * 128)
                                  : ((uint32_t)(c8 >> 3) * bchunk + r * 128);
      raw_store<SPLIT, false>(v, sbase + dst + (((c8 & 7) ^ (r & 7)) << 4), bpart);
      if (!TRANSB && SPLIT == 1 && a.w_copy && blockIdx.x == 0) {
        float4* to = reinterpret_cast<float4*>(a.w_copy + (size_t)gr * a.wld + c8 * 8);
        to[0] = *reinterpret_cast<const float4*>(&x);
        to[1] = *reinterpret_cast<const float4*>(&y);
      }
    }
    for (int n = tid; n < nc; n += LG_THREADS) {
      float b = 0.f;
      if (a.bias[0]) {
        const int m = (n0 + n) / a.wper;
        b = (m == 0 ? a.bias[0] : m == 1 ? a.bias[1] : a.bias[2])[n0 + n - m * a.wper];
        if (SPLIT == 1) b = __bfloat162float(__float2bfloat16_rn(b));
      }
      bias_ptr[n] = b;
    }
    if (TAB)
      for (uint32_t i = tid; i < 2 * Tab<EPI>::LEN; i += LG_THREADS) tab[i] = Tab<EPI>::entry(i);
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  if (s_abort != 0) {
    if (A_BF16) cp_async_wait<0>();
    __syncthreads();
    if (warp == LG_LOADERS) tmem_dealloc(tmem, 512u);
    return;
  }

  if (warp < LG_LOADERS) {
    // ------------------------------------------------------------------ loaders
    int n = 0;
    bool ok = true;
    int tile = blockIdx.x, ch = 0;
    if (tma) {
      for (n = a.nstages; warp == 0 && n < my_chunks; ++n) {
        if (!warp_wait(empty + 8 * (n % a.nstages), (uint32_t)(n / a.nstages - 1) & 1u)) break;
        if (elect_one()) tma_chunk(n);
        __syncwarp();
      }
    } else if constexpr (A_BF16) {
      // LG_DEPTH chunks of copies in flight per thread; a chunk is handed over when the thread's own copies have landed
      auto hand_over = [&](int m) {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * (m % a.nstages));
      };
      while (ld_tile < ntiles) {
        const int st = ld_n % a.nstages, use = ld_n / a.nstages;
        if (use > 0) ok = warp_wait(empty + 8 * st, (uint32_t)(use - 1) & 1u);
        if (!ok) break;
        copy_chunk();
        cp_async_wait<LG_DEPTH>();
        hand_over(ld_n - 1 - LG_DEPTH);
      }
      cp_async_wait<0>();
      if (ok)
        for (int m = max(0, ld_n - LG_DEPTH); m < ld_n; ++m) hand_over(m);
    } else
    while (ok && tile < ntiles) {
      int tile_n = tile, ch_n = ch + 1;
      if (ch_n == nchunks) {
        ch_n = 0; tile_n += G_x;
#pragma unroll
        for (int i = 0; i < R; ++i) row[i].add(a.A, step_b, step_l);
      }
      const AE* col = a_col(ch_n);
      const int st = n % a.nstages, use = n / a.nstages;
      if (use > 0) ok = warp_wait(empty + 8 * st, (uint32_t)(use - 1) & 1u);
      if (!ok) break;
      const uint32_t dst = sA + st * SPLIT * CHUNK;
#pragma unroll
      for (int i = 0; i < R; ++i) {                      // registers freed by a store take the next chunk's load
        const int r = lrow + 32 * i;
        raw_store<SPLIT, false>(cur[i], dst + r * 128 + ((lc8 ^ (r & 7)) << 4), CHUNK);
        if (!TRANSB && SPLIT == 1 && a.x_copy && blockIdx.y == 0 && tile * 128 + r < a.T && ch * 64 + lc8 * 8 < a.K) {
          uint4 w;
          w.x = pack_bf16(__uint_as_float(cur[i].w[0]), __uint_as_float(cur[i].w[1]));
          w.y = pack_bf16(__uint_as_float(cur[i].w[2]), __uint_as_float(cur[i].w[3]));
          w.z = pack_bf16(__uint_as_float(cur[i].w[4]), __uint_as_float(cur[i].w[5]));
          w.w = pack_bf16(__uint_as_float(cur[i].w[6]), __uint_as_float(cur[i].w[7]));
          *reinterpret_cast<uint4*>(a.x_copy + (size_t)(tile * 128 + r) * a.K + ch * 64 + lc8 * 8) = w;
        }
        cur[i] = load_row(col, tile_n, i);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * st);
      ++n;
      tile = tile_n; ch = ch_n;
    }
  } else if (warp == LG_LOADERS) {
    // ------------------------------------------------------------------ MMA issue
    int n = 0, j = 0;
    bool ok = true;
    // every operand descriptor is an add on one of these two
    const bool half_rows = A_BF16 && a.tma == MAP_HEADS && a.A.d == 32;       // two images of 32 features, 64-byte rows
    const uint64_t DA = half_rows ? make_smem_desc(sA, 16, 512, LAYOUT_SW64) : make_smem_desc(sA, 16, 1024, LAYOUT_SW128);
    const uint64_t DB = TRANSB ? make_smem_desc(sbase, 8192, 1024, LAYOUT_SW128) : make_smem_desc(sbase, 16, 1024, LAYOUT_SW128);
    const uint32_t idesc = make_idesc_bf16(128, nc, 0, 0);
    for (int tile = blockIdx.x; ok && tile < ntiles; tile += G_x, ++j) {
      const int buf = j & 1;
      if (j >= 2) ok = warp_wait(acc_empty + 8 * buf, (uint32_t)(j / 2 - 1) & 1u);
      for (int ch = 0; ok && ch < nchunks; ++ch, ++n) {
        const int st = n % a.nstages;
        ok = warp_wait(full + 8 * st, (uint32_t)(n / a.nstages) & 1u);
        if (!ok) break;
        if (elect_one()) {
          tc_fence_after();
          const int nk = min(4, (a.K - 64 * ch) >> 4);
          const uint64_t da = desc_advance(DA, (uint32_t)st * SPLIT * CHUNK), db = desc_advance(DB, (uint32_t)ch * bchunk);
          // fp32 mode: a sum in tensor memory is truncated at every step, so the small products have an accumulator of
          // their own and the leading ones one per chunk as far as they go (nacc == 1: one chunk, everything in one)
          const uint32_t d0 = tmem + buf * 256;
          const bool spread = SPLIT == 3 && a.nacc > 1;
          const int part = SPLIT == 1 && a.parts ? ch / a.parts : 0, ch_in = SPLIT == 1 && a.parts ? ch - part * a.parts : ch;
          const uint32_t dl = part ? d0 + part * 64u : spread ? d0 + (uint32_t)(1 + ch % (a.nacc - 1)) * (256u / a.nacc) : d0;
          const uint32_t acc_s = ch > 0, acc_l = spread ? (ch >= a.nacc - 1) : (ch_in > 0 || SPLIT == 3);
          const int groups = TRANSB ? (nc + 63) >> 6 : 1;
          for (int g = 0; g < groups; ++g) {
            const uint32_t id = TRANSB ? (64 * g + 64 <= nc ? make_idesc_bf16(128, 64, 0, 1) : make_idesc_bf16(128, 32, 0, 1)) : idesc;
#pragma unroll
            for (int pr = 0; pr < Prod<SPLIT>::N; ++pr) {
              const bool lead = pr + 1 == Prod<SPLIT>::N;
              const uint64_t pa = desc_advance(da, Prod<SPLIT>::a(pr) * CHUNK);
              const uint64_t pb = desc_advance(db, Prod<SPLIT>::b(pr) * bpart + (TRANSB ? g * 8192u : 0u));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                if (kk < nk)
                  mma_bf16((lead ? dl : d0) + (TRANSB ? g * 64u : 0u), desc_advance(pa, half_rows ? (kk >> 1) * (CHUNK / 2) + (kk & 1) * 32 : kk * 32), desc_advance(pb, TRANSB ? kk * 2048 : kk * 32),
                           id, kk > 0 ? 1u : (lead ? acc_l : (pr > 0 ? 1u : acc_s)));
            }
          }
          mma_commit(empty + 8 * st);
          if (ch + 1 == nchunks) mma_commit(acc_full + 8 * buf);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------ output rows
    const int q = warp & 3, half = (warp - LG_LOADERS - 1) >> 2;
    const int ngroups = nc >> 5;
    int j = 0;
    if (!TRANSB && a.pen) {                              // spion_expand_keypad, in the time that the first tile takes
      // unsigned: up to 2^31 - 1 of them, and the last step of a thread goes past that
      const unsigned n = (unsigned)a.T * (unsigned)a.pen_heads, all = gridDim.x * gridDim.y * 256u, len = (unsigned)a.pen_L;
      for (unsigned i = (blockIdx.y * gridDim.x + blockIdx.x) * 256u + (unsigned)(tid - 32 * (LG_LOADERS + 1)); i < n; i += all) {
        const unsigned bh = i / len;
        a.pen[i] = 1e6f * (1.0f - a.mask[bh / (unsigned)a.pen_heads * len + (i - bh * len)]);
      }
    }
    RowIt orow;
    const int ostep = G_x * 128, ostep_b = ostep / a.Y.L, ostep_l = ostep - ostep_b * a.Y.L;
    orow.init(a.Y, min(a.T - 1, (int)blockIdx.x * 128 + q * 32 + lane));
    const uint32_t obuf = outs + (uint32_t)(warp - LG_LOADERS - 1) * OWARP, hbuf = obuf + OTILE, hbar = hbars + 8 * (warp - LG_LOADERS - 1);
    const bool staged = STAGED && a.staged;
    uint32_t hpar = 0;
    bool h_due = false;                                  // a copy is on its way to hbuf
    // pre-activations of group g of a tile: staged, a copy into this warp's tile; else registers.  Rows past the last token are zeros.
    uint32_t hw[2][8];
    auto load_h = [&](int tile, int g) {
      const int t0 = tile * 128 + q * 32;
      if (tile >= ntiles || t0 >= a.T || g >= ngroups) return;
      if (staged) {
        h_due = true;
        if (lane == 0) {
          mbar_expect_tx(hbar, 2048u);
          tma_load_2d(hbuf, &maps.h, hbar, n0 + g * 32, t0);
        }
      } else {
#pragma unroll
        for (int x = 0; x < 2; ++x) ld_v8_if(t0 + lane < a.T, a.h + (size_t)(t0 + lane) * a.N + n0 + g * 32 + 16 * x, hw[x]);
      }
    };
    if (EPI == EPI_DGELU) load_h(blockIdx.x, half);
    // 32 outputs of a lane's row to the warp's tile, and from there to column c of Y's rows
    auto put = [&](uint32_t buf, const uint32_t* w, const CUtensorMap* m, int x, int y) {
      if (lane == 0) bulk_wait_read_all();               // the store before has read its tile
      __syncwarp();
#pragma unroll
      for (int p = 0; p < (Y_BF16 ? 4 : 8); ++p) {
        const uint32_t (&v)[4] = *reinterpret_cast<const uint32_t (*)[4]>(w + 4 * p);
        st_shared16(buf + (Y_BF16 ? lane * 64 + ((p ^ ((lane >> 1) & 3)) << 4) : lane * 128 + ((p ^ (lane & 7)) << 4)), v);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(m, buf, x, y);
        bulk_commit();
      }
    };
    for (int tile = blockIdx.x; tile < ntiles; tile += G_x, ++j, orow.add(a.Y, ostep_b, ostep_l)) {
      const int buf = j & 1;
      if (!warp_wait(acc_full + 8 * buf, (uint32_t)(j >> 1) & 1u)) break;
      tc_fence_after();
      const int t0 = tile * 128 + q * 32, t = t0 + lane;
      const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + buf * 256;
      bool ok = true;
      for (int g = half; g < ngroups; g += 2) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(tl + g * 32, v);
        tmem_ld_wait();
        if (SPLIT == 3) {
          for (int x = 1; x < a.nacc && x <= nchunks; ++x) {
            uint32_t u[32];
            tmem_ld32(tl + x * (256 / a.nacc) + g * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(u[i]));
          }
        }
        if (SPLIT == 1 && TRANSB && a.parts) {
          // what three separate layers would hand to their common input: each gradient rounded to bf16, added in bf16 from the
          // last layer to the first
          uint32_t u[32], w[32];
          tmem_ld32(tl + 64 + g * 32, u);
          tmem_ld32(tl + 128 + g * 32, w);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            v[i] = __float_as_uint(round_bf16(round_bf16(__uint_as_float(w[i])) + round_bf16(__uint_as_float(u[i]))) +
                                   round_bf16(__uint_as_float(v[i])));
        }
        if (g + 2 >= ngroups) {                          // this warp has read its columns of the tile
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty + 8 * buf);
        }
        if (t0 >= a.T) continue;                         // whole warps; single lanes past the end go on, what they have is not written
        const float4* bp = reinterpret_cast<const float4*>(bias_ptr + g * 32);
        float f[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 b = bp[i];
          f[4 * i] = __uint_as_float(v[4 * i]) + b.x; f[4 * i + 1] = __uint_as_float(v[4 * i + 1]) + b.y;
          f[4 * i + 2] = __uint_as_float(v[4 * i + 2]) + b.z; f[4 * i + 3] = __uint_as_float(v[4 * i + 3]) + b.w;
        }
        const int c = n0 + g * 32;
        if (EPI == EPI_DGELU) {
          if (staged) {
            if (!(ok = warp_wait(hbar, hpar))) break;
            hpar ^= 1u;
            h_due = false;
#pragma unroll
            for (int p = 0; p < 4; ++p)
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(hw[p >> 1][(p & 1) * 4]), "=r"(hw[p >> 1][(p & 1) * 4 + 1]), "=r"(hw[p >> 1][(p & 1) * 4 + 2]),
                           "=r"(hw[p >> 1][(p & 1) * 4 + 3]) : "r"(hbuf + lane * 64 + ((p ^ ((lane >> 1) & 3)) << 4)) : "memory");
            __syncwarp();
          }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            float slope[16];
            activate<EPI, TAB>(tab, hw[x], slope);
#pragma unroll
            for (int i = 0; i < 16; ++i) f[16 * x + i] = round_bf16(f[16 * x + i]) * slope[i];
          }
          if (g + 2 < ngroups) load_h(tile, g + 2);
          else load_h(tile + G_x, half);
        }
        // where the group goes: matrix, column of its rows, row (one lane's of a tile)
        const int mi = which_matrix(a.Y, c), cm = c - mi * a.Y.per, head = a.Y.L == 0x7fffffff ? 0 : cm >> a.Y.dsh;
        const int x0 = cm - head * a.Y.d, y0 = a.Y.L == 0x7fffffff ? t : (orow.b * (a.Y.per >> a.Y.dsh) + head) * a.Y.L + orow.l;
        if (Y_BF16) {
          uint32_t w[2][8];
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < 8; ++i) w[x][i] = pack_bf16(f[16 * x + 2 * i], f[16 * x + 2 * i + 1]);
          if (staged) put(obuf, w[0], maps.y + mi, x0, y0);
          __nv_bfloat16* dst = tok_col<__nv_bfloat16>(a.Y, c) + orow.off(a.Y);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            if (!staged && t < a.T) st_v8(dst + 16 * x, w[x]);
            if (EPI == EPI_GELU) {
              float act[16];
              activate<EPI, TAB>(tab, w[x], act);
#pragma unroll
              for (int i = 0; i < 8; ++i) w[x][i] = pack_bf16(act[2 * i], act[2 * i + 1]);
              if (!staged && t < a.T) st_v8(a.g + (size_t)t * a.N + c + 16 * x, w[x]);
            }
          }
          if (EPI == EPI_GELU && staged) put(hbuf, w[0], &maps.g, c, t);
        } else {
          float* dst = tok_col<float>(a.Y, c) + orow.off(a.Y);
          uint32_t w[32];
          float probe = 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) w[i] = __float_as_uint(f[i]);
          if (a.accum && t < a.T) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              uint32_t o[8];
              ld_v8(dst + 8 * x, o);
#pragma unroll
              for (int i = 0; i < 8; ++i) w[8 * x + i] = __float_as_uint(__uint_as_float(w[8 * x + i]) + __uint_as_float(o[i]));
            }
          }
          if (SPLIT == 3) {
#pragma unroll
            for (int i = 0; i < 32; ++i) probe = fmaf(__uint_as_float(w[i]), 0.f, probe);
          }
          const bool redo = SPLIT == 3 && t < a.T && !all_finite(probe);
          if (staged && !__any_sync(0xffffffffu, redo)) {
            put(obuf, w, maps.y + mi, x0, y0);
          } else if (t < a.T) {
#pragma unroll
            for (int x = 0; x < 4; ++x) st_v8(dst + 8 * x, *reinterpret_cast<const uint32_t (*)[8]>(w + 8 * x));
            if (redo) redo_outputs(a, TRANSB, t, c, dst);
          }
        }
      }
      if (!ok) break;
      if (half >= ngroups) {                             // nc == 32: the second half of the warps only hands the buffer back
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + 8 * buf);
      }
    }
    if (staged && lane == 0) bulk_wait_all();
    if (EPI == EPI_DGELU && h_due) warp_wait(hbar, hpar);             // after a wait that gave up
  }
  tc_fence_before();
  __syncthreads();
  if (warp == LG_LOADERS) tmem_dealloc(tmem, 512u);
}

// ------------------------------------------------------------------------------------------------ weight gradient
struct WgradArgs {
  TokMat dY, X;
  int T, N, K;
  int nc, kc, nstages;      // features of dY / X per CTA (blockIdx.y, blockIdx.z); nc + kc <= 256, multiples of 64 except at the end
  int nraw;                 // fp32: halves of a tile that are copied ahead; which operands through tensor maps
  bool box_y, box_x;
  float* part;              // [gridDim.x][N * K + N]
};

// Accumulators of a CTA's slice (nlen features of dY, kch chunks of X): sets of columns, two per set at lane offsets 0 and 16 where one
// needs half of the lanes (M = 64).  fp32 mode: the last one takes the small products.
struct WgradAcc {
  int cs, sets, two;
  __host__ __device__ WgradAcc(int nlen, int kch) : cs((nlen + 63) & ~63), sets(512 / cs), two(kch == 1) {}
  __host__ __device__ int total() const { return sets << two; }
  __device__ uint32_t at(int i) const { return two ? (uint32_t)(i >> 1) * cs + ((uint32_t)(i & 1) << 20) : (uint32_t)i * cs; }
};

// Loader warps: what a copy costs is its addresses, and sixteen warps share them better than eight (524288 tokens, two gradients, bf16:
// 135 -> 109 us).
constexpr int WG_LOADERS = 16;
constexpr uint32_t WCHUNK = 64 * 128;                    // [64 tokens x 64 features] bf16

// As redo_outputs: features n .. n + 31 of dY by feature k of X, over the tokens of this CTA
__device__ __noinline__ void redo_gradient(const WgradArgs& a, int n, int k, float* dst) {
  const int ntiles = (a.T + 63) >> 6;
  for (int e = 0; e < 32; ++e) {
    if (fabsf(dst[(size_t)e * a.K]) <= 3.402823466e38f) continue;
    const float *d = tok_col<const float>(a.dY, n + e), *x = tok_col<const float>(a.X, k);
    float s = 0.f;
    for (int tile = blockIdx.x; tile < ntiles && s == s; tile += gridDim.x)
      for (int t = tile * 64; t < min(a.T, tile * 64 + 64); ++t) {
        RowIt rd, rx;
        rd.init(a.dY, t);
        rx.init(a.X, t);
        s = fmaf(d[rd.off(a.dY)], x[rx.off(a.X)], s);
      }
    dst[(size_t)e * a.K] = s;
  }
}

// One CTA per SM and slice of the tokens.  dW^T accumulates in tensor memory over all tokens of the CTA: the chunks of X are one
// MN-major A operand (M = 64 or 128), those of dY one MN-major B operand (N up to 192), so nothing is transposed.  The bias gradient is summed from the registers the loaders hold.
template <bool DY_BF16, bool X_BF16>
__global__ void __launch_bounds__(32 * (WG_LOADERS + 1), 1) k_lin_wgrad(const __grid_constant__ WgradArgs a) {
  constexpr int LOADERS = WG_LOADERS, ROWS = 4 * LOADERS, XR = 64 / ROWS;       // rows of a pass of all loaders, passes per tile
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  next_may_start();                                                    // k_lin_reduce
  const uint32_t sbase = smem_u32(smem_raw);
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int n0 = blockIdx.y * a.nc, k0 = blockIdx.z * a.kc;
  const int nlen = min(a.nc, a.N - n0), klen = min(a.kc, a.K - k0);
  const int nch = (nlen + 63) >> 6, kch = (klen + 63) >> 6, cpt = nch + kch;    // chunks per tile of 64 tokens
  const uint32_t stage = (uint32_t)cpt * WCHUNK;
  const uint32_t bars = sbase + a.nstages * ((a.nc + 63) / 64 + (a.kc + 63) / 64) * WCHUNK;
  const uint32_t full = bars, empty = bars + 64, acc_done = bars + 128, slot = bars + 136, sdb = bars + 256;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  float* sdb_ptr = reinterpret_cast<float*>(smem_raw + (sdb - sbase));        // [LOADERS][256]
  const int ntiles = (a.T + 63) >> 6;
  const int G_x = (int)gridDim.x;
  __shared__ int s_abort;

  if (warp == LOADERS) {
    if (lane == 0) {
      s_abort = *reinterpret_cast<volatile int*>(&g_lin_status);
      for (int i = 0; i < a.nstages; ++i) { mbar_init(full + 8 * i, LOADERS); mbar_init(empty + 8 * i, 1); }
      mbar_init(acc_done, 1);
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(slot, 512u);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  if (s_abort != 0) {
    __syncthreads();
    if (warp == LOADERS) tmem_dealloc(tmem, 512u);
    return;
  }

  if (warp < LOADERS) {
    const int lrow = tid >> 3, lc8 = tid & 7;
    // chunk i of a tile: features i of dY for i < nch, then those of X.  fp32 chunks pass through registers (a tile ahead),
    // bf16 ones are copied straight into their stage (AHEAD tiles ahead).
    Raw<false> cur[4][XR];
    constexpr int AHEAD = (DY_BF16 || X_BF16) ? 2 : 0;
    float db[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) db[i][e] = 0.f;
    using DE = typename std::conditional<DY_BF16, __nv_bfloat16, float>::type;
    using XE = typename std::conditional<X_BF16, __nv_bfloat16, float>::type;
    const DE* dcol[4];                                     // this thread's eight features of every chunk, null past the end
    const XE* xcol[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int cd = n0 + i * 64 + lc8 * 8, cx = k0 + (i - nch) * 64 + lc8 * 8;
      dcol[i] = i < nch && cd < n0 + nlen ? tok_col<const DE>(a.dY, cd) : nullptr;
      xcol[i] = i >= nch && i < cpt && cx < k0 + klen ? tok_col<const XE>(a.X, cx) : nullptr;
    }
    const int step = G_x * 64;
    const int dstep_b = step / a.dY.L, dstep_l = step - dstep_b * a.dY.L, xstep_b = step / a.X.L, xstep_l = step - xstep_b * a.X.L;
    RowIt drow[XR], xrow[XR];                                // rows of the tile whose loads are issued next
    auto row_init = [&](int t0) {
#pragma unroll
      for (int x = 0; x < XR; ++x) {
        drow[x].init(a.dY, min(a.T - 1, t0 + lrow + ROWS * x));
        xrow[x].init(a.X, min(a.T - 1, t0 + lrow + ROWS * x));
      }
    };
    // fp32 chunks of the tile the row iterators stand at -> registers
    auto load_row = [&](int tile, int i, int x) {
      const bool isd = !DY_BF16 && (X_BF16 || i < nch);
      const void* p = isd ? (const void*)(dcol[i] + drow[x].off(a.dY)) : (const void*)(xcol[i] + xrow[x].off(a.X));
      const bool in = (isd ? dcol[i] != nullptr : xcol[i] != nullptr) && tile * 64 + lrow + ROWS * x < a.T;
      ld_v8_if(in, p, cur[i][x].w);
    };
    // bf16 chunks of the current tile -> shared memory
    auto copy_row = [&](int tile, int i, int x, uint32_t dst) {
      const bool tin = tile * 64 + lrow + ROWS * x < a.T;
      if (i < nch) {
        const bool in = tin && dcol[i];
        cp_async16(dst, in ? dcol[i] + drow[x].off(a.dY) : reinterpret_cast<const DE*>(a.dY.p[0]), in);
      } else {
        const bool in = tin && xcol[i];
        cp_async16(dst, in ? xcol[i] + xrow[x].off(a.X) : reinterpret_cast<const XE*>(a.X.p[0]), in);
      }
    };
    auto place = [&](int st, int i, int x) -> uint32_t {
      const int r = lrow + ROWS * x;
      return sbase + st * stage + i * WCHUNK + r * 128 + ((lc8 ^ (r & 7)) << 4);
    };
    bool ok = true;
    int n = 0;
    // this thread's share of tile m is complete: column sums of its bf16 dY pieces, then the hand-over
    auto hand_over = [&](int m) {
      const int st = m % a.nstages;
      if (DY_BF16) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i < nch) {
#pragma unroll
            for (int x = 0; x < XR; ++x) {
              uint32_t w[4];
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(place(st, i, x)) : "memory");
#pragma unroll
              for (int e = 0; e < 4; ++e) { db[i][2 * e] += bf16_lo(w[e]); db[i][2 * e + 1] += bf16_hi(w[e]); }
            }
          }
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * st);
    };
    row_init((int)blockIdx.x * 64);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int x = 0; x < XR; ++x) load_row(blockIdx.x, i, x);
    for (int tile = blockIdx.x; ok && tile < ntiles; tile += G_x, ++n) {
      const int st = n % a.nstages, use = n / a.nstages;
      if (use > 0) ok = warp_wait(empty + 8 * st, (uint32_t)(use - 1) & 1u);
      if (!ok) break;
      if (DY_BF16 || X_BF16) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int x = 0; x < XR; ++x)
            if (i < cpt && (i < nch ? DY_BF16 : X_BF16)) copy_row(tile, i, x, place(st, i, x));
      }
#pragma unroll
      for (int x = 0; x < XR; ++x) { drow[x].add(a.dY, dstep_b, dstep_l); xrow[x].add(a.X, xstep_b, xstep_l); }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < cpt && !(i < nch ? DY_BF16 : X_BF16)) {
#pragma unroll
          for (int x = 0; x < XR; ++x) {
            raw_store<1, false>(cur[i][x], place(st, i, x), WCHUNK);
            if (i < nch) {
#pragma unroll
              for (int e = 0; e < 8; ++e) db[i][e] += __uint_as_float(cur[i][x].w[e]);
            }
            load_row(tile + G_x, i, x);
          }
        }
      }
      if (AHEAD > 0) {
        cp_async_commit();
        if (n >= AHEAD) { cp_async_wait<AHEAD>(); hand_over(n - AHEAD); }
      } else {
        hand_over(n);
      }
    }
    if (AHEAD > 0) {
      cp_async_wait<0>();
      if (ok)
        for (int m = max(0, n - AHEAD); m < n; ++m) hand_over(m);
    }
    // column sums of dY: lanes with the same lc8 of a warp, then the warps in order
    if (blockIdx.z == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < nch) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float s = db[i][e];
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (lane < 8) sdb_ptr[warp * 256 + i * 64 + lane * 8 + e] = s;
          }
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * LOADERS) : "memory");       // the loader warps
    float* part = a.part + (size_t)blockIdx.x * ((size_t)a.N * a.K + a.N);
    if (blockIdx.z == 0 && tid < nlen) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < LOADERS; ++w) s += sdb_ptr[w * 256 + tid];
      part[(size_t)a.N * a.K + n0 + tid] = s;
    }
    if (ok) ok = warp_wait(acc_done, 0u);
    if (ok) {
      tc_fence_after();
      const int q = warp & 3, half = warp >> 2;
      const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16);
      const int m = kch == 1 ? q * 16 + (lane & 15) : q * 32 + lane;           // feature of X
      const bool min_ = (kch == 2 || lane < 16) && m < klen;
      for (int g = half; g < (nlen >> 5); g += LOADERS / 4) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(tl + g * 32, v);
        tmem_ld_wait();
        if (min_) {
          float* dst = part + (size_t)(n0 + g * 32) * a.K + k0 + m;
#pragma unroll
          for (int e = 0; e < 32; ++e) dst[(size_t)e * a.K] = __uint_as_float(v[e]);
        }
      }
    }
  } else {
    bool ok = true;
    int n = 0;
    // D[features of X, features of dY]: both operands MN-major, chunks of 64 features WCHUNK apart
    const uint32_t idesc = make_idesc_bf16(kch == 1 ? 64 : 128, nlen, 1, 1);
    const uint64_t D0 = make_smem_desc(sbase, WCHUNK, 1024, LAYOUT_SW128);
    for (int tile = blockIdx.x; ok && tile < ntiles; tile += G_x, ++n) {
      const int st = n % a.nstages;
      ok = warp_wait(full + 8 * st, (uint32_t)(n / a.nstages) & 1u);
      if (!ok) break;
      if (elect_one()) {
        tc_fence_after();
        const uint64_t dd = desc_advance(D0, st * stage), dx = desc_advance(dd, (uint32_t)nch * WCHUNK);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_bf16(tmem, desc_advance(dx, kk * 2048), desc_advance(dd, kk * 2048), idesc, kk > 0 || n > 0);
        mma_commit(empty + 8 * st);
        if (tile + G_x >= ntiles) mma_commit(acc_done);
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == LOADERS) tmem_dealloc(tmem, 512u);
}

// The same for fp32 operands: both in three bf16 parts, six products.  Half a tile (32 tokens) at a time:
//   warp 17       copies the rows of both operands as they lie in memory (tensor maps, boxes of 32 or 64 features) into a ring of `nraw` halves, a
//                 lane one box of every half: with the addresses formed half by half, or a copy per row, this warp was the limit (64, 236 us)
//   warps 0-15    two groups of eight take halves in turn: sixteen bytes twice per lane and chunk, split, three images
//   warp 16       the products
// Loads through registers kept 64 KB per SM in flight, but a load that waits for room in what shared memory leaves of the L1 cache keeps the
// stores behind it waiting too: three 16-byte stores of a lane took 450 cycles, 60 without the loads, the split itself 5 % of the kernel.
// 262144 tokens, 64 x 192 97 us -> 60, 64 x 64 50 -> 41; 15040 tokens, 192 x 576 39 either way.
constexpr uint32_t HCHUNK = 32 * 128, HRAW = 32 * 256;   // 32 tokens x 64 features: one bf16 image, fp32
// features of a copy: 64 where heads (rows) are whole multiples of that, else 32
__device__ __forceinline__ int copy_width(const TokMat& m) { return (m.d & 63) == 0 ? 64 : 32; }
// What a lane of warp 17 copies of every half: one box of an operand, or, where a half may span two sequences, one row of all boxes
struct HalfCopy {
  const CUtensorMap* map;
  int x, hl, bl;            // column; rows of the map per head of this box, per sequence
  uint32_t dst;
  bool on;
};
__device__ __forceinline__ HalfCopy half_copy(const TokMat& m, const CUtensorMap* maps, int c, int f, int end, uint32_t chunk) {
  const int w = copy_width(m);
  HalfCopy h;
  h.on = c + f < end && f % w == 0;
  h.dst = chunk + (uint32_t)(f / w) * 32u * (uint32_t)(4 * w);
  c += f;
  const int i = h.on ? which_matrix(m, c) : 0;
  c -= i * m.per;
  h.map = maps + i;
  const bool heads = m.L != 0x7fffffff;
  const int head = heads ? c >> m.dsh : 0;
  h.x = c - head * m.d;
  h.hl = heads ? head * m.L : 0;
  h.bl = heads ? (m.per >> m.dsh) * m.L : 0;
  return h;
}
// rows of a half that may span two sequences: lane = token
__device__ __forceinline__ void copy_rows(const TokMat& m, int c, int end, int t, int rows, uint32_t dst, uint32_t bar, int lane) {
  const int w = copy_width(m);
  RowIt r;
  r.init(m, min(t + lane, t + rows - 1));
  for (int f = 0; f < 64 && c + f < end; f += w)
    if (lane < rows)
      bulk_load(dst + (uint32_t)(f / w) * 32u * (uint32_t)(4 * w) + lane * 4 * w, tok_col<const float>(m, c + f) + r.off(m), bar, (uint32_t)(4 * w));
}
// Eight features of one token of a copied chunk.  Lanes of the upper features read their second half first (no two lanes on the same banks).
__device__ __forceinline__ uint32_t half_at(int width, int row, int lc8) {
  return width == 64 ? row * 256 + lc8 * 32 : (lc8 >> 2) * 4096 + row * 128 + (lc8 & 3) * 32;
}
__device__ __forceinline__ void read_half(uint32_t at, bool upper, uint32_t (&v)[8]) {
  uint32_t p[4], q[4];
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(p[0]), "=r"(p[1]), "=r"(p[2]), "=r"(p[3]) : "r"(at + (upper ? 16u : 0u)) : "memory");
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(at + (upper ? 0u : 16u)) : "memory");
#pragma unroll
  for (int e = 0; e < 4; ++e) { v[e] = upper ? q[e] : p[e]; v[4 + e] = upper ? p[e] : q[e]; }
}

struct WgradMaps { CUtensorMap y[3], x[3]; };
__global__ void __launch_bounds__(32 * (WG_LOADERS + 2), 1) k_lin_wgrad_fp32(const __grid_constant__ WgradArgs a, const __grid_constant__ WgradMaps maps) {
  constexpr int LOADERS = WG_LOADERS;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  next_may_start();                                                    // k_lin_reduce
  const uint32_t sbase = smem_u32(smem_raw);
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int n0 = blockIdx.y * a.nc, k0 = blockIdx.z * a.kc;
  const int nlen = min(a.nc, a.N - n0), klen = min(a.kc, a.K - k0);
  const int nch = (nlen + 63) >> 6, kch = (klen + 63) >> 6, cpt = nch + kch;
  const int most = (a.nc + 63) / 64 + (a.kc + 63) / 64;
  const uint32_t stage = (uint32_t)cpt * 3 * HCHUNK;
  const uint32_t raws = sbase + a.nstages * most * 3 * HCHUNK, rawb = (uint32_t)cpt * HRAW;
  const uint32_t bars = raws + a.nraw * most * HRAW;
  const uint32_t full = bars, empty = bars + 64, raw_full = bars + 128, raw_free = bars + 192, acc_done = bars + 256, slot = bars + 264;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  float* sdb_ptr = reinterpret_cast<float*>(smem_raw + (raws - sbase));       // [LOADERS][256], when all halves have been read
  const int ntiles = (a.T + 63) >> 6, G_x = (int)gridDim.x;
  const int my_tiles = (ntiles - (int)blockIdx.x + G_x - 1) / G_x;
  // the last tile of all may have one half only
  const int halves = 2 * my_tiles - ((ntiles - 1) % G_x == (int)blockIdx.x && a.T - (ntiles - 1) * 64 <= 32 ? 1 : 0);
  __shared__ int s_abort;

  if (warp == LOADERS) {
    if (lane == 0) {
      s_abort = *reinterpret_cast<volatile int*>(&g_lin_status);
      for (int i = 0; i < a.nstages; ++i) { mbar_init(full + 8 * i, 8); mbar_init(empty + 8 * i, 1); }
      for (int i = 0; i < a.nraw; ++i) { mbar_init(raw_full + 8 * i, 1); mbar_init(raw_free + 8 * i, 8); }
      mbar_init(acc_done, 1);
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(slot, 512u);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  if (s_abort != 0) {
    __syncthreads();
    if (warp == LOADERS) tmem_dealloc(tmem, 512u);
    return;
  }
  auto first_token = [&](int n) { return ((int)blockIdx.x + (n >> 1) * G_x) * 64 + (n & 1) * 32; };

  // Half n is in raw slot n % nraw and stage n % nstages.  A parity tells two phases apart: at a wait the phase before must be over and the one after
  // must not be.  raw_free, full: one waiter (warp 17, warp 16) for every phase.  raw_full: nraw is even, so a slot's phases are all one group's.
  // empty, three stages: a group waits for the products of half n - 3, the phase before is that of half n - 6; it has waited for those of half
  // n - 5, which were issued later.  The next phase needs what the waiter does after its wait.
  if (warp == LOADERS + 1) {
    const bool by = a.box_y, bx = a.box_x;
    const int u = lane >> 1, f = (lane & 1) * 32;          // this lane's box: chunk and half of it
    const bool isd = u < nch;
    HalfCopy h = isd ? half_copy(a.dY, maps.y, n0 + 64 * u, f, n0 + nlen, u * HRAW) : half_copy(a.X, maps.x, k0 + 64 * (u - nch), f, k0 + klen, u * HRAW);
    h.on = h.on && u < cpt && (isd ? by : bx);
    const TokMat& mine = isd ? a.dY : a.X;
    RowIt at;
    at.init(mine, min((int)blockIdx.x * 64, a.T - 1));
    const int far = 64 * G_x - 32, far_b = far / mine.L, far_l = far - far_b * mine.L;
    int n = 0, s = 0;
    uint32_t round = 0;
    for (; n < halves; ++n) {
      if (round > 0 && !warp_wait(raw_free + 8 * s, (round - 1) & 1u)) break;
      const int t = first_token(n), rows = min(32, a.T - t);
      const uint32_t bar = raw_full + 8 * s, dst = raws + s * rawb;
      if (lane == 0) mbar_expect_tx(bar, (uint32_t)((by ? 32 : rows) * nlen + (bx ? 32 : rows) * klen) * 4u);
      __syncwarp();
      if (h.on) tma_load_2d(dst + h.dst, h.map, bar, h.x, at.b * h.bl + h.hl + at.l);
      if (!by) for (int i = 0; i < nch; ++i) copy_rows(a.dY, n0 + 64 * i, n0 + nlen, t, rows, dst + i * HRAW, bar, lane);
      if (!bx) for (int i = 0; i < kch; ++i) copy_rows(a.X, k0 + 64 * i, k0 + klen, t, rows, dst + (nch + i) * HRAW, bar, lane);
      if (n & 1) at.add(mine, far_b, far_l);
      else at.add(mine, 0, 32);
      if (++s == a.nraw) { s = 0; ++round; }
    }
    // after a wait that gave up: nothing is on its way to this CTA's shared memory when it leaves
    for (int m = max(0, n - a.nraw); n < halves && m < n; ++m) warp_wait(raw_full + 8 * (m % a.nraw), (uint32_t)(m / a.nraw) & 1u);
  } else if (warp < LOADERS) {
    const int group = warp >> 3, lrow = (tid & 255) >> 3, lc8 = tid & 7;
    const bool upper = lc8 >= 4;
    uint32_t from[4];                                      // this thread's eight features of every chunk of a slot
    bool some[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      from[i] = raws + i * HRAW + half_at(copy_width(i < nch ? a.dY : a.X), lrow, lc8);
      some[i] = lc8 * 8 < (i < nch ? nlen - 64 * i : klen - 64 * (i - nch));
    }
    const uint32_t to = sbase + lrow * 128 + ((lc8 ^ (lrow & 7)) << 4);
    float db[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) db[i][e] = 0.f;
    bool ok = true;
    int s = group, st = group;                             // slot and stage of the half, how often they have been used before
    uint32_t s_use = 0, st_use = 0;
    for (int n = group; n < halves; n += 2) {
      ok = warp_wait(raw_full + 8 * s, s_use & 1u);
      if (!ok) break;
      const bool in = first_token(n) + lrow < a.T;
      Raw<false> r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < cpt) read_half(from[i] + s * rawb, upper, r[i].w);
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_free + 8 * s);
      if (st_use > 0) ok = warp_wait(empty + 8 * st, (st_use - 1) & 1u);
      if (!ok) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < cpt) {
          if (!in || !some[i])                             // past the last token or feature: what the ring held before
#pragma unroll
            for (int e = 0; e < 8; ++e) r[i].w[e] = 0u;
          raw_store<3, false>(r[i], to + st * stage + i * 3 * HCHUNK, HCHUNK);
          if (i < nch)
#pragma unroll
            for (int e = 0; e < 8; ++e) db[i][e] += __uint_as_float(r[i].w[e]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * st);
      if ((s += 2) >= a.nraw) { s -= a.nraw; ++s_use; }
      if ((st += 2) >= a.nstages) { st -= a.nstages; ++st_use; }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * LOADERS) : "memory");       // the loader warps
    // column sums of dY: lanes with the same lc8 of a warp, then the warps in order
    if (blockIdx.z == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < nch) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float s = db[i][e];
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (lane < 8) sdb_ptr[warp * 256 + i * 64 + lane * 8 + e] = s;
          }
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * LOADERS) : "memory");
    float* part = a.part + (size_t)blockIdx.x * ((size_t)a.N * a.K + a.N);
    if (blockIdx.z == 0 && tid < nlen) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < LOADERS; ++w) s += sdb_ptr[w * 256 + tid];
      part[(size_t)a.N * a.K + n0 + tid] = s;
    }
    if (ok) ok = warp_wait(acc_done, 0u);
    if (ok) {
      tc_fence_after();
      const int q = warp & 3, half = warp >> 2;
      const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16);
      const WgradAcc acc(nlen, kch);
      const int small = acc.total() - 1, used = min(small, my_tiles);          // leading ones that were used
      const int m = kch == 1 ? q * 16 + (lane & 15) : q * 32 + lane;           // feature of X
      const bool min_ = (kch == 2 || lane < 16) && m < klen;
      for (int g = half; g < (nlen >> 5); g += LOADERS / 4) {
        uint32_t v[32];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = 0u;
        for (int s = 0; s < acc.sets; ++s) {
          const int i = acc.two ? 2 * s + (lane >> 4) : s;                     // the accumulator in this lane
          if ((acc.two ? 2 * s : s) >= used && s + 1 < acc.sets) continue;     // none of the set was used
          uint32_t u[32];
          tmem_ld32(tl + s * acc.cs + g * 32, u);
          tmem_ld_wait();
          const bool in = i < used || i == small;
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = in ? __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(u[e])) : v[e];
        }
        if (acc.two) {
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(__shfl_xor_sync(0xffffffffu, v[e], 16)));
        }
        if (min_) {
          float* dst = part + (size_t)(n0 + g * 32) * a.K + k0 + m;
          float probe = 0.f;
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            dst[(size_t)e * a.K] = __uint_as_float(v[e]);
            probe = fmaf(__uint_as_float(v[e]), 0.f, probe);
          }
          if (!all_finite(probe)) redo_gradient(a, n0 + g * 32, k0 + m, dst);
        }
      }
    }
  } else {
    bool ok = true;
    // D[features of X, features of dY]: both operands MN-major, chunks of 64 features three images apart
    const uint32_t idesc = make_idesc_bf16(kch == 1 ? 64 : 128, nlen, 1, 1);
    const uint64_t D0 = make_smem_desc(sbase, 3 * HCHUNK, 1024, LAYOUT_SW128);
    const WgradAcc acc(nlen, kch);
    const int leads = acc.total() - 1;
    int li = 0, st = 0;                                    // leading accumulator of the tile; stage of the half
    uint32_t st_use = 0;
    for (int n = 0; ok && n < halves; ++n) {
      ok = warp_wait(full + 8 * st, st_use & 1u);
      if (!ok) break;
      if (elect_one()) {
        tc_fence_after();
        const uint64_t dd = desc_advance(D0, st * stage), dx = desc_advance(dd, (uint32_t)nch * 3 * HCHUNK);
        const uint32_t lead_set = tmem + acc.at(li), small_set = tmem + acc.at(leads);
        const uint32_t acc_l = (n & 1) || (n >> 1) >= leads, acc_s = n > 0;
#pragma unroll
        for (int pr = 0; pr < Prod<3>::N; ++pr) {
          const bool lead = pr + 1 == Prod<3>::N;
#pragma unroll
          for (int kk = 0; kk < 2; ++kk)
            mma_bf16(lead ? lead_set : small_set, desc_advance(dx, Prod<3>::b(pr) * HCHUNK + kk * 2048),
                     desc_advance(dd, Prod<3>::a(pr) * HCHUNK + kk * 2048), idesc, kk > 0 ? 1u : (lead ? acc_l : (pr > 0 ? 1u : acc_s)));
        }
        mma_commit(empty + 8 * st);
        if (n + 1 == halves) mma_commit(acc_done);
      }
      __syncwarp();
      if (n & 1) li = li + 1 < leads ? li + 1 : 0;
      if (++st == a.nstages) { st = 0; ++st_use; }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == LOADERS) tmem_dealloc(tmem, 512u);
}

// out[i] = sum over the CTAs' partial results, in a fixed order: 32 groups of four values x 8 slices of the CTAs per block
__global__ void __launch_bounds__(256) k_lin_reduce(const float* part, int nparts, long long n, long long nw,
                                                    float* __restrict__ dW, float* __restrict__ db) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long i = ((long long)blockIdx.x * 32 + lane) * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  wait_for_kernel_before();
  if (i < n) {
    const int per = (nparts + 7) / 8, b0 = w * per, b1 = min(nparts, b0 + per);
#pragma unroll 10
    for (int b = b0; b < b1; ++b) {
      const float4 v = *reinterpret_cast<const float4*>(part + (size_t)b * n + i);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
  __shared__ float4 sm[8][32];
  sm[w][lane] = s;
  __syncthreads();
  if (w == 0 && i < n) {
    for (int x = 1; x < 8; ++x) { s.x += sm[x][lane].x; s.y += sm[x][lane].y; s.z += sm[x][lane].z; s.w += sm[x][lane].w; }
    float* dst = i < nw ? dW + i : db + (i - nw);         // both lengths are multiples of four
    *reinterpret_cast<float4*>(dst) = s;
  }
}

// ------------------------------------------------------------------------------------------------ host
constexpr size_t SMEM_MAX = 227 * 1024 - 1024;

TokMat to_mat(const spion_tokens* t) {
  TokMat m;
  for (int i = 0; i < 3; ++i) m.p[i] = t->ptr[i];
  m.per = t->cols;
  if (t->heads > 0) {
    m.d = t->head_dim; m.L = t->seq_len;
    m.dsh = 0;
    while ((1 << m.dsh) < m.d) ++m.dsh;
    m.hstride = (long long)m.L * m.d; m.bstride = m.hstride * t->heads;
  } else {
    m.d = t->cols; m.L = 0x7fffffff; m.dsh = 31; m.hstride = 0; m.bstride = 0;
  }
  return m;
}
bool mat_ok(const spion_tokens* t) {
  if (!t || t->count < 1 || t->count > 3 || t->cols < 32 || t->cols % 32) return false;
  if (t->heads > 0 && (t->head_dim < 32 || (t->head_dim & (t->head_dim - 1)) || t->heads * t->head_dim != t->cols || t->seq_len < 1))
    return false;
  for (int i = 0; i < t->count; ++i)
    if (!t->ptr[i] || ((uintptr_t)t->ptr[i] & 31)) return false;
  return true;
}

// The form in which bf16 tokens are read through tensor maps (MAP_NONE: the kernels copy by themselves).  With one tile per CTA
// the copies are no limit, and making the maps costs the host a microsecond (inference of 1024 tokens: 45.6 us, 46.8 with maps).
int map_form(const spion_tokens* t, long long T) {
  if (!t->is_bf16 || (T + 127) / 128 <= sm_count()) return MAP_NONE;
  if (t->heads <= 0) return t->cols >= 64 && (t->count == 1 || t->cols % 64 == 0) ? MAP_ROWS : MAP_NONE;
  return (t->head_dim == 32 || t->head_dim == 64) && t->cols % 64 == 0 && t->seq_len % 64 == 0 && T % t->seq_len == 0 &&
         T * t->heads <= 0x7fffffffLL ? MAP_HEADS : MAP_NONE;
}
int encoder(TcState* s) {
  static std::atomic<void*> encode{nullptr};
  void* fn = encode.load(std::memory_order_acquire);
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    SPION_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !fn) return SPION_ERR_CUDA;
    encode.store(fn, std::memory_order_release);
  }
  int dev = 0;                                           // a thread whose first call this is has no current context, and encoding wants one
  SPION_CUDA_TRY(cudaGetDevice(&dev));
  SPION_CUDA_TRY(cudaSetDevice(dev));
  s->encode = (EncodeTiledFn)fn;
  return SPION_OK;
}
int token_maps(const spion_tokens* t, long long T, CUtensorMap* m) {
  TcState s;
  int rc = encoder(&s);
  if (rc) return rc;
  for (int i = 0; i < t->count; ++i) {
    rc = t->heads > 0 ? make_map(&s, m + i, t->ptr[i], (uint64_t)T * t->heads, (uint32_t)t->head_dim, (uint32_t)t->head_dim, 64)
                                : make_map(&s, m + i, t->ptr[i], (uint64_t)T, (uint32_t)t->cols, 64, 128);
    if (rc) return rc;
  }
  return SPION_OK;
}

// fp32 operands of the weight gradient: boxes of 32 tokens, 64 features where heads (rows) are whole multiples of that, else 32
bool half_boxes(const spion_tokens* t, long long T) {
  return t->heads <= 0 || (t->seq_len % 32 == 0 && T % t->seq_len == 0 && T * t->heads <= 0x7fffffffLL);
}
int half_maps(const spion_tokens* t, long long T, CUtensorMap* m) {
  TcState s;
  const int rc = encoder(&s);
  if (rc) return rc;
  const uint32_t width = (uint32_t)(t->heads > 0 ? t->head_dim : t->cols);
  const cuuint64_t dims[2] = {width, (cuuint64_t)T * (t->heads > 0 ? t->heads : 1)}, strides[1] = {(cuuint64_t)width * 4};
  const cuuint32_t box[2] = {width % 64 == 0 ? 64u : 32u, 32u}, estr[2] = {1, 1};
  for (int i = 0; i < t->count; ++i)
    if (s.encode(m + i, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, t->ptr[i], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return SPION_ERR_CUDA;
  return SPION_OK;
}

// tiles of 32 tokens by 32 features of the outputs; worth their maps when a CTA has more than one tile (half a microsecond of host time each)
// Not where bf16 operands split into heads of 32 come through maps: their boxes of 64-byte rows are what the copy engine is busy with (524288
// tokens, gradient of the input from three gradients 63.5 us, 67.4 staged; output projection 27.0, 27.4, its gradient 25.2, 25.7).
bool staged_outputs(const spion_tokens* in, const spion_tokens* out, long long T) {
  auto narrow = [](const spion_tokens* t) { return t->is_bf16 && t->heads > 0 && t->head_dim == 32; };
  return (T + 127) / 128 > sm_count() && half_boxes(out, T) && !narrow(in) && !(in->is_bf16 && narrow(out));
}
size_t staged_bytes(bool gelu, bool y_bf16) { return 8 * (size_t)(gelu ? 2 : 1) * (y_bf16 ? 2048 : 4096); }
int output_maps(const spion_tokens* t, const GemmArgs& a, LinMaps& maps) {
  TcState s;
  int rc = encoder(&s);
  if (rc) return rc;
  auto one = [&](CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, bool bf16) -> int {
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * (bf16 ? 2u : 4u)};
    const cuuint32_t box[2] = {32u, 32u}, estr[2] = {1, 1};
    return s.encode(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, bf16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? SPION_OK : SPION_ERR_CUDA;
  };
  for (int i = 0; i < t->count && !rc; ++i)
    rc = one(maps.y + i, t->ptr[i], (uint64_t)a.T * (t->heads > 0 ? t->heads : 1), (uint64_t)(t->heads > 0 ? t->head_dim : t->cols), t->is_bf16);
  if (!rc && a.g) rc = one(&maps.g, a.g, (uint64_t)a.T, (uint64_t)a.N, true);
  if (!rc && a.h) rc = one(&maps.h, a.h, (uint64_t)a.T, (uint64_t)a.N, true);
  return rc;
}

// columns per CTA, accumulators and ring stages of the GEMM; false when the weights do not fit
bool plan_gemm(int split, bool trans, int K, int N, int* nc, int* nacc, int* stages, size_t* smem, int widest = 256, size_t table = 0, size_t outs = 0) {
  const int least = split == 1 ? LG_DEPTH + 1 : 2;           // bf16 operands keep LG_DEPTH chunks in flight
  const int nchunks = (K + 63) / 64;
  const int most = split == 3 && nchunks > 1 ? 64 : widest;     // several accumulators of 64 columns keep the fp32 chains short
  for (int parts = 1; parts <= 64; ++parts) {
    int c = ((N + parts - 1) / parts + 31) / 32 * 32;
    if (parts > 1 && trans) c = (c + 63) / 64 * 64;
    if (c > most) continue;
    const size_t bchunk = trans ? (size_t)((c + 63) / 64) * 8192 : (size_t)c * 128;
    const size_t b = split * ((nchunks * bchunk + 1023) / 1024 * 1024);
    for (int st = split == 1 ? 8 : 4; st >= least; --st) {
      const size_t total = b + (size_t)st * split * CHUNK + 1024 + 256 + (outs ? (table + 1023) / 1024 * 1024 + 1024 + outs : table);
      if (total <= SMEM_MAX) { *nc = c; *nacc = split == 3 && nchunks > 1 ? 4 : 1; *stages = st; *smem = total; return true; }
    }
    if (c <= 64) break;
  }
  return false;
}

// The table of the activation and the tiles of the outputs take shared memory from the weights: fewer columns per CTA, so that A is fetched once more
// for every further slice of them.  `worth`: values of A per token that may be fetched again for the cheaper epilogue (FREE: any number).  65536 and 200000
// tokens, widths of 32 to 1024, time with both ÷ without where the columns get fewer:
//   fp32 0.68 - 0.88, derivative of GELU 0.40 - 0.77
//   GELU: bf16 tokens 0.57 - 0.85 up to 384 features, 0.85 - 1.45 from 512 on (the table alone, where that leaves the columns, 0.75 - 0.97);
//         fp32 tokens 0.70 - 0.88 at 256 features, 0.83 - 1.15 at 320 and 384, 0.95 - 1.48 from 512 on
//   fp32 gradients of bf16 ones: up to one value of A for every output 0.75 - 1.0 (320 features), 0.85 - 1.09 (384; 0.91 at most up to 3 / 4); beyond 1.0 - 1.5
//   else, bf16 outputs: forward 0.91 - 1.01 up to half a value at 256 features, 0.98 - 1.6 else; gradients 0.96 - 1.54
// 65536 tokens, bf16, us, before there were tiles, always with both, now: 512 x 512 57, 78, 57; 768 x 768 143, 202, 142; gradient of 512 x 512 75, 105, 75; GELU
// of 768 x 768 170, 213, 175.
constexpr long long FREE = 1LL << 40;
template <class PLAN>
bool choose_epilogue(GemmArgs& a, int epi, bool stage, size_t outs, long long worth, PLAN plan) {
  const size_t table = epi == EPI_GELU ? Tab<EPI_GELU>::BYTES : epi == EPI_DGELU ? Tab<EPI_DGELU>::BYTES : 0;
  auto slices = [&]() { return (long long)((a.N + a.nc - 1) / a.nc); };
  a.table = a.staged = 0;
  if (!plan(0, 0)) return false;
  const long long fewest = slices();
  const bool options[3][2] = {{true, true}, {true, false}, {false, true}};       // (the kernels that form the activation have no tiles)
  for (const auto& [t, o] : options) {
    if ((t && !table) || (o && !stage) || (o && !t && table) || !plan(t ? table : 0, o ? outs : 0) || (slices() - fewest) * a.K > worth) continue;
    a.table = t;
    a.staged = o;
    return true;
  }
  return plan(0, 0);
}

// Shared-memory opt-in of a kernel, once per device; the call also loads the kernel.  `done` belongs to the kernel.
template <class K>
int opt_in(K k, std::atomic<bool> (&done)[64]) {
  int dev = 0;
  SPION_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return SPION_OK;
  SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
  if (dev < 64) done[dev].store(true, std::memory_order_release);
  return SPION_OK;
}
// fp32: a kernel for staged outputs and one without, which small calls take (a tile per CTA: the code of both in one kernel costs them 0.3 of
// 8 us: a training step of 6144 fp32 tokens 472 -> 467)
template <int SPLIT, bool A_BF16, bool TRANSB, int EPI, bool Y_BF16, bool STAGED = true, bool TAB = EPI != EPI_NONE>
int prepare_gemm() {
  static std::atomic<bool> done[64];
  return opt_in(k_lin_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16, STAGED, TAB>, done);
}
template <bool DY_BF16, bool X_BF16>
int prepare_wgrad() {
  static std::atomic<bool> done[64];
  return opt_in(k_lin_wgrad<DY_BF16, X_BF16>, done);
}
int prepare_wgrad_fp32() {
  static std::atomic<bool> done[64];
  return opt_in(k_lin_wgrad_fp32, done);
}

template <int SPLIT, bool A_BF16, bool TRANSB, int EPI, bool Y_BF16>
int launch_gemm(GemmArgs& a, const spion_tokens* tok, const spion_tokens* out, size_t smem, cudaStream_t st) {
  constexpr bool TAB = EPI != EPI_NONE;
  const bool plain = SPLIT == 3 && !a.staged, functions = TAB && !a.table;
  auto k = plain ? k_lin_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16, SPLIT != 3, TAB>
                 : functions ? k_lin_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16, EPI == EPI_NONE, false> : k_lin_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16, true, TAB>;
  int rc = plain ? prepare_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16, SPLIT != 3>()
                 : functions ? prepare_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16, EPI == EPI_NONE, false>() : prepare_gemm<SPLIT, A_BF16, TRANSB, EPI, Y_BF16>();
  if (rc) return rc;
  LinMaps maps;
  a.tma = A_BF16 ? map_form(tok, a.T) : MAP_NONE;
  if (a.tma && (rc = token_maps(tok, a.T, maps.m))) return rc;
  if (a.staged && (rc = output_maps(out, a, maps))) return rc;
  const int ny = (a.N + a.nc - 1) / a.nc;
  const int sms = sm_count(), tiles = (a.T + 127) / 128;
  if (sms < 1) return SPION_ERR_CUDA;
  int gx = sms / ny > 0 ? sms / ny : 1;
  if (gx > tiles) gx = tiles;
  k<<<dim3(gx, ny), LG_THREADS, smem, st>>>(a, maps);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

template <bool DY_BF16, bool X_BF16>
int launch_wgrad(const WgradArgs& a, int gx, size_t smem, cudaStream_t st) {
  const int rc = prepare_wgrad<DY_BF16, X_BF16>();
  if (rc) return rc;
  const dim3 grid(gx, (a.N + a.nc - 1) / a.nc, (a.K + a.kc - 1) / a.kc);
  k_lin_wgrad<DY_BF16, X_BF16><<<grid, 32 * (WG_LOADERS + 1), smem, st>>>(a);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}
int launch_wgrad_fp32(WgradArgs& a, const spion_tokens* dY, const spion_tokens* X, int gx, size_t smem, cudaStream_t st) {
  int rc = prepare_wgrad_fp32();
  if (rc) return rc;
  WgradMaps maps;
  a.box_y = half_boxes(dY, a.T);
  a.box_x = half_boxes(X, a.T);
  if ((a.box_y && (rc = half_maps(dY, a.T, maps.y))) || (a.box_x && (rc = half_maps(X, a.T, maps.x)))) return rc;
  const dim3 grid(gx, (a.N + a.nc - 1) / a.nc, (a.K + a.kc - 1) / a.kc);
  k_lin_wgrad_fp32<<<grid, 32 * (WG_LOADERS + 2), smem, st>>>(a, maps);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

// chunking of the weight gradient: at most four 64-wide chunks of dY and X per CTA, and what tensor memory holds
bool plan_wgrad(int split, int N, int K, int* nc, int* kc, int* stages, int* raws, size_t* smem) {
  const int kw = K <= 64 ? 64 : 128;
  int nw = (N + 63) / 64 * 64;
  if (nw + kw > 256) nw = 256 - kw;
  const int cpt = (nw + kw) / 64;
  *nc = nw; *kc = kw; *raws = 0;
  if (split == 3) {
    for (int st = 3; st >= 2; --st)
      for (int raw = 6; raw >= 4; raw -= 2) {            // even: a slot belongs to one of the two groups
        *smem = (size_t)cpt * (st * 3 * HCHUNK + raw * HRAW) + 512;
        if (*smem <= SMEM_MAX) { *stages = st; *raws = raw; return true; }
      }
    return false;
  }
  for (int st = 6; st >= 3; --st) {                      // two stages of copies in flight
    *smem = (size_t)st * cpt * WCHUNK + 256 + WG_LOADERS * 256 * 4;
    if (*smem <= SMEM_MAX) { *stages = st; return true; }
  }
  return false;
}

// CTAs along the tokens: one per SM over all slices; fp32 mode: as many more as keep the chains in tensor memory short (above).
// Relative error of dW and db against fp64, normal operands (in brackets the library's product and reduction in their place): 262144
// tokens, 64 x 64 1.7e-7, 1.7e-7 (1.1e-6, 1.7e-7); 64 x 192 5.6e-7, 1.7e-7 (1.3e-6, 3.1e-7); 256 x 1024 5.8e-7, 1.8e-7 (2.2e-6, 2.1e-7).
// dW from operands of one sign, where every truncation adds up: 1.4e-7 (1.5e-7), 9.4e-7 (1.9e-7), 9.9e-7 (4.0e-7).
constexpr int CHAIN = 40;
int wgrad_grid(long long T, int N, int K, int split) {
  int nc, kc, st, raws;
  size_t smem;
  if (!plan_wgrad(split, N, K, &nc, &kc, &st, &raws, &smem)) return 0;
  const int per = ((N + nc - 1) / nc) * ((K + kc - 1) / kc);
  const long long tiles = (T + 63) / 64;
  long long gx = sm_count() / per;
  if (gx < 1) gx = 1;
  if (split == 3) {
    const long long most = (long long)CHAIN * (WgradAcc(nc, kc / 64).total() - 1) / 4;       // tiles of a CTA, four steps each
    gx *= (tiles + gx * most - 1) / (gx * most);
  }
  return (int)(gx < tiles ? gx : tiles);
}

}  // namespace

// longest contraction (a multiple of 64) of one launch of the input-gradient GEMM
static int max_contraction(int split, int N) {
  int nc, nacc, st;
  size_t smem;
  int k = 1024;
  while (k > 64 && !plan_gemm(split, true, k, N, &nc, &nacc, &st, &smem)) k -= 64;
  return k;
}

extern "C" int spion_linear_supported(int in_features, int out_features, int fp32) {
  int nc, kc, nacc, st, raws;
  size_t smem;
  const int sp = fp32 ? 3 : 1;
  if (in_features < 32 || out_features < 32 || in_features % 32 || out_features % 32) return 0;
  if (in_features > 1024 || out_features > 1024) return 0;
  return plan_gemm(sp, false, in_features, out_features, &nc, &nacc, &st, &smem) &&
         plan_gemm(sp, true, fp32 ? 64 : out_features, in_features, &nc, &nacc, &st, &smem) &&
         plan_wgrad(sp, out_features, in_features, &nc, &kc, &st, &raws, &smem);
}

extern "C" int spion_linear_prepare(int fp32) {
  int rc;
  if (fp32) {
    if ((rc = prepare_gemm<3, false, false, EPI_NONE, false>()) || (rc = prepare_gemm<3, false, true, EPI_NONE, false>()) ||
        (rc = prepare_gemm<3, false, false, EPI_NONE, false, false>()) || (rc = prepare_gemm<3, false, true, EPI_NONE, false, false>()))
      return rc;
    return prepare_wgrad_fp32();
  }
  if ((rc = prepare_gemm<1, true, false, EPI_GELU, true, false, false>()) || (rc = prepare_gemm<1, false, false, EPI_GELU, true, false, false>()) ||
      (rc = prepare_gemm<1, true, true, EPI_DGELU, true, false, false>()))
    return rc;
  if ((rc = prepare_gemm<1, true, false, EPI_NONE, true>()) || (rc = prepare_gemm<1, false, false, EPI_NONE, true>()) ||
      (rc = prepare_gemm<1, true, false, EPI_GELU, true>()) || (rc = prepare_gemm<1, false, false, EPI_GELU, true>()) ||
      (rc = prepare_gemm<1, true, true, EPI_DGELU, true>()) || (rc = prepare_gemm<1, true, true, EPI_NONE, true>()) ||
      (rc = prepare_gemm<1, true, true, EPI_NONE, false>()) || (rc = prepare_wgrad<true, false>()))
    return rc;
  return prepare_wgrad<true, true>();
}

int linear_status(int reset, cudaStream_t st) {
  int v = 0;
  SPION_CUDA_TRY(cudaMemcpyFromSymbolAsync(&v, g_lin_status, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
  SPION_CUDA_TRY(cudaStreamSynchronize(st));
  if (v == 0) return SPION_OK;
  if (reset) {
    void* word = nullptr;
    SPION_CUDA_TRY(cudaGetSymbolAddress(&word, g_lin_status));
    SPION_CUDA_TRY(cudaMemsetAsync(word, 0, sizeof(int), st));
    SPION_CUDA_TRY(cudaStreamSynchronize(st));
  }
  fprintf(stderr, "spion_b200: status word of the linear layers = 0x%x (a bounded wait gave up)\n", v);
  return SPION_ERR_TIMEOUT;
}

extern "C" int spion_linear_status(int reset) {
  SPION_CUDA_TRY(cudaDeviceSynchronize());               // the layers may run on streams that the copy below is not ordered after
  return linear_status(reset, 0);
}

// One CTA waits, with a limit, on a barrier that nothing arrives on.
__global__ void k_lin_wait_selftest(long long limit_cycles) {
  __shared__ __align__(8) unsigned long long bar_storage;
  const uint32_t bar = smem_u32(&bar_storage);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const bool ok = __syncthreads_and(mbar_wait_limit(bar, 0, limit_cycles));
  if (!ok && threadIdx.x == 0) report(&g_lin_status, ERR_LOAD_WAIT);
}

extern "C" int spion_linear_selftest_bounded_wait(long long limit_cycles, void* cuda_stream) {
  if (limit_cycles < 1 || limit_cycles > 2000000000LL) return SPION_ERR_ARG;
  k_lin_wait_selftest<<<1, 128, 0, (cudaStream_t)cuda_stream>>>(limit_cycles);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

extern "C" int spion_linear_forward(const spion_tokens* X, const float* const* W, const float* const* bias, int nw, int fp32,
                                    const spion_tokens* Y, void* gelu_out, long long T, int in_features, int out_features,
                                    void* cuda_stream) {
  return spion_linear_forward_keep(X, W, bias, nw, fp32, Y, gelu_out, nullptr, nullptr, T, in_features, out_features, cuda_stream);
}

static int forward(const spion_tokens* X, const float* const* W, const float* const* bias, int nw, int fp32, const spion_tokens* Y, void* gelu_out,
                   void* x_copy, float* w_copy, long long T, int in_features, int out_features, const float* mask, int heads, int seq_len, float* pen,
                   void* cuda_stream) {
  if (!mat_ok(X) || !mat_ok(Y) || !W || nw < 1 || nw > 3 || T < 1 || T > 0x7fffffffLL - 256) return SPION_ERR_ARG;
  if (X->cols * X->count != in_features || Y->cols * Y->count != out_features || out_features % nw) return SPION_ERR_ARG;
  if (fp32 && (X->is_bf16 || Y->is_bf16 || gelu_out)) return SPION_ERR_UNSUPPORTED;
  if (gelu_out && (!Y->is_bf16 || ((uintptr_t)gelu_out & 31))) return SPION_ERR_UNSUPPORTED;
  if ((fp32 && (x_copy || w_copy)) || (x_copy && X->is_bf16)) return SPION_ERR_UNSUPPORTED;
  if (((uintptr_t)x_copy | (uintptr_t)w_copy) & 15) return SPION_ERR_ARG;
  GemmArgs a;
  a.A = to_mat(X); a.Y = to_mat(Y);
  a.wper = out_features / nw; a.wld = in_features;
  for (int i = 0; i < 3; ++i) { a.W[i] = i < nw ? W[i] : nullptr; a.bias[i] = (bias && i < nw) ? bias[i] : nullptr; }
  for (int i = 0; i < nw; ++i) if (!a.W[i] || ((uintptr_t)a.W[i] & 15)) return SPION_ERR_ARG;
  a.T = (int)T; a.K = in_features; a.N = out_features;
  a.h = nullptr; a.g = (__nv_bfloat16*)gelu_out; a.x_copy = (__nv_bfloat16*)x_copy; a.w_copy = w_copy;
  a.mask = mask; a.pen = pen; a.pen_heads = heads; a.pen_L = seq_len;
  size_t smem;
  a.k0 = 0; a.accum = 0; a.parts = 0;
  const int most = X->is_bf16 ? 384 : 256;
  if (!choose_epilogue(a, gelu_out ? EPI_GELU : EPI_NONE, staged_outputs(X, Y, T), staged_bytes(gelu_out != nullptr, Y->is_bf16),
                       fp32 ? FREE : gelu_out ? (a.K <= most ? FREE : 0) : Y->is_bf16 && a.K <= 256 ? a.N / 2 : 0, [&](size_t table, size_t outs) {
                         return plan_gemm(fp32 ? 3 : 1, false, a.K, a.N, &a.nc, &a.nacc, &a.nstages, &smem, 256, table, outs);
                       }))
    return SPION_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  if (fp32) return launch_gemm<3, false, false, EPI_NONE, false>(a, X, Y, smem, st);
  if (gelu_out)
    return X->is_bf16 ? launch_gemm<1, true, false, EPI_GELU, true>(a, X, Y, smem, st) : launch_gemm<1, false, false, EPI_GELU, true>(a, X, Y, smem, st);
  if (Y->is_bf16)
    return X->is_bf16 ? launch_gemm<1, true, false, EPI_NONE, true>(a, X, Y, smem, st) : launch_gemm<1, false, false, EPI_NONE, true>(a, X, Y, smem, st);
  return X->is_bf16 ? launch_gemm<1, true, false, EPI_NONE, false>(a, X, Y, smem, st) : launch_gemm<1, false, false, EPI_NONE, false>(a, X, Y, smem, st);
}

extern "C" int spion_linear_forward_keep(const spion_tokens* X, const float* const* W, const float* const* bias, int nw, int fp32,
                                         const spion_tokens* Y, void* gelu_out, void* x_copy, float* w_copy, long long T,
                                         int in_features, int out_features, void* cuda_stream) {
  return forward(X, W, bias, nw, fp32, Y, gelu_out, x_copy, w_copy, T, in_features, out_features, nullptr, 0, 0, nullptr, cuda_stream);
}

extern "C" int spion_linear_forward_keypad(const spion_tokens* X, const float* const* W, const float* const* bias, int nw, int fp32,
                                           const spion_tokens* Y, void* x_copy, float* w_copy, long long T, int in_features, int out_features,
                                           const float* mask, int batch, int heads, int seq_len, float* pen, void* cuda_stream) {
  if (!mask || !pen || batch < 1 || heads < 1 || seq_len < 1) return SPION_ERR_ARG;
  if ((long long)batch * seq_len != T || T * heads > 0x7fffffffLL) return SPION_ERR_SHAPE;
  return forward(X, W, bias, nw, fp32, Y, nullptr, x_copy, w_copy, T, in_features, out_features, mask, heads, seq_len, pen, cuda_stream);
}

extern "C" int spion_linear_backward_input(const spion_tokens* dY, const float* const* W, int nw, int fp32, const void* gelu_in,
                                           const spion_tokens* dX, long long T, int in_features, int out_features,
                                           void* cuda_stream) {
  if (!mat_ok(dY) || !mat_ok(dX) || !W || nw < 1 || nw > 3 || T < 1 || T > 0x7fffffffLL - 256) return SPION_ERR_ARG;
  if (dX->cols * dX->count != in_features || dY->cols * dY->count != out_features || out_features % nw) return SPION_ERR_ARG;
  if (fp32 && (dX->is_bf16 || dY->is_bf16 || gelu_in)) return SPION_ERR_UNSUPPORTED;
  if (gelu_in && (!dX->is_bf16 || ((uintptr_t)gelu_in & 31))) return SPION_ERR_UNSUPPORTED;
  GemmArgs a;
  a.A = to_mat(dY); a.Y = to_mat(dX);
  a.wper = out_features / nw; a.wld = in_features;
  for (int i = 0; i < 3; ++i) { a.W[i] = i < nw ? W[i] : nullptr; a.bias[i] = nullptr; }
  for (int i = 0; i < nw; ++i) if (!a.W[i] || ((uintptr_t)a.W[i] & 15)) return SPION_ERR_ARG;
  a.T = (int)T; a.K = out_features; a.N = in_features;
  a.h = (const __nv_bfloat16*)gelu_in; a.g = nullptr; a.x_copy = nullptr; a.w_copy = nullptr; a.mask = nullptr; a.pen = nullptr;
  size_t smem;
  a.k0 = 0; a.accum = 0;
  a.parts = !fp32 && dX->is_bf16 && nw == 3 ? a.wper / 64 : 0;
  if (a.parts && a.wper % 64) return SPION_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  if (fp32) {                                            // the split weights of a long contraction fill shared memory: several launches
    const int total = a.K, step = max_contraction(3, a.N);
    for (a.k0 = 0; a.k0 < total; a.k0 += step) {
      a.K = total - a.k0 < step ? total - a.k0 : step;
      a.accum = a.k0 > 0;
      if (!choose_epilogue(a, EPI_NONE, total <= step && staged_outputs(dY, dX, T), staged_bytes(false, false), FREE, [&](size_t, size_t outs) {
            return plan_gemm(3, true, a.K, a.N, &a.nc, &a.nacc, &a.nstages, &smem, 256, 0, outs);
          }))
        return SPION_ERR_UNSUPPORTED;
      const int rc = launch_gemm<3, false, true, EPI_NONE, false>(a, dY, dX, smem, st);
      if (rc) return rc;
    }
    return SPION_OK;
  }
  if (!choose_epilogue(a, gelu_in ? EPI_DGELU : EPI_NONE, staged_outputs(dY, dX, T), staged_bytes(gelu_in != nullptr, dX->is_bf16),
                       gelu_in ? FREE : dY->is_bf16 && !dX->is_bf16 ? (a.K <= 320 ? a.N : a.N * 3 / 4) : 0, [&](size_t table, size_t outs) {
                         return plan_gemm(1, true, a.K, a.N, &a.nc, &a.nacc, &a.nstages, &smem, a.parts ? 64 : 256, table, outs);
                       }))
    return SPION_ERR_UNSUPPORTED;
  if (gelu_in)
    return dY->is_bf16 ? launch_gemm<1, true, true, EPI_DGELU, true>(a, dY, dX, smem, st) : launch_gemm<1, false, true, EPI_DGELU, true>(a, dY, dX, smem, st);
  if (dX->is_bf16)
    return dY->is_bf16 ? launch_gemm<1, true, true, EPI_NONE, true>(a, dY, dX, smem, st) : launch_gemm<1, false, true, EPI_NONE, true>(a, dY, dX, smem, st);
  return dY->is_bf16 ? launch_gemm<1, true, true, EPI_NONE, false>(a, dY, dX, smem, st) : launch_gemm<1, false, true, EPI_NONE, false>(a, dY, dX, smem, st);
}

extern "C" long long spion_linear_workspace_floats(long long T, int in_features, int out_features, int fp32) {
  return (long long)wgrad_grid(T, out_features, in_features, fp32 ? 3 : 1) * ((long long)in_features * out_features + out_features);
}

extern "C" int spion_linear_backward_weight(const spion_tokens* dY, const spion_tokens* X, int fp32, float* dW, float* db,
                                            float* workspace, long long T, int in_features, int out_features, void* cuda_stream) {
  if (!mat_ok(dY) || !mat_ok(X) || !dW || !db || !workspace || T < 1 || T > 0x7fffffffLL - 256) return SPION_ERR_ARG;
  if (((uintptr_t)dW | (uintptr_t)db | (uintptr_t)workspace) & 15) return SPION_ERR_ARG;
  if (X->cols * X->count != in_features || dY->cols * dY->count != out_features) return SPION_ERR_ARG;
  if (fp32 && (X->is_bf16 || dY->is_bf16)) return SPION_ERR_UNSUPPORTED;
  WgradArgs a;
  a.dY = to_mat(dY); a.X = to_mat(X);
  a.T = (int)T; a.N = out_features; a.K = in_features; a.part = workspace;
  size_t smem;
  if (!plan_wgrad(fp32 ? 3 : 1, a.N, a.K, &a.nc, &a.kc, &a.nstages, &a.nraw, &smem)) return SPION_ERR_UNSUPPORTED;
  const int gx = wgrad_grid(T, a.N, a.K, fp32 ? 3 : 1);
  if (gx < 1) return SPION_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  int rc;
  if (fp32) rc = launch_wgrad_fp32(a, dY, X, gx, smem, st);
  else if (dY->is_bf16) rc = X->is_bf16 ? launch_wgrad<true, true>(a, gx, smem, st) : launch_wgrad<true, false>(a, gx, smem, st);
  else rc = X->is_bf16 ? launch_wgrad<false, true>(a, gx, smem, st) : launch_wgrad<false, false>(a, gx, smem, st);
  if (rc) return rc;
  const long long nw = (long long)a.N * a.K, n = nw + a.N;
  SPION_CUDA_TRY(launch_after(k_lin_reduce, dim3((unsigned)((n / 4 + 31) / 32)), dim3(256), 0, st, workspace, gx, n, nw, dW, db));
  return SPION_OK;
}
