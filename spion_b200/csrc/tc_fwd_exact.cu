// Forward on the full mask (the dense warm-up phase; sm_100a, bf16, 64 x 64 blocks, no stored P): two passes over a row, the maximum first, and the
// sums in a fixed order (four chains a half tile), so that O and lse are bit for bit what a two-pass kernel gives.  Some results there
// are sums that cancel to nothing but rounding (the gradient of the key projection's bias is zero in dense attention), so that every other
// order of the additions gives other numbers.
//
// One persistent CTA per SM with four groups.  A group has four arithmetic warps (one per tensor-memory quadrant), a warp that issues its MMAs
// and one that loads its tiles, and walks block rows of its own, two blocks ("a pair") at a time, every pair twice:
//     S = Q K_e^T   (M = 64, the second block at lane offset 16: query rows along the lanes, a row owned by lanes l and l + 16)
//     P = exp2(S scale log2e - m), unnormalised, bf16 into shared memory
//     O += P V_e    (M = 64, one accumulator: the products of the two blocks one after the other)
// S of pair j + 1 is computed while pair j is in the arithmetic, and the rows of a finished unit are written before the first product of the
// next one.  Nothing is exchanged between the groups: they only fill each other's waits.  (tc_fwd_stream.cu sums the products of the two
// blocks of a pair apart, P from tensor memory, which is faster and another order.)
//
// What bounds it: the chain of a pair; the dense phase has about one unit per group.  18 matrices, L = 1984, d 32: 54 us with one warp per
// group for loads and MMAs, 46 now.
//
// Every wait is bounded; on a time-out the waiting warp records a code in the status word and the CTA winds down.
#include "tc_stream.cuh"

using namespace tc;

namespace {


constexpr int NG = 4;                                             // groups
// Warps: four arithmetic ones per group, then one per group that issues its MMAs, one per group that loads its tiles; the arithmetic warps take
// registers of the others (setmaxnreg: 16 * 96 + 8 * 48 = 24 * 80 that the CTA is launched with).
constexpr int FX_THREADS = 32 * 24;

template <int D> struct Fx {
  using T = OpTile<D>;
  static constexpr int KB = D == 64 ? 1 : 2, VB = KB;             // buffers for the K tiles, the V tiles of a pair
  static constexpr uint32_t O_Q = 0, O_K = T::BYTES, O_V = O_K + 2 * KB * T::BYTES, O_P = O_V + 2 * VB * T::BYTES, GROUP = O_P + 2 * VT_BYTES;
  static constexpr uint32_t O_BAR = NG * GROUP;
  static constexpr uint32_t GBAR = 128;                           // barriers of a group
  static constexpr uint32_t O_INFO = O_BAR + NG * GBAR + 16;      // of a group: records of eight pairs, flags of four
  static constexpr size_t SMEM = O_INFO + NG * 256;
  static constexpr uint32_t T_O = 64, COLS = 64 + D;              // tensor-memory columns of a group: S, O
};

// two blocks; no pair; the pair's values are used, the first ones of the unit
constexpr int PR_TWO = 1, PR_END = 2, PR_VALUES = 4, PR_FRESH = 8;

struct FsArgs {
  __nv_bfloat16* O;
  float* lse;
  const float* keypad;
  const int4 *rec, *pair;                                         // block rows and their pairs (k_line_recs)
  int L, BH, nb, heads, by_rank;
  float scale, floor_v;
  int* status;
};

template <int D, bool KP>
__global__ void __launch_bounds__(FX_THREADS, 1) k_fwd_exact(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ FsArgs a) {
  using C = Fx<D>;
  using T = OpTile<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);                      // must be 1024-aligned (checked below)
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int grp = warp < 4 * NG ? warp >> 2 : (warp - 4 * NG) & 3;          // arithmetic warps, four for MMAs, four for loads
  const uint32_t gb = sbase + grp * C::GROUP, bars = sbase + C::O_BAR + grp * C::GBAR;
  // k_full[KB]: K tiles of a pair, Q with the first of a unit, and the pair's record; k_free[KB]: S of that pair complete; v_full[VB]: V tiles
  // landed; v_free[VB]: product of that pair complete; s_ready: S of a pair complete; s_free: read out (4 warps); p_ready: P of a pair written
  // (4 warps); pv_done: O += P V of a pair complete; pi_full[4]: flags of a pair written.  As in tc_fwd_stream.cu.
  constexpr uint32_t B_KFULL = 0, B_KFREE = 16, B_VFULL = 32, B_VFREE = 48, B_SREADY = 64, B_SFREE = 72, B_PREADY = 80, B_PV = 88, B_PI = 96;
  const uint32_t k_full = bars + B_KFULL, k_free = bars + B_KFREE, v_full = bars + B_VFULL, v_free = bars + B_VFREE, s_ready = bars + B_SREADY,
                 s_free = bars + B_SFREE, p_ready = bars + B_PREADY, pv_done = bars + B_PV, pi_full = bars + B_PI;
  constexpr int KB = C::KB, VB = C::VB;
  const uint32_t slot = sbase + C::O_BAR + NG * C::GBAR, abort_w = slot + 4;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  volatile int* abort_ptr = reinterpret_cast<volatile int*>(smem_raw + (abort_w - sbase));
  // records [8]: PR_*;  flags [4][8]: which blocks have different penalties, block columns, -, one penalty per block in base-2 units
  int4* ring = reinterpret_cast<int4*>(smem_raw + C::O_INFO + grp * 256);
  int* info = reinterpret_cast<int*>(smem_raw + C::O_INFO + grp * 256 + 128);

  if (warp == 0 && lane == 0) {
    int ab = *reinterpret_cast<volatile int*>(a.status);
    if ((sbase & 1023u) != 0u) { report(a.status, ERR_LOAD_WAIT); ab = 1; }
    *abort_ptr = ab;
    for (int g = 0; g < NG; ++g) {
      const uint32_t b = sbase + C::O_BAR + g * C::GBAR;
      for (int x = 0; x < 16; ++x) mbar_init(b + 8 * x, x == 9 || x == 10 ? 4 : 1);     // s_free, p_ready: the group's warps
    }
    fence_barrier_init();
  }
  __syncthreads();
  if (*abort_ptr != 0) return;
  if (warp == 0) {
    tmem_alloc(slot, 512u);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr, tS = tmem + grp * C::COLS, tO = tS + C::T_O;
  auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool { return warp_wait(bar, parity & 1u, a.status, code); };
  const UnitMap um{a.nb, a.BH, a.by_rank};
  // group g of CTA b walks units b + g G, + NG G, ...
  const int first = (int)blockIdx.x + grp * (int)gridDim.x, step = NG * (int)gridDim.x, total = a.nb * a.BH;

  auto wait_one = [&](uint32_t bar, uint32_t parity, int code) -> bool {           // one thread
    if (mbar_wait(bar, parity & 1u)) return true;
    report(a.status, code);
    return false;
  };
  if (warp < 4 * NG) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
  else asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");

  if (warp >= 4 * NG + 4) {
    // ================================================================== loads of a group
    Walk w;
    w.init(um, a.rec, first, step, total);
    w.skip();
    int4 pr = w.valid() ? a.pair[w.cur.y] : make_int4(0, -1, 0, 0), nx = pr;       // records of pairs j, j + 1
    int jv = 0;                                                   // value pairs before pair j
    bool values = false;                                          // the pairs of a unit come twice, for the maximum and for the values
    for (int j = 0;; ++j) {
      const int kj = j / KB;
      if (j >= KB && !wait_all(k_free + 8 * (j % KB), (uint32_t)(kj - 1), ERR_MMA_WAIT)) break;
      const uint32_t kb = k_full + 8 * (j % KB);
      if (!w.valid()) {
        if (lane == 0) {
          ring[j & 7] = make_int4(PR_END, 0, 0, 0);
          mbar_arrive(kb);
        }
        break;
      }
      const bool two = w.cnt() == 2, with_q = w.k == 0 && !values, with_v = values;
      const OpPos pos = op_pos(w.bh, a.L, a.heads, D);
      const int bh = w.bh, line = w.cur.x;
      // Q of the unit before was read by all S up to pair j - 1
      if (KB == 2 && with_q && j >= 1 && !wait_all(k_free + 8 * ((j - 1) % KB), (uint32_t)((j - 1) / KB), ERR_MMA_WAIT)) break;
      if (elect_one()) {
        ring[j & 7] = make_int4((two ? PR_TWO : 0) | (values ? PR_VALUES : 0) | (values && w.k == 0 ? PR_FRESH : 0), 0, 0, 0);
        mbar_expect_tx(kb, ((two ? 2 : 1) + (with_q ? 1 : 0)) * T::BYTES);
        const uint32_t dst = gb + C::O_K + (j % KB) * 2 * T::BYTES;
        tma_load_2d(dst, &tmK, kb, pos.x0, pos.row0 + pr.x * BS);
        if (two) tma_load_2d(dst + T::BYTES, &tmK, kb, pos.x0, pos.row0 + pr.y * BS);
        if (with_q) tma_load_2d(gb + C::O_Q, &tmQ, kb, pos.x0, pos.row0 + line * BS);
      }
      __syncwarp();
      if (w.last() && !values) {
        values = true;
        w.k = 0;
      } else {
        if (w.last()) values = false;
        w.next();
      }
      if (w.valid()) nx = a.pair[w.cur.y + w.k];
      if (KP) {
        const int e = lane >> 4, o = e ? (two ? pr.y : -1) : pr.x;
        uint32_t mixed = 0u;
        Pen4 p = {};
        if (o >= 0) pen_load(p, a.keypad + (size_t)bh * a.L + o * BS);
        const float pen = pen_of(p, mixed) * LOG2E, pen1 = __shfl_sync(0xffffffffu, pen, 16);
        if (lane == 0) {
          int* x = info + 8 * (j & 3);
          x[0] = (int)mixed;
          x[1] = pr.x; x[2] = pr.y;
          x[4] = __float_as_int(pen); x[5] = __float_as_int(pen1);
          mbar_arrive(pi_full + 8 * (j & 3));
        }
        __syncwarp();
      }
      if (with_v) {
        if (jv >= VB && !wait_all(v_free + 8 * (jv % VB), (uint32_t)(jv / VB - 1), ERR_MMA2_WAIT)) break;
        if (elect_one()) {
          const uint32_t vb = v_full + 8 * (jv % VB), dst = gb + C::O_V + (jv % VB) * 2 * T::BYTES;
          mbar_expect_tx(vb, (two ? 2 : 1) * T::BYTES);
          tma_load_2d(dst, &tmV, vb, pos.x0, pos.row0 + pr.x * BS);
          if (two) tma_load_2d(dst + T::BYTES, &tmV, vb, pos.x0, pos.row0 + pr.y * BS);
        }
        __syncwarp();
        ++jv;
      }
      pr = nx;
    }
  } else if (warp >= 4 * NG) {
    // ================================================================== MMAs of a group: one thread
    if (elect_one()) {
      constexpr uint32_t IDESC_S = make_idesc_bf16(64, 64, 0, 0), IDESC_O = make_idesc_bf16(64, D, 0, 1);
      const uint64_t dQ = T::kmajor(gb + C::O_Q, 0), dK = T::kmajor(gb + C::O_K, 0), dV = T::mnmajor(gb + C::O_V, 0),
                     dP = ValTile::kmajor(gb + C::O_P, 0);
      int prev = 0, jp = 0;                                       // record of pair j - 1, value pairs before it
      for (int j = 0;; ++j) {
        if (!wait_one(k_full + 8 * (j % KB), (uint32_t)(j / KB), ERR_LOAD_WAIT)) break;
        const int now = ring[j & 7].x;
        if (!(now & PR_END)) {                                    // S of pair j
          if (j >= 1 && !wait_one(s_free, (uint32_t)(j - 1), ERR_MMA_WAIT)) break;
          tc_fence_after();
          const uint64_t k = desc_advance(dK, (j % KB) * 2 * T::BYTES);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_bf16(tS, desc_advance(dQ, kk * T::K_STEP), desc_advance(k, kk * T::K_STEP), IDESC_S, kk > 0);
          if (now & PR_TWO) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              mma_bf16(tS + (16u << 16), desc_advance(dQ, kk * T::K_STEP), desc_advance(k, T::BYTES + kk * T::K_STEP), IDESC_S, kk > 0);
          }
          mma_commit(s_ready);
          mma_commit(k_free + 8 * (j % KB));
        }
        if (prev & PR_VALUES) {                                   // O += P V of pair j - 1
          if (!wait_one(v_full + 8 * (jp % VB), (uint32_t)(jp / VB), ERR_LOAD_WAIT)) break;
          if (!wait_one(p_ready, (uint32_t)jp, ERR_MMA_WAIT)) break;
          tc_fence_after();
          const uint32_t more = (prev & PR_FRESH) ? 0u : 1u;      // not the first product of its unit
          const uint64_t v = desc_advance(dV, (jp % VB) * 2 * T::BYTES);
#pragma unroll
          for (int kk = 0; kk < BS / 16; ++kk) mma_bf16(tO, desc_advance(dP, kk * ValTile::K_STEP), desc_advance(v, kk * T::MN_STEP), IDESC_O, kk > 0 ? 1u : more);
          if (prev & PR_TWO) {
#pragma unroll
            for (int kk = 0; kk < BS / 16; ++kk)
              mma_bf16(tO, desc_advance(dP, VT_BYTES + kk * ValTile::K_STEP), desc_advance(v, T::BYTES + kk * T::MN_STEP), IDESC_O, 1u);
          }
          mma_commit(pv_done);
          mma_commit(v_free + 8 * (jp % VB));
          ++jp;
        }
        if (now & PR_END) break;
        prev = now;
      }
    }
    __syncwarp();
  } else {
    // ================================================================== arithmetic warps of a group
    const int q = warp & 3, hf = lane >> 4, row = q * 16 + (lane & 15);
    const uint32_t lS = tS + ((uint32_t)(q * 32) << 16), lO = lS + C::T_O;
    const uint32_t tile = gb + C::O_P + hf * VT_BYTES + row * 128;
    const float sc2 = a.scale * LOG2E, floor2 = a.floor_v * LOG2E, inv_scale = 1.0f / a.scale;
    bool ok = true;
    // the finished unit whose rows are still in tensor memory (lanes 0-15 of every quadrant)
    bool pend = false;
    float pend_inv = 0.f;
    __nv_bfloat16* pend_dst = nullptr;
    auto write_rows = [&](__nv_bfloat16* dst, float inv) {
#pragma unroll
      for (int h = 0; h < D / 32; ++h) {
        uint32_t v[32];
        tmem_ld32(lO + h * 32, v);
        tmem_ld_wait();
        if (hf == 0) {
#pragma unroll
          for (int x = 0; x < 32; x += 8)
            *reinterpret_cast<uint4*>(dst + h * 32 + x) = make_uint4(pack_bf16(__uint_as_float(v[x]) * inv, __uint_as_float(v[x + 1]) * inv),
                                                                     pack_bf16(__uint_as_float(v[x + 2]) * inv, __uint_as_float(v[x + 3]) * inv),
                                                                     pack_bf16(__uint_as_float(v[x + 4]) * inv, __uint_as_float(v[x + 5]) * inv),
                                                                     pack_bf16(__uint_as_float(v[x + 6]) * inv, __uint_as_float(v[x + 7]) * inv));
        }
      }
    };
    Walk u;
    u.init(um, a.rec, first, step, total);
    int j = 0, jv = 0;                                            // pairs, value pairs
    for (; u.valid() && ok; u.shift()) {
      const int n = u.cur.w;
      const OpPos pos = op_pos(u.bh, a.L, a.heads, D);
      __nv_bfloat16* dst = a.O + (size_t)(pos.row0 + u.cur.x * BS + row) * pos.ld + pos.x0;
      float* lse = a.lse + (size_t)u.bh * a.L + u.cur.x * BS + row;
      const float* kpu = KP ? a.keypad + (size_t)u.bh * a.L : nullptr;
      float m = floor2, mx = floor2, l = 0.f;                     // reference exponent, true maximum, sum
      int n_sel = 0;
      const int np = u.pairs();
      for (int kx = -np; kx < np && ok; ++kx, ++j) {
        const bool values = kx >= 0;
        const int k = values ? kx : kx + np;
        const bool mine = 2 * k + hf < n;
        const float* kp = nullptr;
        float pen = 0.f;
        if (KP) {
          if (!wait_all(pi_full + 8 * (j & 3), (uint32_t)(j >> 2), ERR_MMA_WAIT)) { ok = false; break; }
          const int* x = info + 8 * (j & 3);
          const bool mixed = (x[0] >> hf) & 1;
          pen = mixed ? 0.f : __int_as_float(x[4 + hf]);
          if (mixed) kp = kpu + x[1 + hf] * BS;
        }
        if (values) n_sel += mine ? BS : 0;
        if (!wait_all(s_ready, (uint32_t)j, ERR_MMA_WAIT)) { ok = false; break; }
        tc_fence_after();
        uint32_t v0[32], v1[32];
        tmem_ld32(lS, v0);
        tmem_ld32(lS + 32u, v1);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
        if (KP && kp) {
          take_penalty(v0, kp, inv_scale);
          take_penalty(v1, kp + 32, inv_scale);
        }
        float cm = -INFINITY;
        if (!values) {                                            // the scale is positive: compare raw scores
          float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            m0 = max3(m0, __uint_as_float(v0[x]), __uint_as_float(v0[x + 1]));
            m1 = max3(m1, __uint_as_float(v0[x + 2]), __uint_as_float(v0[x + 3]));
            m2 = max3(m2, __uint_as_float(v1[x]), __uint_as_float(v1[x + 1]));
            m3 = max3(m3, __uint_as_float(v1[x + 2]), __uint_as_float(v1[x + 3]));
          }
          if (mine) cm = fmaxf(fmaf(fmaxf(m0, m1), sc2, -pen), fmaf(fmaxf(m2, m3), sc2, -pen));
        }
        cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, 16));     // both owners of a row agree
        mx = fmaxf(mx, cm);
        m = mx;
        if (!values) continue;
        // the P tiles of the pair before have been consumed
        if (jv >= 1 && !wait_all(pv_done, (uint32_t)(jv - 1), ERR_MMA2_WAIT)) { ok = false; break; }
        tc_fence_after();
        const uint64_t sc22 = pack2(sc2, sc2), nm2 = pack2(-(m + pen), -(m + pen));
        auto half_row = [&](const uint32_t (&v)[32], int g) {
          float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {                        // eight columns: one 16-byte piece of the tile row
            uint32_t w[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int c = cc * 8 + 2 * x;
              float e0, e1;
              unpack2(fma2(pack2(v[c], v[c + 1]), sc22, nm2), e0, e1);
              e0 = ex2_approx(e0); e1 = ex2_approx(e1);
              l4[x] += e0 + e1;
              w[x] = pack_bf16(e0, e1);
            }
            st_shared_v4(tile + (uint32_t)(((g * 4 + cc) ^ (row & 7)) << 4), w);
          }
          l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
        };
        if (mine) {
          half_row(v0, 0);
          half_row(v1, 1);
        }
        if (pend) {                                               // the previous unit, before this one's first product
          write_rows(pend_dst, pend_inv);
          pend = false;
        }
        fence_proxy_async();                                      // P rows -> visible to the MMA
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready);
        ++jv;
      }
      if (!ok) break;
      n_sel += __shfl_xor_sync(0xffffffffu, n_sel, 16);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      const float z = l + (float)(a.L - n_sel) * exp2f(-mx);
      if (hf == 0) *lse = mx + log2f(z);
      pend = true; pend_inv = 1.0f / z; pend_dst = dst;
    }
    if (ok && pend && wait_all(pv_done, (uint32_t)(jv - 1), ERR_MMA2_WAIT)) {
      tc_fence_after();
      write_rows(pend_dst, pend_inv);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512u);
}

}  // namespace

namespace tc {

template <int D, bool KP>
static int fx_launch(spion_ctx* c, TcState* s, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const FsArgs& a) {
  using C = Fx<D>;
  static_assert(C::SMEM <= 227 * 1024 && NG * C::COLS <= 512, "shared or tensor memory");
  const long long total = (long long)c->BH * a.nb;
  const int grid = (int)(total < (long long)s->sms ? total : (long long)s->sms);       // one CTA per SM (all 512 TMEM columns)
  k_fwd_exact<D, KP><<<grid, FX_THREADS, C::SMEM, c->stream>>>(mq, mk, mv, a);
  SPION_LAUNCH_CHECK();
  c->launches += 1;
  return SPION_OK;
}

template <int D>
static int fx_forward(spion_ctx* c, TcState* s, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const float* keypad,
                      void* O, float* lse) {
  const TcView vw = tc_view(c, s);
  FsArgs a;
  a.O = (__nv_bfloat16*)O; a.lse = lse; a.keypad = keypad;
  a.rec = s->line_rec + SPION_MAX_NB; a.pair = s->line_pair + s->line_pair_cap;
  a.L = c->L; a.BH = c->BH; a.nb = vw.nb; a.heads = c->heads; a.by_rank = order_by_rank(c);
  a.scale = c->scale; a.floor_v = keypad ? 0.0f : -100.0f; a.status = c->status_dev;
  return keypad ? fx_launch<D, true>(c, s, mq, mk, mv, a) : fx_launch<D, false>(c, s, mq, mk, mv, a);
}

template <int D>
static int fx_attrs() {
  for (auto k : {k_fwd_exact<D, false>, k_fwd_exact<D, true>})
    SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Fx<D>::SMEM));
  return SPION_OK;
}
int exact_forward_set_attrs(int d) { return d == 64 ? fx_attrs<64>() : fx_attrs<32>(); }

int exact_forward(spion_ctx* c, TcState* s, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const float* keypad, void* O,
                  float* lse) {
  return c->d == 64 ? fx_forward<64>(c, s, mq, mk, mv, keypad, O, lse) : fx_forward<32>(c, s, mq, mk, mv, keypad, O, lse);
}

}  // namespace tc
