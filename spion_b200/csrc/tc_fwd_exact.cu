// Forward on the full mask (the dense warm-up phase; sm_100a, bf16, 64 x 64 blocks, no stored P): two passes over a row, the maximum first, and the
// sums in a fixed order (four chains a half tile), so that O and lse are bit for bit what a two-pass kernel gives.  Some results there
// are sums that cancel to nothing but rounding (the gradient of the key projection's bias is zero in dense attention), so that every other
// order of the additions gives other numbers.
//
// One persistent CTA per SM with four groups.  A group has one service warp (TMA loads, MMA issue) and four arithmetic warps (one per
// tensor-memory quadrant) and walks block rows of its own, two blocks ("a pair") at a time:
//     S = Q K_e^T   (M = 64, the second block at lane offset 16: query rows along the lanes, a row owned by lanes l and l + 16)
//     P = exp2(S scale log2e - m), unnormalised, bf16 into shared memory (over the K tiles when they are as large)
//     O += P V_e    (M = 64, tensor memory, lane offset 16 x parity of the row among the rows with blocks)
// S of pair j + 1 is computed while pair j is in the arithmetic (its 64 values per lane are in registers), and the rows of a
// finished unit are written after the first pair of the next one.  Nothing is exchanged between the groups: they only fill each
// other's waits.  (tc_fwd_stream.cu sums the products of the two blocks of a pair apart, which is faster and another order.)
//
// Every wait is bounded; on a time-out the waiting warp records a code in the status word and the CTA winds down.
#include "tc_stream.cuh"

using namespace tc;

namespace {

constexpr int NG = 4;                                             // groups
constexpr int FS_THREADS = 32 * (4 + 4 * NG);

template <int D> struct Fs {
  using T = OpTile<D>;
  static constexpr bool ALIAS = D == 64;                          // P tiles over the K tiles
  static constexpr uint32_t PB = 2 * VT_BYTES;                    // P tiles of a pair (ALIAS: K tiles first), two buffers
  static constexpr uint32_t O_Q = 0, O_P = T::BYTES, O_V = O_P + 2 * PB, O_K = O_V + 2 * T::BYTES;
  static constexpr uint32_t GROUP = O_K + (ALIAS ? 0 : 2 * T::BYTES);
  static constexpr uint32_t O_BAR = NG * GROUP;
  static constexpr uint32_t GBAR = 112;                           // barriers of a group
  static constexpr size_t SMEM = O_BAR + NG * GBAR + 16 + NG * 64;
  static constexpr uint32_t COLS = 64 + D;                        // tensor-memory columns of a group: S, O
};

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
__global__ void __launch_bounds__(FS_THREADS, 1) k_fwd_exact(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ FsArgs a) {
  using C = Fs<D>;
  using T = OpTile<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);                      // must be 1024-aligned (checked below)
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int grp = warp < 4 ? warp : (warp - 4) >> 2;
  const uint32_t gb = sbase + grp * C::GROUP, bars = sbase + C::O_BAR + grp * C::GBAR;
  // q_full, k_full[2], v_full: tiles landed; s_ready: S of a pair complete; s_free: read out (4 warps); p_ready[2]: P tiles written (4
  // warps); pv_done[2]: O += P V of a pair complete, with every MMA issued before it; pi_full[2]: flags of a pair written
  const uint32_t q_full = bars, k_full = bars + 8, v_full = bars + 24, s_ready = bars + 32, s_free = bars + 40, p_ready = bars + 48,
                 pv_done = bars + 64, pi_full = bars + 80;
  const uint32_t slot = sbase + C::O_BAR + NG * C::GBAR, abort_w = slot + 4;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  volatile int* abort_ptr = reinterpret_cast<volatile int*>(smem_raw + (abort_w - sbase));
  // [2][8]: flags, block columns of the pair, -, penalties of its blocks in base-2 units
  int* info = reinterpret_cast<int*>(smem_raw + (slot - sbase) + 16 + grp * 64);

  if (warp == 0 && lane == 0) {
    int ab = *reinterpret_cast<volatile int*>(a.status);
    if ((sbase & 1023u) != 0u) { report(a.status, ERR_LOAD_WAIT); ab = 1; }
    *abort_ptr = ab;
    for (int g = 0; g < NG; ++g) {
      const uint32_t b = sbase + C::O_BAR + g * C::GBAR;
      for (int x = 0; x < 5; ++x) mbar_init(b + 8 * x, 1);        // q_full, k_full[2], v_full, s_ready
      for (int x = 5; x < 8; ++x) mbar_init(b + 8 * x, 4);        // s_free, p_ready[2]
      for (int x = 8; x < 12; ++x) mbar_init(b + 8 * x, 1);       // pv_done[2], pi_full[2]
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
  const uint32_t tmem = *slot_ptr, tS = tmem + grp * C::COLS, tO = tS + 64u;
  auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool { return warp_wait(bar, parity & 1u, a.status, code); };
  const UnitMap um{a.nb, a.BH, a.by_rank};
  // group g of CTA b walks units b + g G, + NG G, ...
  const int first = (int)blockIdx.x + grp * (int)gridDim.x, step = NG * (int)gridDim.x, total = a.nb * a.BH;

  if (warp < 4) {
    // ================================================================== service warp of a group
    constexpr uint32_t IDESC_S = make_idesc_bf16(64, 64, 0, 0), IDESC_O = make_idesc_bf16(64, D, 0, 1);
    const uint64_t dQ = T::kmajor(gb + C::O_Q, 0);
    Walk c, ld;                                                   // MMAs; loads (a pair ahead)
    c.init(um, a.rec, first, step, total);
    c.skip();
    ld = c;
    int4 pr = ld.valid() ? a.pair[ld.cur.y] : make_int4(0, -1, 0, 0);      // record of the pair whose K tiles are loaded next
    int4 prv = pr;                                                // ... whose V tiles are loaded next
    bool c_val = false, ld_val = false, p_val = false;          // pair of the value pass: c, ld, the pair before c
    Pen4 pen_l = {};
    auto flags_load = [&](const Walk& w, const int4& p) {         // requested with the pair's K tiles, used a pair later
      const int e = lane >> 4, o = e ? p.y : p.x;
      if (KP && o >= 0) pen_load(pen_l, a.keypad + (size_t)w.bh * a.L + o * BS);
    };
    auto load_k = [&](int j) {                                    // K tiles of the pair at `ld` (pair j), Q with the first of a unit
      const uint32_t bar = k_full + 8 * (C::ALIAS ? (j & 1) : 0), dst = gb + (C::ALIAS ? C::O_P + (j & 1) * C::PB : C::O_K);
      const int cnt = ld.cnt();
      const OpPos pos = op_pos(ld.bh, a.L, a.heads, D);
      const bool with_q = ld.k == 0 && !ld_val;
      if (lane == 0) {
        mbar_expect_tx(bar, cnt * T::BYTES);
        if (with_q) mbar_expect_tx(q_full, T::BYTES);
      }
      __syncwarp();
      if (lane < cnt) tma_load_2d(dst + lane * T::BYTES, &tmK, bar, pos.x0, pos.row0 + (lane ? pr.y : pr.x) * BS);
      if (lane == 4 && with_q) tma_load_2d(gb + C::O_Q, &tmQ, q_full, pos.x0, pos.row0 + ld.cur.x * BS);
    };
    auto load_v = [&](const Walk& w) {
      const int cnt = w.cnt();
      const OpPos pos = op_pos(w.bh, a.L, a.heads, D);
      if (lane == 0) mbar_expect_tx(v_full, cnt * T::BYTES);
      __syncwarp();
      if (lane < cnt) tma_load_2d(gb + C::O_V + lane * T::BYTES, &tmV, v_full, pos.x0, pos.row0 + (lane ? prv.y : prv.x) * BS);
    };
    // the pairs of a unit come twice, for the maximum and for the values
    auto step_on = [&](Walk& w, bool& values) {
      if (w.last() && !values) { values = true; w.k = 0; return; }
      const bool end = w.last();
      w.next();
      if (end) values = false;
    };
    bool ok = true;
    int units = 0, jv = 0;                                        // units with blocks begun; value pairs before pair j
    if (c.valid()) {
      flags_load(ld, pr);
      load_k(0);
      prv = pr;
      if (ld_val) load_v(ld);
      step_on(ld, ld_val);
      if (ld.valid()) pr = a.pair[ld.cur.y + ld.k];
    }
    int p_cnt = 0, p_par = 0;                                     // the pair before c
    bool p_first = false;
    for (int j = 0; ok; ++j) {
      const bool have = c.valid();
      if (have) {
        if (KP) {                                                 // flags of pair j: its buffer was read before P of pair j - 2 was written
          uint32_t mixed = 0u;
          const float pen = pen_of(pen_l, mixed) * LOG2E, pen1 = __shfl_sync(0xffffffffu, pen, 16);
          if (lane == 0) {
            int* x = info + 8 * (j & 1);
            x[0] = (int)mixed;
            x[1] = prv.x; x[2] = prv.y;
            x[4] = __float_as_int(pen); x[5] = __float_as_int(pen1);
            mbar_arrive(pi_full + 8 * (j & 1));
          }
          __syncwarp();
        }
        // S of pair j
        const int kb = C::ALIAS ? (j & 1) : 0, ku = C::ALIAS ? (j >> 1) : j;
        if (c.k == 0 && !c_val) { if (!wait_all(q_full, (uint32_t)units, ERR_LOAD_WAIT)) { ok = false; break; } ++units; }
        if (!wait_all(k_full + 8 * kb, (uint32_t)ku, ERR_LOAD_WAIT)) { ok = false; break; }
        if (j >= 1 && !wait_all(s_free, (uint32_t)(j - 1), ERR_MMA_WAIT)) { ok = false; break; }
        const bool two = warp_uniform(c.cnt() == 2);
        if (elect_one()) {
          tc_fence_after();
          const uint64_t dK = T::kmajor(gb + (C::ALIAS ? C::O_P + kb * C::PB : C::O_K), 0);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_bf16(tS, desc_advance(dQ, kk * T::K_STEP), desc_advance(dK, kk * T::K_STEP), IDESC_S, kk > 0);
          if (two) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              mma_bf16(tS + (16u << 16), desc_advance(dQ, kk * T::K_STEP), desc_advance(dK, T::BYTES + kk * T::K_STEP), IDESC_S, kk > 0);
          }
          mma_commit(s_ready);
        }
        __syncwarp();
      }
      if (j >= 1) {                                               // O += P V of pair j - 1
        const int jp = j - 1;
        if (!wait_all(p_ready + 8 * (jp & 1), (uint32_t)(jp >> 1), ERR_MMA_WAIT)) { ok = false; break; }
        if (p_val) { if (!wait_all(v_full, (uint32_t)jv, ERR_LOAD_WAIT)) { ok = false; break; } ++jv; }
        const bool two = warp_uniform(p_cnt == 2), fresh = warp_uniform((int)p_first) != 0, value_pair = warp_uniform((int)p_val) != 0;
        if (elect_one()) {
          tc_fence_after();
          const uint32_t acc = tO + ((uint32_t)(p_par * 16) << 16);
          const uint64_t dP = ValTile::kmajor(gb + C::O_P + (jp & 1) * C::PB, 0), dV = T::mnmajor(gb + C::O_V, 0);
          if (value_pair) {                                       // else nothing to multiply: the commit alone says that S has been read
#pragma unroll
          for (int kk = 0; kk < BS / 16; ++kk)
            mma_bf16(acc, desc_advance(dP, kk * ValTile::K_STEP), desc_advance(dV, kk * T::MN_STEP), IDESC_O, (kk > 0 || !fresh) ? 1u : 0u);
          if (two) {
#pragma unroll
            for (int kk = 0; kk < BS / 16; ++kk)
              mma_bf16(acc, desc_advance(dP, VT_BYTES + kk * ValTile::K_STEP), desc_advance(dV, T::BYTES + kk * T::MN_STEP), IDESC_O, 1u);
          }
          }
          mma_commit(pv_done + 8 * (jp & 1));
        }
        __syncwarp();
      }
      if (!have) break;
      // Loads.  O += P V of pair j - 1 complete implies S of pair j (issued before it): K (its own buffer, or the P buffer of
      // pair j - 1), Q and V are free.
      if (j >= 1) {
        if (!wait_all(pv_done + 8 * ((j - 1) & 1), (uint32_t)((j - 1) >> 1), ERR_MMA2_WAIT)) { ok = false; break; }
        if (c_val) load_v(c);                                     // V of pair j (pair 0's was requested above)
      } else if (!wait_all(s_ready, 0u, ERR_MMA_WAIT)) { ok = false; break; }
      if (ld.valid()) {
        flags_load(ld, pr);
        load_k(j + 1);
        prv = pr;
        step_on(ld, ld_val);
        if (ld.valid()) pr = a.pair[ld.cur.y + ld.k];
      }
      p_cnt = c.cnt(); p_par = units & 1; p_first = c.k == 0; p_val = c_val;
      step_on(c, c_val);
    }
  } else {
    // ================================================================== arithmetic warps of a group
    const int q = warp & 3, hf = lane >> 4, row = q * 16 + (lane & 15);
    const uint32_t lS = tS + ((uint32_t)(q * 32) << 16), lO = tO + ((uint32_t)(q * 32) << 16);
    const float sc2 = a.scale * LOG2E, floor2 = a.floor_v * LOG2E, inv_scale = 1.0f / a.scale;
    bool ok = true;
    // the finished unit whose rows are still in tensor memory
    bool pend = false;
    int pend_par = 0, pend_j = 0;
    float pend_inv = 0.f;
    __nv_bfloat16* pend_dst = nullptr;
    auto write_rows = [&](__nv_bfloat16* dst, bool have, float inv, bool mine) {
#pragma unroll
      for (int h = 0; h < D / 32; ++h) {
        uint32_t v[32];
        if (have) {
          tmem_ld32(lO + h * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int x = 0; x < 32; ++x) v[x] = 0u;
        }
        if (mine) {
#pragma unroll
          for (int x = 0; x < 32; x += 8)
            *reinterpret_cast<uint4*>(dst + h * 32 + x) = make_uint4(pack_bf16(__uint_as_float(v[x]) * inv, __uint_as_float(v[x + 1]) * inv),
                                                                     pack_bf16(__uint_as_float(v[x + 2]) * inv, __uint_as_float(v[x + 3]) * inv),
                                                                     pack_bf16(__uint_as_float(v[x + 4]) * inv, __uint_as_float(v[x + 5]) * inv),
                                                                     pack_bf16(__uint_as_float(v[x + 6]) * inv, __uint_as_float(v[x + 7]) * inv));
        }
      }
    };
    auto flush = [&]() -> bool {
      if (!wait_all(pv_done + 8 * (pend_j & 1), (uint32_t)(pend_j >> 1), ERR_MMA2_WAIT)) return false;
      tc_fence_after();
      write_rows(pend_dst, true, pend_inv, hf == pend_par);
      tc_fence_before();
      pend = false;
      return true;
    };
    Walk u;
    u.init(um, a.rec, first, step, total);
    int j = 0;
    // Units with blocks begun.  Two of them in a row must not share their lanes: the rows of the first are read while the product of
    // the second is issued.  Rows without blocks have no product and hand nothing over, so they do not count.
    int units = 0;
    for (; u.valid() && ok; u.shift()) {
      const int n = u.cur.w;
      const OpPos pos = op_pos(u.bh, a.L, a.heads, D);
      __nv_bfloat16* dst = a.O + (size_t)(pos.row0 + u.cur.x * BS + row) * pos.ld + pos.x0;
      float* lse = a.lse + (size_t)u.bh * a.L + u.cur.x * BS + row;
      if (n == 0) {                                               // a row without blocks: every key counts as score 0
        const float m0 = fmaxf(floor2, -INFINITY);
        if (hf == 0) *lse = m0 + log2f((float)a.L * exp2f(-m0));
        write_rows(dst, false, 0.f, hf == 0);
        continue;
      }
      const int par = ++units & 1;
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
          if (!wait_all(pi_full + 8 * (j & 1), (uint32_t)(j >> 1), ERR_MMA_WAIT)) { ok = false; break; }
          const int* x = info + 8 * (j & 1);
          const int f = x[0];
          const bool mixed = (f >> hf) & 1;
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
        // the P tiles of pair j - 2 have been consumed
        if (j >= 2 && !wait_all(pv_done + 8 * (j & 1), (uint32_t)(j >> 1) - 1u, ERR_MMA2_WAIT)) { ok = false; break; }
        const uint32_t tile = gb + C::O_P + (j & 1) * C::PB + hf * VT_BYTES + row * 128;
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
        if (mine && values) {
          half_row(v0, 0);
          half_row(v1, 1);
        }
        fence_proxy_async();                                      // P rows -> visible to the MMA
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready + 8 * (j & 1));
        if (pend) ok = flush();                                   // the previous unit: its last product has long been issued
      }
      if (!ok) break;
      n_sel += __shfl_xor_sync(0xffffffffu, n_sel, 16);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      const float z = l + (float)(a.L - n_sel) * exp2f(-mx);
      if (hf == 0) *lse = mx + log2f(z);
      pend = true; pend_par = par; pend_j = j - 1; pend_inv = 1.0f / z; pend_dst = dst;
    }
    if (ok && pend) flush();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512u);
}

}  // namespace

namespace tc {

template <int D, bool KP>
static int fx_launch(spion_ctx* c, TcState* s, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const FsArgs& a) {
  using C = Fs<D>;
  static_assert(C::SMEM <= 227 * 1024 && NG * C::COLS <= 512, "shared or tensor memory");
  const long long total = (long long)c->BH * a.nb;
  const int grid = (int)(total < (long long)s->sms ? total : (long long)s->sms);       // one CTA per SM (all 512 TMEM columns)
  k_fwd_exact<D, KP><<<grid, FS_THREADS, C::SMEM, c->stream>>>(mq, mk, mv, a);
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
    SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Fs<D>::SMEM));
  return SPION_OK;
}
int exact_forward_set_attrs(int d) { return d == 64 ? fx_attrs<64>() : fx_attrs<32>(); }

int exact_forward(spion_ctx* c, TcState* s, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const float* keypad, void* O,
                  float* lse) {
  return c->d == 64 ? fx_forward<64>(c, s, mq, mk, mv, keypad, O, lse) : fx_forward<32>(c, s, mq, mk, mv, keypad, O, lse);
}

}  // namespace tc
