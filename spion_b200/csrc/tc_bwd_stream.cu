// Backward of the block-sparse attention without P or dS in global memory, as two streaming pipelines (sm_100a, bf16,
// 64 x 64 blocks).  With the forward's log-sum-exp, lse2_i = m_i log2(e) + log2(Z_i) (Z_i includes the reference's term for the
// non-selected keys, models/block_attn.cu:65-71),
//     P_ij  = exp2(s_ij scale log2(e) - pad_j log2(e) - lse2_i)                      (:72-87)
//     dS_ij = P_ij (dP_ij - delta_i) scale,   delta_i = sum_n dO_in O_in             (:107-129)
// are functions of Q, K, V, dO, O alone:
//   ROW   dQ[r] = sum_c dS(r,c) K[c], and delta                           unit: a block row;    streamed: K[c], V[c]
//   COL   dK[c] = sum_r dS(r,c)^T Q[r],  dV[c] = sum_r P(r,c)^T dO[r]     unit: a block column; streamed: Q[r], dO[r]
// Both are one kernel: a unit has two fixed tiles F0, F1 (COL: K[c], V[c]; ROW: Q[r], dO[r]) and streams the tiles A0, A1 of its
// entries two entries ("a pair") at a time:
//     S, dP    COL: [Q0; Q1] K^T and [dO0; dO1] V^T as one 128-row product each; ROW: Q K_e^T and dO V_e^T, the second entry at
//              lane offset 16: query rows along the lanes in both, so that lse and delta are one register each
//     accumulators += dS^T Q, P^T dO (COL),  += dS K (ROW)
// One persistent CTA per SM, 640 threads:
//   warp 0   loads: pairs in stream order into a ring of slots, the fixed tiles of a unit into one of two sets (TMA)
//   warp 1   S / dP products into one of three tensor-memory sets, up to two pairs ahead of the arithmetic
//   warp 2   second products, when the tiles of a pair are written
//   warp 3   lse and -delta scale of the next pair's (COL) or unit's (ROW) query rows into shared memory, which blocks have padded
//            keys
//   warps 4-19   arithmetic, two groups of eight: even and odd pairs; each warp one tensor-memory quadrant and half of the columns.
//            Two groups because the chain of one pair (tensor-memory load, exponentials, tile store, proxy fence, hand-over) is
//            about three times as long as its instructions take to issue.  ROW: they form delta first, while the first tiles
//            arrive, and leave it in global memory, for COL too.
// What bounds it: per pair at head_dim 64 the tensor pipe needs 920 (COL) or 660 cycles (ROW), the exponentials 512.
// Measured, rows + columns, against the backward from stored P of tc_engine.cu: 64 matrices, d 64: L = 4096, 5 % 168 us (stored 155,
// its forward 25 slower), 30 % 458 (stored path 906 with its forward); L = 16384, 5 % 1271 (2610); 256 matrices, L = 4096,
// d 32, 10 %, padded keys 791 (1413).  Which of the two serves a mask: _recompute_pays in native.py.
//
// Every wait is bounded; on a time-out the waiting warp records a code in the status word and the CTA winds down.
#include "tc_stream.cuh"

using namespace tc;

namespace {

constexpr int BW_THREADS = 640;
constexpr int COL = 0, ROW = 1;

template <int D, int SIDE> struct Bw {
  using T = OpTile<D>;
  static constexpr int NP = (D == 64) ? 4 : 8;                        // pair slots
  static constexpr uint32_t SLOT = 4 * T::BYTES;                      // A0 of both entries, A1 of both entries
  static constexpr uint32_t FIX = 2 * T::BYTES;                       // F0, F1; two sets
  static constexpr uint32_t PD = (SIDE == COL ? 4 : 2) * VT_BYTES;    // value tiles of a pair: dS of both entries, then P of both
  static constexpr uint32_t O_FIX = NP * SLOT, O_PD = O_FIX + 2 * FIX, O_BAR = O_PD + 2 * PD;
  // per parity of the pair: {pad flags and submasks of the two entries, their lines}, and in COL lse, -delta scale of their 128
  // query rows; ROW: those of the unit's 64 rows per parity of the unit
  static constexpr uint32_t O_INFO = O_BAR + 352, O_STAT = O_INFO + 32;
  static constexpr uint32_t ROWS = SIDE == COL ? 128 : 64;
  static constexpr size_t SMEM = O_STAT + 2 * 2 * ROWS * 4;
};

struct BwArgs {
  const float *lse, *delta, *keypad;         // [BH*L]; delta: COL only; keypad may be null
  float* delta_out;                          // ROW
  const __nv_bfloat16 *O, *dO;               // ROW: for delta
  __nv_bfloat16 *out0, *out1;                // dK (COL) or dQ (ROW); dV (COL)
  const int4 *rec, *pair;                    // lines and pairs (k_line_recs)
  const uint8_t* submask;
  int L, BH, nb, heads, by_rank;
  float scale;
  int* status;
};

template <int D, int SIDE, bool SUB>
__global__ void __launch_bounds__(BW_THREADS, 1) k_bwd_stream(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                                                              const __grid_constant__ CUtensorMap tmF0, const __grid_constant__ CUtensorMap tmF1,
                                                              const __grid_constant__ BwArgs a) {
  using C = Bw<D, SIDE>;
  using T = OpTile<D>;
  constexpr int NP = C::NP;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);                          // must be 1024-aligned (checked below)
  const uint32_t bars = sbase + C::O_BAR;
  // pfull / pdone[slot]: tiles landed / second products that read the slot retired; s_ready / t_free[3]: S and dP of a pair in
  // tensor memory / read out (8 warps); p_ready[2]: value tiles of a pair written (8 warps); acc_done / acc_free[2]: a unit's
  // accumulators complete / read out (8 warps); f_full / f_free[2]: fixed tiles landed / no longer read; pi_full / pi_free[2]:
  // what warp 3 wrote for a pair is there / has been read (8 warps); st_full / st_free[2]: ROW, the same for a unit (16 warps)
  const uint32_t pfull = bars, pdone = bars + 64, s_ready = bars + 128, t_free = bars + 152, p_ready = bars + 176, acc_done = bars + 192,
                 acc_free = bars + 208, f_full = bars + 224, f_free = bars + 240, st_full = bars + 256, st_free = bars + 272,
                 pi_full = bars + 288, pi_free = bars + 304, slot = bars + 320, abort_w = bars + 324;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  volatile int* abort_ptr = reinterpret_cast<volatile int*>(smem_raw + (abort_w - sbase));

  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int G = (int)gridDim.x, total = a.nb * a.BH;
  const UnitMap um{a.nb, a.BH, a.by_rank};
  constexpr uint32_t ACC = 384u;                                      // three S / dP sets of 128 columns, two accumulator sets of 64

  if (warp == 0 && lane == 0) {
    int ab = *reinterpret_cast<volatile int*>(a.status);
    if ((sbase & 1023u) != 0u) { report(a.status, ERR_LOAD_WAIT); ab = 1; }
    *abort_ptr = ab;
    for (int i = 0; i < NP; ++i) { mbar_init(pfull + 8 * i, 1); mbar_init(pdone + 8 * i, 1); }
    for (int i = 0; i < 3; ++i) { mbar_init(s_ready + 8 * i, 1); mbar_init(t_free + 8 * i, 8); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(p_ready + 8 * i, 8);
      mbar_init(acc_done + 8 * i, 1);
      mbar_init(acc_free + 8 * i, 8);
      mbar_init(f_full + 8 * i, 1);
      mbar_init(f_free + 8 * i, 1);
      mbar_init(st_full + 8 * i, 1);
      mbar_init(st_free + 8 * i, 16);
      mbar_init(pi_full + 8 * i, 1);
      mbar_init(pi_free + 8 * i, 8);
    }
    fence_barrier_init();
  }
  __syncthreads();
  if (*abort_ptr != 0) return;
  if (warp == 1) {
    tmem_alloc(slot, 512u);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool { return warp_wait(bar, parity & 1u, a.status, code); };
  Walk c;
  c.init(um, a.rec, (int)blockIdx.x, G, total);

  if (warp == 0) {
    // ================================================================== loads
    bool ok = true;
    int loads0 = 0, loads1 = 0;                                       // units whose fixed tiles went to set 0 / 1
    c.skip();
    // lane l keeps the record of pair l of the current unit and of the next one, both requested a unit early
    int4 prs = make_int4(0, -1, 0, 0), prs_n = prs;
    int cached_i = -1;
    for (int j = 0; ok && c.valid(); ++j, c.next()) {
      const int ps = j % NP;
      if (c.i != cached_i) {
        prs = (cached_i >= 0 && c.i == cached_i + 1) ? prs_n : (lane < c.pairs() ? a.pair[c.cur.y + lane] : prs);
        cached_i = c.i;
        if (c.i + 1 < c.n_my && lane < c.nxt.z) prs_n = a.pair[c.nxt.y + lane];
      }
      int4 pr;
      if (c.k < 32) {
        pr.x = __shfl_sync(0xffffffffu, prs.x, c.k);
        pr.y = __shfl_sync(0xffffffffu, prs.y, c.k);
      } else {
        pr = a.pair[c.cur.y + c.k];
      }
      if (j >= NP && !wait_all(pdone + 8 * ps, (uint32_t)(j / NP - 1), ERR_MMA2_WAIT)) { ok = false; break; }
      const int par = c.i & 1;
      if (c.k == 0) {
        const int loads = par ? loads1 : loads0;
        if (loads >= 1 && !wait_all(f_free + 8 * par, (uint32_t)(loads - 1), ERR_MMA2_WAIT)) { ok = false; break; }
      }
      const int cnt = c.cnt();
      const OpPos pos = op_pos(c.bh, a.L, a.heads, D);
      if (lane == 0) {
        mbar_expect_tx(pfull + 8 * ps, 2 * cnt * T::BYTES);
        if (c.k == 0) mbar_expect_tx(f_full + 8 * par, 2 * T::BYTES);
      }
      __syncwarp();
      if (c.k == 0) {
        const uint32_t f = sbase + C::O_FIX + par * C::FIX;
        if (lane == 4) tma_load_2d(f, &tmF0, f_full + 8 * par, pos.x0, pos.row0 + c.cur.x * BS);
        if (lane == 5) tma_load_2d(f + T::BYTES, &tmF1, f_full + 8 * par, pos.x0, pos.row0 + c.cur.x * BS);
        if (par) ++loads1; else ++loads0;
      }
      if (lane < 2 * cnt) {
        const int e = lane >> 1;
        const int orow = pos.row0 + (e ? pr.y : pr.x) * BS;
        const uint32_t dst = sbase + ps * C::SLOT + ((lane & 1) * 2 + e) * T::BYTES;
        if (lane & 1) tma_load_2d(dst, &tmA1, pfull + 8 * ps, pos.x0, orow);
        else tma_load_2d(dst, &tmA0, pfull + 8 * ps, pos.x0, orow);
      }
    }
  } else if (warp == 1) {
    // ================================================================== S and dP
    constexpr uint32_t IDESC = make_idesc_bf16(SIDE == COL ? 128 : 64, 64, 0, 0);
    const uint64_t KM = T::kmajor(sbase, 0);
    bool ok = true;
    int waits0 = 0, waits1 = 0;
    c.skip();
    for (int j = 0; ok && c.valid(); ++j, c.next()) {
      const int ps = j % NP, set = j % 3, par = c.i & 1;
      if (j >= 3 && !wait_all(t_free + 8 * set, (uint32_t)(j / 3 - 1), ERR_MMA_WAIT)) { ok = false; break; }
      if (c.k == 0) {
        const int w = par ? waits1 : waits0;
        if (!wait_all(f_full + 8 * par, (uint32_t)w, ERR_LOAD_WAIT)) { ok = false; break; }
        if (par) ++waits1; else ++waits0;
      }
      if (!wait_all(pfull + 8 * ps, (uint32_t)(j / NP), ERR_LOAD_WAIT)) { ok = false; break; }
      const bool last = warp_uniform((int)c.last()) != 0, two = warp_uniform(c.cnt()) == 2;
      if (elect_one()) {
        tc_fence_after();
        const uint64_t a0 = desc_advance(KM, ps * C::SLOT), a1 = desc_advance(a0, 2 * T::BYTES);
        const uint64_t f0 = desc_advance(KM, C::O_FIX + par * C::FIX), f1 = desc_advance(f0, T::BYTES);
        const uint32_t d0 = tmem + (uint32_t)set * 128u;
        if (SIDE == COL) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_bf16(d0, desc_advance(a0, kk * T::K_STEP), desc_advance(f0, kk * T::K_STEP), IDESC, kk > 0);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_bf16(d0 + 64u, desc_advance(a1, kk * T::K_STEP), desc_advance(f1, kk * T::K_STEP), IDESC, kk > 0);
        } else {
          auto products = [&](int e) {
            const uint32_t de = d0 + ((uint32_t)(e * 16) << 16);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              mma_bf16(de, desc_advance(f0, kk * T::K_STEP), desc_advance(a0, e * T::BYTES + kk * T::K_STEP), IDESC, kk > 0);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              mma_bf16(de + 64u, desc_advance(f1, kk * T::K_STEP), desc_advance(a1, e * T::BYTES + kk * T::K_STEP), IDESC, kk > 0);
          };
          products(0);
          if (two) products(1);
        }
        mma_commit(s_ready + 8 * set);
        if (last) mma_commit(f_free + 8 * par);                       // the fixed tiles are read by these products only
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    // ================================================================== second products
    constexpr uint32_t IDESC = make_idesc_bf16(64, D, SIDE == COL ? 1 : 0, 1);
    constexpr uint32_t V_STEP = SIDE == COL ? ValTile::MN_STEP : ValTile::K_STEP;
    const uint64_t MN = T::mnmajor(sbase, 0), VT = SIDE == COL ? ValTile::mnmajor(sbase, 0) : ValTile::kmajor(sbase, 0);
    bool ok = true;
    int uses0 = 0, uses1 = 0;
    c.skip();
    for (int j = 0; ok && c.valid(); ++j, c.next()) {
      const int ps = j % NP, set = j & 1, par = c.i & 1;
      const int uses = par ? uses1 : uses0;
      if (c.k == 0 && uses >= 1 && !wait_all(acc_free + 8 * par, (uint32_t)(uses - 1), ERR_MMA2_WAIT)) { ok = false; break; }
      if (!wait_all(p_ready + 8 * set, (uint32_t)(j >> 1), ERR_MMA_WAIT)) { ok = false; break; }
      const bool last = warp_uniform((int)c.last()) != 0, two = warp_uniform(c.cnt()) == 2, fresh = warp_uniform(c.k) == 0;
      if (elect_one()) {
        tc_fence_after();
        const uint32_t acc = tmem + ACC + (uint32_t)par * 64u;
        const uint64_t vt = desc_advance(VT, C::O_PD + set * C::PD), b0 = desc_advance(MN, ps * C::SLOT);
        auto products = [&](int e, bool first) {
#pragma unroll
          for (int kk = 0; kk < BS / 16; ++kk)                        // dK or dQ (lanes 0-15 of every quadrant)
            mma_bf16(acc, desc_advance(vt, e * VT_BYTES + kk * V_STEP), desc_advance(b0, e * T::BYTES + kk * T::MN_STEP), IDESC,
                     (kk > 0) ? 1u : (first ? 0u : 1u));
          if (SIDE == COL) {
#pragma unroll
            for (int kk = 0; kk < BS / 16; ++kk)                      // dV (lanes 16-31)
              mma_bf16(acc + (16u << 16), desc_advance(vt, (2 + e) * VT_BYTES + kk * V_STEP),
                       desc_advance(b0, (2 + e) * T::BYTES + kk * T::MN_STEP), IDESC, (kk > 0) ? 1u : (first ? 0u : 1u));
          }
        };
        products(0, fresh);
        if (two) products(1, false);
        mma_commit(pdone + 8 * ps);
        if (last) mma_commit(acc_done + 8 * par);
      }
      __syncwarp();
      if (last) { if (par) ++uses1; else ++uses0; }
    }
  } else if (warp == 3) {
    // ================================================================== statistics and flags for the arithmetic warps
    if (SIDE == ROW) asm volatile("bar.sync 1, 544;" ::: "memory");   // delta of this CTA's rows is in global memory
    bool ok = true;
    int sets0 = 0, sets1 = 0;
    int j = 0;
    int4 pr = make_int4(0, -1, 0, 0);
    for (; ok && c.valid(); c.shift()) {
      const int par = c.i & 1;
      const bool used = c.cur.w > 0;
      const size_t base = (size_t)c.bh * a.L;
      const float* kpu = a.keypad ? a.keypad + base : nullptr;
      if (used) pr = a.pair[c.cur.y];
      int unit_pad = 0;
      if (SIDE == COL) {
        if (used && kpu) unit_pad = __any_sync(0xffffffffu, pad4(kpu + c.cur.x * BS));
      } else {
        float dl[2], hh[2];                                           // rows lane and lane + 32
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const size_t ri = base + (size_t)c.cur.x * BS + lane + 32 * x;
          dl[x] = *reinterpret_cast<volatile float*>(a.delta_out + ri);       // written by this CTA
          hh[x] = a.lse[ri];
        }
        if (used) {
          const int sets = par ? sets1 : sets0;
          if (sets >= 1 && !wait_all(st_free + 8 * par, (uint32_t)(sets - 1), ERR_MMA_WAIT)) { ok = false; break; }
          float* st = reinterpret_cast<float*>(smem_raw + C::O_STAT) + par * 2 * 64;
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            st[lane + 32 * x] = hh[x];
            st[64 + lane + 32 * x] = -dl[x] * a.scale;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(st_full + 8 * par);
          if (par) ++sets1; else ++sets0;
        }
      }
      const int np = c.pairs();
      for (int k = 0; ok && k < np; ++k, ++j) {
        // lanes 0-15: first entry, 16-31: second; four query rows (COL) or keys (ROW) each
        const int e = lane >> 4, o = e ? pr.y : pr.x, blk = e ? pr.w : pr.z;
        const size_t ri = base + (size_t)max(o, 0) * BS;
        float h4[4] = {0.f, 0.f, 0.f, 0.f}, d4[4] = {0.f, 0.f, 0.f, 0.f};
        int pad = unit_pad;
        if (SIDE == COL) {
          if (o >= 0) {
#pragma unroll
            for (int x = 0; x < 4; ++x) { h4[x] = a.lse[ri + (lane & 15) + 16 * x]; d4[x] = a.delta[ri + (lane & 15) + 16 * x]; }
          }
        } else if (kpu) {
          const uint32_t any = __ballot_sync(0xffffffffu, o >= 0 && pad4(a.keypad + ri));
          pad = ((any & 0xffffu) ? 1 : 0) | ((any >> 16) ? 2 : 0);
        }
        const int sub = SUB && o >= 0 ? a.submask[blk] : 0xff;
        const int4 pr_next = k + 1 < np ? a.pair[c.cur.y + k + 1] : pr;
        if (j >= 2 && !wait_all(pi_free + 8 * (j & 1), (uint32_t)((j >> 1) - 1), ERR_MMA_WAIT)) { ok = false; break; }
        int* info = reinterpret_cast<int*>(smem_raw + C::O_INFO) + 4 * (j & 1);
        const int sub1 = __shfl_sync(0xffffffffu, sub, 16);
        if (lane == 0) { info[0] = pad | (sub << 8) | (sub1 << 16); info[1] = pr.x; info[2] = pr.y; }
        if (SIDE == COL) {
          float* st = reinterpret_cast<float*>(smem_raw + C::O_STAT) + (j & 1) * 2 * 128 + e * 64 + (lane & 15);
#pragma unroll
          for (int x = 0; x < 4; ++x) { st[16 * x] = h4[x]; st[128 + 16 * x] = -d4[x] * a.scale; }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(pi_full + 8 * (j & 1));
        pr = pr_next;
      }
    }
  } else {
    // ================================================================== arithmetic
    const int mw = warp - 4, q = warp & 3, g = (mw >> 2) & 1, grp = mw >> 3;
    if (SIDE == ROW) {
      // delta = rowsum(dO.O) of all rows of this CTA, four units of loads in flight: D / 8 lanes per row, 16 bytes each
      constexpr int LPR = D / 8, RPW = 32 / LPR, UN = 4;
      static_assert(16 * RPW >= BS, "rows of a unit");
      const int r0 = mw * RPW + lane / LPR;
      for (int i0 = 0; i0 < c.n_my; i0 += UN) {
        uint4 u[UN], v[UN];
        size_t ri[UN];
#pragma unroll
        for (int x = 0; x < UN; ++x) {
          u[x] = v[x] = make_uint4(0, 0, 0, 0);
          ri[x] = 0;
          if (i0 + x < c.n_my && r0 < BS) {
            int bh, rank;
            um.at((int)blockIdx.x + (i0 + x) * G, bh, rank);
            const int line = a.rec[rank].x;
            const OpPos pos = op_pos(bh, a.L, a.heads, D);
            const size_t off = (size_t)(pos.row0 + line * BS + r0) * pos.ld + pos.x0 + (lane % LPR) * 8;
            u[x] = *reinterpret_cast<const uint4*>(a.dO + off);
            v[x] = *reinterpret_cast<const uint4*>(a.O + off);
            ri[x] = (size_t)bh * a.L + line * BS + r0;
          }
        }
#pragma unroll
        for (int x = 0; x < UN; ++x) {
          const float t = bf16_lo(u[x].x) * bf16_lo(v[x].x) + bf16_hi(u[x].x) * bf16_hi(v[x].x) + bf16_lo(u[x].y) * bf16_lo(v[x].y) +
                          bf16_hi(u[x].y) * bf16_hi(v[x].y) + bf16_lo(u[x].z) * bf16_lo(v[x].z) + bf16_hi(u[x].z) * bf16_hi(v[x].z) +
                          bf16_lo(u[x].w) * bf16_lo(v[x].w) + bf16_hi(u[x].w) * bf16_hi(v[x].w);
          // half of the head dimension in order, then the two halves: as the row kernel of the stored path adds them
          float half = __shfl_sync(0xffffffffu, t, lane & ~(LPR / 2 - 1));
#pragma unroll
          for (int y = 1; y < LPR / 2; ++y) half += __shfl_sync(0xffffffffu, t, (lane & ~(LPR / 2 - 1)) + y);
          const float d = half + __shfl_xor_sync(0xffffffffu, half, LPR / 2);
          if (lane % LPR == 0 && i0 + x < c.n_my && r0 < BS) a.delta_out[ri[x]] = d;
        }
      }
      __threadfence_block();
      asm volatile("bar.sync 1, 544;" ::: "memory");                  // with warp 3, which hands delta out
    }
    // entry of the pair and query row of this lane: COL rows 0-63 first entry, 64-127 second; ROW second entry in lanes 16-31
    const int es = SIDE == COL ? q >> 1 : lane >> 4;
    const int row = SIDE == COL ? (q & 1) * 32 + lane : q * 16 + (lane & 15);
    const int orow = q * 16 + (lane & 15);                            // output row (64-row accumulators)
    const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16);
    const float sc2 = a.scale * LOG2E, inv_scale = 1.0f / a.scale;
    bool ok = true;
    bool pend = false;                                                // a finished unit whose rows this group has to write
    int pend_par = 0, pend_phase = 0;
    __nv_bfloat16* pend_dst = nullptr;
    int done0 = 0, done1 = 0;                                         // units that went to accumulator set 0 / 1

    auto write_rows = [&](__nv_bfloat16* dst, uint32_t taddr, bool have, bool mine) {
      constexpr int W = D / 2;
      uint32_t v[W];
      if (have) {
        if constexpr (W == 32) tmem_ld32(taddr + g * W, v); else tmem_ld16(taddr + g * W, v);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int e = 0; e < W; ++e) v[e] = 0u;
      }
      if (!mine) return;
#pragma unroll
      for (int e = 0; e < W; e += 8)
        *reinterpret_cast<uint4*>(dst + e) = make_uint4(pack_bf16(__uint_as_float(v[e]), __uint_as_float(v[e + 1])),
                                                        pack_bf16(__uint_as_float(v[e + 2]), __uint_as_float(v[e + 3])),
                                                        pack_bf16(__uint_as_float(v[e + 4]), __uint_as_float(v[e + 5])),
                                                        pack_bf16(__uint_as_float(v[e + 6]), __uint_as_float(v[e + 7])));
    };
    const bool writes = SIDE == COL || lane < 16;
    auto flush = [&]() -> bool {
      if (!wait_all(acc_done + 8 * pend_par, (uint32_t)pend_phase, ERR_MMA2_WAIT)) return false;
      tc_fence_after();
      write_rows(pend_dst, t_lane + ACC + (uint32_t)pend_par * 64u, true, writes);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free + 8 * pend_par);
      pend = false;
      return true;
    };

    int j = 0;
    int stat_waits0 = 0, stat_waits1 = 0;
    for (; c.valid() && ok; c.shift()) {
      const int i = c.i, n = c.cur.w, par = i & 1;
      const OpPos pos = op_pos(c.bh, a.L, a.heads, D);
      __nv_bfloat16* dst = (SIDE == COL && lane >= 16 ? a.out1 : a.out0) + (size_t)(pos.row0 + c.cur.x * BS + orow) * pos.ld + pos.x0 + g * (D / 2);
      if (n == 0) {                                                   // a unit without entries: zero rows
        if (grp == (i & 1)) write_rows(dst, 0u, false, writes);
        continue;
      }
      const int npairs = c.pairs();
      const float* kpu = a.keypad + (size_t)c.bh * a.L + g * 32;
      float h = 0.f, nds = 0.f;
      if (SIDE == ROW) {
        const int w = par ? stat_waits1 : stat_waits0;
        if (!wait_all(st_full + 8 * par, (uint32_t)w, ERR_MMA_WAIT)) { ok = false; break; }
        if (par) ++stat_waits1; else ++stat_waits0;
        const float* st = reinterpret_cast<const float*>(smem_raw + C::O_STAT) + par * 2 * 64;
        h = st[row]; nds = st[64 + row];
        __syncwarp();
        if (lane == 0) mbar_arrive(st_free + 8 * par);
      }
      for (int k = 0; k < npairs && ok; ++k, ++j) {
        if ((j & 1) != grp) continue;
        if (!wait_all(pi_full + 8 * grp, (uint32_t)(j >> 1), ERR_MMA_WAIT)) { ok = false; break; }
        const bool mine = 2 * k + es < n;
        const int* info = reinterpret_cast<const int*>(smem_raw + C::O_INFO) + 4 * grp;
        const int flags = info[0], oth = info[1 + es];
        if (SIDE == COL) {
          const float* st = reinterpret_cast<const float*>(smem_raw + C::O_STAT) + grp * 2 * 128 + es * 64 + row;
          h = st[0]; nds = st[128];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(pi_free + 8 * grp);
        // blocks without padded keys (most of them) take no penalty; columns are keys in both
        const float* kp = ((flags >> (SIDE == COL ? 0 : es)) & 1) ? kpu + (SIDE == COL ? c.cur.x : oth) * BS : nullptr;
        const int sb = (SIDE == COL ? (q & 1) : (q >> 1)) * 2 + g;      // quarter: 2 (query / 32) + key / 32
        const bool live = !SUB || ((flags >> (8 + 8 * es + sb)) & 1);
        // the group's value tiles must have been consumed (pair j - 2)
        if (j >= 2 && !wait_all(pdone + 8 * ((j - 2) % NP), (uint32_t)((j - 2) / NP), ERR_MMA2_WAIT)) { ok = false; break; }
        if (!wait_all(s_ready + 8 * (j % 3), (uint32_t)(j / 3), ERR_MMA_WAIT)) { ok = false; break; }
        tc_fence_after();
        const uint32_t ts = t_lane + (uint32_t)(j % 3) * 128u + g * 32;
        uint32_t sv[32], gv[32];
        tmem_ld32(ts, sv);
        tmem_ld32(ts + 64u, gv);
        tmem_ld_wait();
        if (mine) {
          if (kp) take_penalty(sv, kp, inv_scale);
          const uint32_t tds = sbase + C::O_PD + grp * C::PD + es * VT_BYTES + row * 128, tp = tds + 2 * VT_BYTES;
          const uint64_t sc22 = pack2(sc2, sc2), scale2 = pack2(a.scale, a.scale), nds2 = pack2(nds, nds), nh2 = pack2(-h, -h);
          auto piece = [&](int cc) {             // eight columns: one 16-byte piece of each tile
            uint32_t wp[4], wd[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int e = cc * 8 + 2 * x;
              float p0, p1, d0, d1;
              unpack2(fma2(pack2(sv[e], sv[e + 1]), sc22, nh2), p0, p1);
              p0 = ex2_approx(p0); p1 = ex2_approx(p1);
              wp[x] = pack_bf16(p0, p1);
              unpack2(mul2(pack2(p0, p1), fma2(pack2(gv[e], gv[e + 1]), scale2, nds2)), d0, d1);
              wd[x] = pack_bf16(d0, d1);
              if (SUB && !live) { wp[x] = 0u; wd[x] = 0u; }
            }
            const uint32_t off = (uint32_t)(((g * 4 + cc) ^ (row & 7)) << 4);
            st_shared_v4(tds + off, wd);
            if (SIDE == COL) st_shared_v4(tp + off, wp);
          };
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) piece(cc);
        }
        tc_fence_before();
        fence_proxy_async();                                          // tiles -> visible to the MMAs
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(t_free + 8 * (j % 3));
          mbar_arrive(p_ready + 8 * grp);
        }
        if (pend) ok = flush();                                       // an earlier unit: its last products have long been issued
        if (k + 1 == npairs) {                                        // this group worked on the unit's last pair: it writes the rows
          pend = true; pend_par = par; pend_dst = dst; pend_phase = par ? done1 : done0;
        }
      }
      if (par) ++done1; else ++done0;
    }
    if (ok && pend) flush();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512u);
}

// Lines (block rows or block columns) from the longest to the shortest, and their entries in pairs.  One CTA.
//   rec[x] = {line, index of its first pair, pairs, entries};  pair[p] = {other line of entry 0, of entry 1 (-1: none), CSR block ids}
__global__ void k_line_recs(const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx, const int32_t* __restrict__ pos, int nb,
                            int4* __restrict__ rec, int4* __restrict__ pair) {
  __shared__ int s_n[SPION_MAX_NB], s_order[SPION_MAX_NB], s_first[SPION_MAX_NB];
  for (int c = threadIdx.x; c < nb; c += blockDim.x) s_n[c] = ptr[c + 1] - ptr[c];
  __syncthreads();
  for (int c = threadIdx.x; c < nb; c += blockDim.x) {
    const int n = s_n[c];
    int rank = 0;
    for (int o = 0; o < nb; ++o) rank += (s_n[o] > n) || (s_n[o] == n && o < c);
    s_order[rank] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int x = 0; x < nb; ++x) { s_first[x] = acc; acc += (s_n[s_order[x]] + 1) >> 1; }
  }
  __syncthreads();
  for (int x = threadIdx.x >> 5; x < nb; x += blockDim.x >> 5) {
    const int c = s_order[x], beg = ptr[c], n = s_n[c], np = (n + 1) >> 1;
    if ((threadIdx.x & 31) == 0) rec[x] = make_int4(c, s_first[x], np, n);
    for (int k = threadIdx.x & 31; k < np; k += 32) {
      const int e0 = beg + 2 * k;
      const bool two = 2 * k + 1 < n;
      pair[s_first[x] + k] = make_int4(idx[e0], two ? idx[e0 + 1] : -1, pos ? pos[e0] : e0, two ? (pos ? pos[e0 + 1] : e0 + 1) : 0);
    }
  }
}

}  // namespace

namespace tc {

template <int D, int SIDE, bool SUB>
static int bw_launch(spion_ctx* c, TcState* s, const CUtensorMap& a0, const CUtensorMap& a1, const CUtensorMap& f0, const CUtensorMap& f1,
                     const BwArgs& a) {
  using C = Bw<D, SIDE>;
  static_assert(C::SMEM <= 227 * 1024, "shared memory");
  auto k = k_bwd_stream<D, SIDE, SUB>;
  const long long total = (long long)c->BH * a.nb;
  const int grid = (int)(total < (long long)s->sms ? total : (long long)s->sms);       // one CTA per SM (all 512 TMEM columns)
  k<<<grid, BW_THREADS, C::SMEM, c->stream>>>(a0, a1, f0, f1, a);
  SPION_LAUNCH_CHECK();
  c->launches += 1;
  return SPION_OK;
}

template <int D>
static int bw_attrs() {
  for (auto k : {k_bwd_stream<D, ROW, false>, k_bwd_stream<D, ROW, true>})
    SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Bw<D, ROW>::SMEM));
  for (auto k : {k_bwd_stream<D, COL, false>, k_bwd_stream<D, COL, true>})
    SPION_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Bw<D, COL>::SMEM));
  return SPION_OK;
}
int stream_backward_set_attrs(int d) { return d == 64 ? bw_attrs<64>() : bw_attrs<32>(); }

int stream_prepare(spion_ctx* c, TcState* s) {
  const TcView vw = tc_view(c, s);
  if (!s->line_rec && device_alloc((void**)&s->line_rec, 2 * (size_t)SPION_MAX_NB * sizeof(int4)) != SPION_OK) return SPION_ERR_ALLOC;
  if ((size_t)vw.nnzb > s->line_pair_cap) {                         // at most one pair per entry, columns and rows
    device_free(s->line_pair);
    s->line_pair = nullptr;
    s->line_pair_cap = 0;
    if (device_alloc((void**)&s->line_pair, 2 * (size_t)vw.nnzb * sizeof(int4)) != SPION_OK) return SPION_ERR_ALLOC;
    s->line_pair_cap = (size_t)vw.nnzb;
  }
  k_line_recs<<<1, 512, 0, c->stream>>>(vw.col_ptr, vw.row_idx, vw.csc_pos, vw.nb, s->line_rec, s->line_pair);
  SPION_LAUNCH_CHECK();
  k_line_recs<<<1, 512, 0, c->stream>>>(vw.row_ptr, vw.col_idx, nullptr, vw.nb, s->line_rec + SPION_MAX_NB, s->line_pair + s->line_pair_cap);
  SPION_LAUNCH_CHECK();
  c->launches += 2;
  return SPION_OK;
}

template <int D>
static int bwd_stream(spion_ctx* c, TcState* s, const void* Q, const void* K, const void* V, const void* O, const void* dO, const float* lse,
                      const float* keypad, void* dQ, void* dK, void* dV) {
  const TcView vw = tc_view(c, s);
  CUtensorMap mq, mk, mv, mdo;
  int rc;
  if ((rc = make_operand_map(c, s, &mq, Q, D)) || (rc = make_operand_map(c, s, &mk, K, D)) || (rc = make_operand_map(c, s, &mv, V, D)) ||
      (rc = make_operand_map(c, s, &mdo, dO, D)))
    return rc;
  BwArgs a;
  a.lse = lse; a.keypad = keypad;
  a.delta = a.delta_out = s->delta_ws;
  a.O = (const __nv_bfloat16*)O; a.dO = (const __nv_bfloat16*)dO;
  a.submask = vw.submask;
  a.L = c->L; a.BH = c->BH; a.nb = vw.nb; a.heads = c->heads; a.by_rank = order_by_rank(c);
  a.scale = c->scale; a.status = c->status_dev;
  prof_mark(c, -1);
  a.rec = s->line_rec + SPION_MAX_NB; a.pair = s->line_pair + s->line_pair_cap;
  a.out0 = (__nv_bfloat16*)dQ; a.out1 = nullptr;
  rc = a.submask ? bw_launch<D, ROW, true>(c, s, mk, mv, mq, mdo, a) : bw_launch<D, ROW, false>(c, s, mk, mv, mq, mdo, a);
  if (rc) return rc;
  prof_mark(c, SPION_STAGE_BWD_ROW_RC);
  a.rec = s->line_rec; a.pair = s->line_pair;
  a.out0 = (__nv_bfloat16*)dK; a.out1 = (__nv_bfloat16*)dV;
  rc = a.submask ? bw_launch<D, COL, true>(c, s, mq, mdo, mk, mv, a) : bw_launch<D, COL, false>(c, s, mq, mdo, mk, mv, a);
  if (rc) return rc;
  prof_mark(c, SPION_STAGE_BWD_COL_RC);
  return SPION_OK;
}

int recompute_backward(spion_ctx* c, TcState* s, const void* Q, const void* K, const void* V, const void* O, const void* dO, const float* lse,
                       const float* keypad, void* dQ, void* dK, void* dV) {
  return c->d == 64 ? bwd_stream<64>(c, s, Q, K, V, O, dO, lse, keypad, dQ, dK, dV)
                    : bwd_stream<32>(c, s, Q, K, V, O, dO, lse, keypad, dQ, dK, dV);
}

}  // namespace tc
