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
// One persistent CTA per SM, 640 threads.  Warps 0 to 2 are one thread each: as whole warps they took 300 cycles a pair for records, waits and
// votes around 450 to 650 cycles of issue, and S / dP (rows) and the second products (columns) were what a pair waited for.
//   warp 0   loads: the tiles of a pair into a ring of slots, the fixed tiles of a unit into one of two sets (TMA)
//   warp 1   S / dP products into one of three tensor-memory sets
//   warp 2   second products, when the tiles of a pair are written
//   warp 3   the walk: 16 byte records of the CTA's pairs, 16 at a time (which tiles, first or last of its unit, which blocks have padded
//            keys), in shared memory for all other warps.  With a walk of its own in every warp and the statistics handed out pair by
//            pair, that warp was what the others waited for: each value it copied from one variable to the next to have it early is a
//            wait for global memory.
//   warps 4-19   arithmetic, in groups that take pairs in turn, each warp one tensor-memory quadrant.  Four groups of four warps, a warp
//            the whole 64 columns of its rows in two halves: what a pair costs besides its values (waits, fences, hand-over) is paid by
//            half as many warps than with two groups of eight, and four chains fill each other's waits.  COL at head_dim 64: two groups of
//            eight (value tiles of four pairs do not fit shared memory).  ROW: dS over the V tiles, which only dP reads; delta
//            first, while the first tiles arrive, left in global memory, for COL too.
// What bounds it: per pair at head_dim 64 the tensor pipe needs 920 (COL) or 660 cycles (ROW), the exponentials 512; a pair takes
// about 1450.
// Measured, ROW and COL, before (two groups of eight, a walk in every warp) and now: 64 matrices, L = 16384, d 64, 5 %: 637 and 639 us, now
// 561 and 591; 256 matrices, L = 4096, d 32, 10 %, padded keys, two full columns: 425 and 394, now 341 and 306.  Kernels of their own for
// calls without key penalties, and blocks whose keys share one penalty taken with the row's constant: 529 and 571; 255 and 254.
// One thread for loads and MMAs: head_dim 32, L = 16384, 5 %: 417 and 428, now 369 and 399; the padded case 244 and 243.  COL at head_dim 32: five
// slots and four sets of value tiles 306 us, seven and three 317.  Which mask is served by rebuilt and which by stored tiles:
// _recompute_pays in native.py.
//
// Every wait is bounded; on a time-out the waiting warp records a code in the status word and the CTA winds down.
#include <type_traits>

#include "tc_stream.cuh"

using namespace tc;

namespace {

constexpr int BW_THREADS = 640;
constexpr int COL = 0, ROW = 1;

template <int D, int SIDE> struct Bw {
  using T = OpTile<D>;
  static constexpr int NGR = SIDE == COL && D == 64 ? 2 : 4;          // arithmetic groups
  static constexpr int NS = NGR == 2 ? 3 : 4;                         // barriers that hand S and dP over, pair j: j % NS
  static constexpr int WPG = 16 / NGR, HALVES = NGR / 2;              // warps of a group; halves of a tile's columns a warp does
  static constexpr int NP = SIDE == COL ? (D == 64 ? 4 : 5) : (D == 64 ? 6 : 8);      // pair slots
  static constexpr uint32_t PD = (SIDE == COL ? 4 : 2) * VT_BYTES;    // value tiles of a pair: dS of both entries, then P of both
  // A0 of both entries, A1 of both entries; ROW: the dS tiles take the place of A1, which only the first products read
  static constexpr uint32_t SLOT = 2 * T::BYTES + (SIDE == COL ? 2 * T::BYTES : PD);
  static constexpr int NPD = SIDE == ROW ? 0 : NGR;                   // sets of value tiles beside the slots
  static constexpr uint32_t FIX = 2 * T::BYTES;                       // F0, F1; two sets
  static constexpr int NACC = SIDE == COL && D == 64 ? 2 : 4;         // accumulator sets
  static constexpr uint32_t O_FIX = NP * SLOT, O_PD = O_FIX + 2 * FIX, O_BAR = O_PD + NPD * PD;
  static constexpr uint32_t O_RING = O_BAR + 432;                     // records of 32 pairs
  static constexpr size_t SMEM = O_RING + 32 * 16;
};

struct BwArgs {
  const float *lse, *delta, *keypad;         // [BH*L]; delta: COL only; keypad may be null; RND: lse holds the rows' exponents
  const float* factor;                       // RND: [BH*L]
  float* delta_out;                          // ROW
  const __nv_bfloat16 *O, *dO;               // ROW: for delta
  __nv_bfloat16 *out0, *out1;                // dK (COL) or dQ (ROW); dV (COL)
  const int4 *rec, *pair;                    // lines and pairs (k_line_recs)
  const uint8_t* submask;
  int L, BH, nb, heads, by_rank;
  float scale;
  int* status;
};

// Record of a pair: {flags, line of entry 0 | line of entry 1 << 16, line of the unit, (b,h) matrix}.  Flags: 1, 2: the keys of entry 0, 1 have
// different penalties; 1 << 24, 1 << 25: one that is not zero; the accumulator set << 4; the selected quarters of entry 0 << 8, of entry 1 << 16.
constexpr int PF_LAST = 4, PF_TWO = 8, PF_FIRST = 64, PF_END = (int)0x80000000;

// The penalties of 64 keys (see Pen4), per lane: PAD_NONE, PAD_ONE (the same for all) or PAD_MIXED.
constexpr int PAD_NONE = 0, PAD_MIXED = 1, PAD_ONE = 1 << 24;
__device__ __forceinline__ int pad64(const float* kp) {
  const float first = kp[0];
  bool other = !(first == first);
  if ((reinterpret_cast<uintptr_t>(kp) & 15) == 0) {
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      const float4 f = reinterpret_cast<const float4*>(kp)[x];
      other |= f.x != first || f.y != first || f.z != first || f.w != first;
    }
  } else {
    for (int x = 0; x < 64; ++x) other |= kp[x] != first;
  }
  return other ? PAD_MIXED : first != 0.f ? PAD_ONE : PAD_NONE;
}

// Scores of 32 keys -> exponents: (s scale log2e) - (pad log2e + h), rounded as the forward does.
__device__ __forceinline__ void take_exponent(uint32_t (&s)[32], const float* kp, float sc2, float h) {
#pragma unroll
  for (int x = 0; x < 32; ++x) s[x] = __float_as_uint(fmaf(__uint_as_float(s[x]), sc2, -fmaf(kp[x], LOG2E, h)));
}

// KP: with key penalties.  RND: dS from the P that the forward wrote or would have written, rounded as there (stat of k_fwd_fused), and not
// from P before it is rounded: the gradients are bit for bit those of kernels that read stored tiles.
template <int D, int SIDE, bool SUB, bool KP, bool RND>
__global__ void __launch_bounds__(BW_THREADS, 1) k_bwd_stream(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                                                              const __grid_constant__ CUtensorMap tmF0, const __grid_constant__ CUtensorMap tmF1,
                                                              const __grid_constant__ BwArgs a) {
  using C = Bw<D, SIDE>;
  using T = OpTile<D>;
  constexpr int NP = C::NP, NGR = C::NGR, WPG = C::WPG, NACC = C::NACC;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);                          // must be 1024-aligned (checked below)
  const uint32_t bars = sbase + C::O_BAR;
  // pfull / pdone[slot]: tiles landed / second products that read the slot retired; p_ready[slot]: value tiles of its pair written (the
  // group's warps); s_ready[pair % NS]: S and dP of a pair in tensor memory; t_free[set]: ... read out (the group's warps);
  // acc_done[group][parity of the units it writes]: accumulators complete; acc_free[set]: ... read out (the group's warps); f_full /
  // f_free[2]: fixed tiles landed / no longer read; r_full / r_free[half]: 16 records written / read (all warps but warp 3).
  // A parity tells two phases apart: at a wait for a phase the one before it must be over, and the one after it must not be.  Most
  // barriers have one waiter (a warp, a group's warps; r_full: each reader for itself) that waits for each of their phases, and the next
  // phase needs something that comes after the wait.  The others:
  //   s_ready, fewer or more barriers than groups (COL at head_dim 64: three, two groups): the group of pair j did not wait for pair j - NS.
  //     It has waited for pdone of pair j - NPD, whose products warp 2 issued after those of pair j - NS, for which that pair's group had
  //     to see its S.  S of pair j + NS is issued after that of pair j + 3, which waits for this group's t_free of pair j.
  //   pdone, waited for by warp 0 and by the groups of COL, with more slots than value tiles (head_dim 32: five, four groups, a group sees
  //     every fourth phase of a slot): pair i = j - NPD is the group's own, and its tiles were requested when warp 0 had seen pdone of
  //     pair i - NP.  The products of pair i + NP come after those of pair j, which wait for this group's p_ready.
  // A group writes the rows of a finished unit after its next pair, so there must be a set of accumulators for each group's last unit.
  static_assert(C::NS >= 3 && (C::NS == NGR || (SIDE == COL && C::NPD <= C::NS)), "s_ready");
  static_assert(SIDE == ROW || (C::NPD % NGR == 0 && C::NPD <= NP), "pdone");
  static_assert(NACC >= NGR, "accumulators");
  const uint32_t pfull = bars, pdone = bars + 64, p_ready = bars + 128, s_ready = bars + 192, t_free = bars + 224, acc_done = bars + 248,
                 acc_free = bars + 312, f_full = bars + 344, f_free = bars + 360, r_full = bars + 376, r_free = bars + 392,
                 slot = bars + 408, abort_w = bars + 412;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  volatile int* abort_ptr = reinterpret_cast<volatile int*>(smem_raw + (abort_w - sbase));

  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int G = (int)gridDim.x, total = a.nb * a.BH;
  const int n_my = total > (int)blockIdx.x ? (total - (int)blockIdx.x + G - 1) / G : 0;         // units blockIdx.x, + G, ...
  const UnitMap um{a.nb, a.BH, a.by_rank};
  constexpr uint32_t ACC = 384u;                                      // three S / dP sets of 128 columns, then the accumulators

  if (SIDE == ROW) next_may_start();                                  // the columns
  else wait_for_kernel_before();
  if (warp == 0 && lane == 0) {
    int ab = *reinterpret_cast<volatile int*>(a.status);
    if ((sbase & 1023u) != 0u) { report(a.status, ERR_LOAD_WAIT); ab = 1; }
    *abort_ptr = ab;
    for (int i = 0; i < NP; ++i) { mbar_init(pfull + 8 * i, 1); mbar_init(pdone + 8 * i, 1); mbar_init(p_ready + 8 * i, WPG); }
    for (int i = 0; i < C::NS; ++i) mbar_init(s_ready + 8 * i, 1);
    for (int i = 0; i < 3; ++i) mbar_init(t_free + 8 * i, WPG);
    for (int i = 0; i < 2 * NGR; ++i) mbar_init(acc_done + 8 * i, 1);
    for (int i = 0; i < NACC; ++i) mbar_init(acc_free + 8 * i, WPG);
    for (int i = 0; i < 2; ++i) {
      mbar_init(f_full + 8 * i, 1);
      mbar_init(f_free + 8 * i, 1);
      mbar_init(r_full + 8 * i, 1);
      mbar_init(r_free + 8 * i, 19);
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
  // columns and lanes of accumulator set x: COL beside each other (dK in lanes 0-15 of every quadrant, dV in 16-31); ROW (dQ alone): two
  // beside each other, the other two at lane offset 16
  auto acc_at = [](int x) -> uint32_t {
    return ACC + (SIDE == ROW ? (uint32_t)(x & 1) * D + ((uint32_t)((x >> 1) * 16) << 16) : (uint32_t)x * D);
  };
  const int4* ring = reinterpret_cast<const int4*>(smem_raw + C::O_RING);
  // A reader takes the records of pairs j, j + step, ...: it waits where it enters a half and hands it back with its last record there.
  auto record = [&](uint32_t j, uint32_t step, int4& r) -> bool {
    if ((j & 15) < step && !wait_all(r_full + 8 * ((j >> 4) & 1), j >> 5, ERR_LOAD_WAIT)) return false;
    r = ring[j & 31];
    __syncwarp();
    if ((j & 15) + step >= 16 && lane == 0) mbar_arrive(r_free + 8 * ((j >> 4) & 1));
    return true;
  };

  // One thread of a warp does all that the loads and the products need: nothing there is worth the other lanes.
  auto wait_one = [&](uint32_t bar, uint32_t parity, int code) -> bool {
    if (mbar_wait(bar, parity & 1u)) return true;
    report(a.status, code);
    return false;
  };
  auto record_one = [&](uint32_t j, int4& r) -> bool {
    if ((j & 15) == 0 && !wait_one(r_full + 8 * ((j >> 4) & 1), j >> 5, ERR_LOAD_WAIT)) return false;
    r = ring[j & 31];
    if ((j & 15) == 15) mbar_arrive(r_free + 8 * ((j >> 4) & 1));
    return true;
  };
  if (warp == 0) {
    // ================================================================== loads
    if (elect_one()) {
      int u = 0, ps = 0, round = 0;
      int4 r;
      for (uint32_t j = 0; record_one(j, r) && r.x >= 0; ++j) {
        const bool first = r.x & PF_FIRST, two = r.x & PF_TWO;
        const int fs = u & 1;
        const OpPos pos = op_pos(r.w, a.L, a.heads, D);
        const uint32_t dst = sbase + ps * C::SLOT;
        if (first) {
          if (u >= 2 && !wait_one(f_free + 8 * fs, (uint32_t)((u >> 1) - 1), ERR_MMA2_WAIT)) break;
          const uint32_t f = sbase + C::O_FIX + fs * C::FIX;
          mbar_expect_tx(f_full + 8 * fs, 2 * T::BYTES);
          tma_load_2d(f, &tmF0, f_full + 8 * fs, pos.x0, pos.row0 + r.z * BS);
          tma_load_2d(f + T::BYTES, &tmF1, f_full + 8 * fs, pos.x0, pos.row0 + r.z * BS);
        }
        if (round >= 1 && !wait_one(pdone + 8 * ps, (uint32_t)(round - 1), ERR_MMA2_WAIT)) break;
        mbar_expect_tx(pfull + 8 * ps, (two ? 4 : 2) * T::BYTES);
        const int y0 = pos.row0 + (r.y & 0xffff) * BS, y1 = pos.row0 + (r.y >> 16) * BS;
        tma_load_2d(dst, &tmA0, pfull + 8 * ps, pos.x0, y0);
        tma_load_2d(dst + 2 * T::BYTES, &tmA1, pfull + 8 * ps, pos.x0, y0);
        if (two) {
          tma_load_2d(dst + T::BYTES, &tmA0, pfull + 8 * ps, pos.x0, y1);
          tma_load_2d(dst + 3 * T::BYTES, &tmA1, pfull + 8 * ps, pos.x0, y1);
        }
        if (r.x & PF_LAST) ++u;
        if (++ps == NP) { ps = 0; ++round; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================================================== S and dP
    if (elect_one()) {
      constexpr uint32_t IDESC = make_idesc_bf16(SIDE == COL ? 128 : 64, 64, 0, 0);
      const uint64_t KM = T::kmajor(sbase, 0);
      int u = 0, ps = 0, round = 0, set = 0, sround = 0, sr = 0;
      int4 r;
      for (uint32_t j = 0; record_one(j, r) && r.x >= 0; ++j) {
        const int par = u & 1;
        if ((r.x & PF_FIRST) && !wait_one(f_full + 8 * par, (uint32_t)(u >> 1), ERR_LOAD_WAIT)) break;
        if (!wait_one(pfull + 8 * ps, (uint32_t)round, ERR_LOAD_WAIT)) break;
        if (sround >= 1 && !wait_one(t_free + 8 * set, (uint32_t)(sround - 1), ERR_MMA_WAIT)) break;
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
          if (r.x & PF_TWO) products(1);
        }
        mma_commit(s_ready + 8 * sr);
        if (r.x & PF_LAST) {                                          // the fixed tiles are read by these products only
          mma_commit(f_free + 8 * par);
          ++u;
        }
        if (++ps == NP) { ps = 0; ++round; }
        if (++set == 3) { set = 0; ++sround; }
        if (++sr == C::NS) sr = 0;
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ================================================================== second products
    if (elect_one()) {
      constexpr uint32_t IDESC = make_idesc_bf16(64, D, SIDE == COL ? 1 : 0, 1);
      constexpr uint32_t V_STEP = SIDE == COL ? ValTile::MN_STEP : ValTile::K_STEP;
      const uint64_t MN = T::mnmajor(sbase, 0), VT = SIDE == COL ? ValTile::mnmajor(sbase, 0) : ValTile::kmajor(sbase, 0);
      int u = 0, ps = 0, round = 0, grp = 0, pd = 0;
      uint32_t odd = 0;                                               // bit g: group g has written an odd number of units
      int4 r;
      for (uint32_t j = 0; record_one(j, r) && r.x >= 0; ++j) {
        const int x = u % NACC;
        if ((r.x & PF_FIRST) && u >= NACC && !wait_one(acc_free + 8 * x, (uint32_t)(u / NACC - 1), ERR_MMA2_WAIT)) break;
        if (!wait_one(p_ready + 8 * ps, (uint32_t)round, ERR_MMA_WAIT)) break;
        tc_fence_after();
        const uint32_t acc = tmem + acc_at(x), more = (r.x & PF_FIRST) ? 0u : 1u;
        const uint64_t b0 = desc_advance(MN, ps * C::SLOT);
        const uint64_t vt = desc_advance(VT, SIDE == COL ? C::O_PD + pd * C::PD : ps * C::SLOT + 2 * T::BYTES);
        auto products = [&](int e, uint32_t first) {
#pragma unroll
          for (int kk = 0; kk < BS / 16; ++kk)                        // dK or dQ
            mma_bf16(acc, desc_advance(vt, e * VT_BYTES + kk * V_STEP), desc_advance(b0, e * T::BYTES + kk * T::MN_STEP), IDESC, kk > 0 ? 1u : first);
          if (SIDE == COL) {
#pragma unroll
            for (int kk = 0; kk < BS / 16; ++kk)                      // dV (lanes 16-31)
              mma_bf16(acc + (16u << 16), desc_advance(vt, (2 + e) * VT_BYTES + kk * V_STEP),
                       desc_advance(b0, (2 + e) * T::BYTES + kk * T::MN_STEP), IDESC, kk > 0 ? 1u : first);
          }
        };
        products(0, more);
        if (r.x & PF_TWO) products(1, 1u);
        mma_commit(pdone + 8 * ps);
        if (r.x & PF_LAST) {
          mma_commit(acc_done + 8 * (2 * grp + ((odd >> grp) & 1)));
          ++u;
          odd ^= 1u << grp;
        }
        if (++ps == NP) { ps = 0; ++round; }
        if (++grp == NGR) grp = 0;
        if (SIDE == COL && ++pd == C::NPD) pd = 0;
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ================================================================== the walk: records of the CTA's pairs, 16 at a time
    // 32 units at a time, one per lane; lanes t and t + 16 look at entries 0 and 1 of pair t of a half.
    auto unit_at = [&](int i, int& bh) -> int4 {
      bh = 0;
      if (i >= n_my) return make_int4(0, 0, 0, 0);
      int rank;
      um.at((int)blockIdx.x + i * G, bh, rank);
      return a.rec[rank];
    };
    int bh, bh_n, i0 = 0, pos = 0, tot = 0, units = 0;                // units with entries before the 32
    int4 un = unit_at(lane, bh), un_n = unit_at(32 + lane, bh_n);
    int end = 0;                                                      // pairs of the 32 units up to this lane's
    uint32_t used = 0;                                                // those with entries
    auto enter = [&]() {
      end = un.z;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, s);
        if (lane >= s) end += v;
      }
      pos = 0;
      tot = __shfl_sync(0xffffffffu, end, 31);
      used = __ballot_sync(0xffffffffu, un.z > 0);
      uint32_t none = __ballot_sync(0xffffffffu, un.z == 0 && i0 + lane < n_my);
      while (none) {                                                  // lines without entries: zero rows
        const int x = __ffs(none) - 1;
        none &= none - 1;
        const int line = __shfl_sync(0xffffffffu, un.x, x);
        const OpPos pos0 = op_pos(__shfl_sync(0xffffffffu, bh, x), a.L, a.heads, D);
        for (int y = lane; y < BS * (D / 8); y += 32) {
          const size_t off = (size_t)(pos0.row0 + line * BS + y / (D / 8)) * pos0.ld + pos0.x0 + (y % (D / 8)) * 8;
          *reinterpret_cast<uint4*>(a.out0 + off) = make_uint4(0, 0, 0, 0);
          if (SIDE == COL) *reinterpret_cast<uint4*>(a.out1 + off) = make_uint4(0, 0, 0, 0);
        }
      }
    };
    enter();
    const int e = lane >> 4;
    bool more = true;
    for (uint32_t f = 0; more; ++f) {
      if (f >= 2 && !wait_all(r_free + 8 * (f & 1), (f >> 1) - 1, ERR_MMA_WAIT)) break;
      int4* half = reinterpret_cast<int4*>(smem_raw + C::O_RING) + 16 * (f & 1);
      int filled = 0;
      while (filled < 16) {
        if (pos >= tot) {
          if (i0 + 32 >= n_my) {
            if (lane >= filled && lane < 16) half[lane] = make_int4(PF_END, 0, 0, 0);       // every reader meets one
            more = filled > 16 - NGR;                                 // ... in this half or the next one
            filled = 16;
            break;
          }
          i0 += 32;
          units += __popc(used);
          un = un_n; bh = bh_n;
          un_n = unit_at(i0 + 32 + lane, bh_n);
          enter();
          continue;
        }
        const int n = min(16 - filled, tot - pos), t = (lane & 15) - filled;
        const bool active = t >= 0 && t < n;
        const int p = pos + (active ? t : 0);
        int x = 0;                                                    // the unit of pair p: the first whose pairs end after it
#pragma unroll
        for (int s = 16; s; s >>= 1)
          if (__shfl_sync(0xffffffffu, end, x + s - 1) <= p) x += s;
        const int line = __shfl_sync(0xffffffffu, un.x, x), first = __shfl_sync(0xffffffffu, un.y, x), np = __shfl_sync(0xffffffffu, un.z, x),
                  n_e = __shfl_sync(0xffffffffu, un.w, x), b = __shfl_sync(0xffffffffu, bh, x), k = p - (__shfl_sync(0xffffffffu, end, x) - np);
        const int4 pr = a.pair[first + k];
        const bool two = 2 * k + 1 < n_e, here = e == 0 || two;
        const int o = e ? pr.y : pr.x;
        int pad = PAD_NONE, sub = 0xff;
        if (KP && here) pad = pad64(a.keypad + (size_t)b * a.L + (SIDE == COL ? line : o) * BS);
        if (SUB) sub = here ? a.submask[e ? pr.w : pr.z] : 0;
        const int fl = pad | (sub << 8), fl1 = __shfl_down_sync(0xffffffffu, fl, 16);
        const int ux = units + __popc(used & ((1u << x) - 1));
        if (active && e == 0)
          half[lane] = make_int4(fl | (fl1 & (PAD_MIXED | PAD_ONE)) << 1 | (fl1 & 0xff00) << 8 | (k + 1 == np ? PF_LAST : 0) | (two ? PF_TWO : 0) |
                                     (k == 0 ? PF_FIRST : 0) | (ux % NACC) << 4,
                                 pr.x | (two ? pr.y << 16 : 0), line, b);
        filled += n;
        pos += n;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(r_full + 8 * (f & 1));
    }
  } else {
    // ================================================================== arithmetic
    const int mw = warp - 4, q = warp & 3, grp = mw / WPG, g0 = WPG == 8 ? (mw >> 2) & 1 : 0;
    if (SIDE == ROW) {
      // delta = rowsum(dO.O) of all rows of this CTA: D / 8 lanes per row, 16 bytes each, a warp RPW rows of a unit, eight such loads in
      // flight.  Lane l knows where unit l of the next 32 is.
      constexpr int LPR = D / 8, RPW = 32 / LPR, WPU = BS / RPW, UPS = 16 / WPU, UN = 8;       // warps per unit, units per step
      const int r0 = (mw % WPU) * RPW + lane / LPR;
      int l_row = 0, l_x = 0, l_out = 0;
      for (int i0 = 0; i0 < n_my; i0 += UN * UPS) {
        if (i0 % 32 == 0 && i0 + lane < n_my) {
          int bh, rank;
          um.at((int)blockIdx.x + (i0 + lane) * G, bh, rank);
          const int line = a.rec[rank].x;
          const OpPos pos = op_pos(bh, a.L, a.heads, D);
          l_row = pos.row0 + line * BS; l_x = pos.x0; l_out = bh * a.L + line * BS;
        }
        uint4 u[UN], v[UN];
#pragma unroll
        for (int x = 0; x < UN; ++x) {
          const int i = i0 + x * UPS + mw / WPU;
          const int rw = __shfl_sync(0xffffffffu, l_row, i & 31), x0 = __shfl_sync(0xffffffffu, l_x, i & 31);
          u[x] = v[x] = make_uint4(0, 0, 0, 0);
          if (i < n_my) {
            const size_t off = (size_t)(rw + r0) * (a.heads ? a.heads * D : D) + x0 + (lane % LPR) * 8;
            u[x] = *reinterpret_cast<const uint4*>(a.dO + off);
            v[x] = *reinterpret_cast<const uint4*>(a.O + off);
          }
        }
#pragma unroll
        for (int x = 0; x < UN; ++x) {
          const int i = i0 + x * UPS + mw / WPU;
          const int out = __shfl_sync(0xffffffffu, l_out, i & 31);
          const float t = bf16_lo(u[x].x) * bf16_lo(v[x].x) + bf16_hi(u[x].x) * bf16_hi(v[x].x) + bf16_lo(u[x].y) * bf16_lo(v[x].y) +
                          bf16_hi(u[x].y) * bf16_hi(v[x].y) + bf16_lo(u[x].z) * bf16_lo(v[x].z) + bf16_hi(u[x].z) * bf16_hi(v[x].z) +
                          bf16_lo(u[x].w) * bf16_lo(v[x].w) + bf16_hi(u[x].w) * bf16_hi(v[x].w);
          // half of the head dimension in order, then the two halves: as the row kernel of the stored path adds them
          float half = __shfl_sync(0xffffffffu, t, lane & ~(LPR / 2 - 1));
#pragma unroll
          for (int y = 1; y < LPR / 2; ++y) half += __shfl_sync(0xffffffffu, t, (lane & ~(LPR / 2 - 1)) + y);
          const float d = half + __shfl_xor_sync(0xffffffffu, half, LPR / 2);
          if (lane % LPR == 0 && i < n_my) a.delta_out[(size_t)out + r0] = d;
        }
      }
      __threadfence_block();
      asm volatile("bar.sync 1, 512;" ::: "memory");                  // delta of this CTA's rows is in global memory
    }
    // entry of the pair and query row of this lane: COL rows 0-63 first entry, 64-127 second; ROW second entry in lanes 16-31
    const int es = SIDE == COL ? q >> 1 : lane >> 4;
    const int row = SIDE == COL ? (q & 1) * 32 + lane : q * 16 + (lane & 15);
    const int orow = q * 16 + (lane & 15);                            // output row (64-row accumulators)
    const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16);
    const float sc2 = a.scale * LOG2E, inv_scale = 1.0f / a.scale;
    bool ok = true;
    bool pend = false;                                                // a finished unit whose rows this group has to write
    int pend_acc = 0, units = 0;                                      // its accumulator set; units written by this group before it
    size_t pend_off = 0;

    auto flush = [&]() -> bool {
      if (!wait_all(acc_done + 8 * (2 * grp + (units & 1)), (uint32_t)(units >> 1), ERR_MMA2_WAIT)) return false;
      ++units;
      tc_fence_after();
      __nv_bfloat16* dst = (SIDE == COL && lane >= 16 ? a.out1 : a.out0) + pend_off;
      const uint32_t taddr = t_lane + ACC + (SIDE == ROW ? (uint32_t)(pend_acc & 1) * D : (uint32_t)pend_acc * D);
      const bool mine = SIDE == COL || (lane >> 4) == (pend_acc >> 1);
#pragma unroll
      for (int h = 0; h < D; h += 32) {
        if (WPG == 8 && h / 32 != g0) continue;
        uint32_t v[32];
        tmem_ld32(taddr + h, v);
        tmem_ld_wait();
        if (mine) {
#pragma unroll
          for (int x = 0; x < 32; x += 8)
            *reinterpret_cast<uint4*>(dst + h + x) = make_uint4(pack_bf16(__uint_as_float(v[x]), __uint_as_float(v[x + 1])),
                                                                pack_bf16(__uint_as_float(v[x + 2]), __uint_as_float(v[x + 3])),
                                                                pack_bf16(__uint_as_float(v[x + 4]), __uint_as_float(v[x + 5])),
                                                                pack_bf16(__uint_as_float(v[x + 6]), __uint_as_float(v[x + 7])));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free + 8 * pend_acc);
      pend = false;
      return true;
    };

    // record and statistics of this row are requested a pair early
    int4 rec = make_int4(PF_END, 0, 0, 0);
    float h_next = 0.f, d_next = 0.f, f_next = 0.f;
    auto request = [&](uint32_t j) -> bool {
      if (!record(j, NGR, rec)) return false;
      if (rec.x >= 0 && (es == 0 || (rec.x & PF_TWO))) {
        const size_t ri = (size_t)rec.w * a.L + (SIDE == COL ? (es ? rec.y >> 16 : rec.y & 0xffff) : rec.z) * BS + row;
        h_next = a.lse[ri];
        if (RND) f_next = a.factor[ri];
        d_next = SIDE == COL ? a.delta[ri] : __ldcg(a.delta_out + ri);            // ROW: written by this CTA
        // one penalty for all keys goes with the log-sum-exp (here, where it waits for the load: a value of its own costs every pair 2 %)
        if (KP && ((rec.x >> es) & PAD_ONE))
          h_next = fmaf(a.keypad[(size_t)rec.w * a.L + (SIDE == COL ? rec.z : es ? rec.y >> 16 : rec.y & 0xffff) * BS], LOG2E, h_next);
      }
      return true;
    };
    ok = request(grp);
    for (uint32_t j = grp; ok && rec.x >= 0; j += NGR) {
      const int flags = rec.x, line = rec.z, key = SIDE == COL ? rec.z : es ? rec.y >> 16 : rec.y & 0xffff, bh = rec.w;
      const float h = h_next, nds = -d_next * a.scale;
      uint32_t f_hi = 0u, f_lo = 0u;
      if (RND) row_factor(f_next, f_hi, f_lo);
      if (!request(j + NGR)) { ok = false; break; }
      const uint32_t ps = j % NP, set = j % 3;
      const bool mine = es == 0 || (flags & PF_TWO);
      // COL: the value tiles of pair j - NPD must have been consumed
      if (SIDE == COL && j >= C::NPD && !wait_all(pdone + 8 * ((j - C::NPD) % NP), (j - C::NPD) / NP, ERR_MMA2_WAIT)) { ok = false; break; }
      if (!wait_all(s_ready + 8 * (j % C::NS), j / C::NS, ERR_MMA_WAIT)) { ok = false; break; }
      tc_fence_after();
      const uint32_t ts = t_lane + set * 128u;
      const uint32_t tds = sbase + (SIDE == COL ? C::O_PD + (j % (SIDE == COL ? C::NPD : 1)) * C::PD : ps * C::SLOT + 2 * T::BYTES) + es * VT_BYTES + row * 128;
      const uint64_t sc22 = pack2(sc2, sc2), scale2 = pack2(a.scale, a.scale), nds2 = pack2(nds, nds), nh2 = pack2(-h, -h);
      auto tiles = [&](auto mixed) {
        constexpr bool MIXED = decltype(mixed)::value;
#pragma unroll
        for (int hf = 0; hf < C::HALVES; ++hf) {
          const int g = C::HALVES == 2 ? hf : g0;                       // 32 columns (keys)
          uint32_t sv[32], gv[32];
          tmem_ld32(ts + g * 32, sv);
          tmem_ld32(ts + 64u + g * 32, gv);
          tmem_ld_wait();
          if (hf + 1 == C::HALVES) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(t_free + 8 * set);
          }
          if (mine) {
            // columns are keys in both
            const float* kp = MIXED && ((flags >> es) & 1) ? a.keypad + (size_t)bh * a.L + key * BS + g * 32 : nullptr;
            if (MIXED && !RND && kp) take_penalty(sv, kp, inv_scale);
            if (MIXED && RND && kp) take_exponent(sv, kp, sc2, h);
            const int sb = (SIDE == COL ? (q & 1) : (q >> 1)) * 2 + g;  // quarter: 2 (query / 32) + key / 32
            const bool live = !SUB || ((flags >> (8 + 8 * es + sb)) & 1);
            const uint64_t m22 = kp ? pack2(1.f, 1.f) : sc22, mh2 = kp ? 0ull : nh2;      // RND: sv holds exponents already
            auto piece = [&](int cc) {             // eight columns: one 16-byte piece of each tile
              uint32_t wp[4], wd[4];
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                const int c = cc * 8 + 2 * x;
                float p0, p1, d0, d1;
                unpack2(fma2(pack2(sv[c], sv[c + 1]), MIXED && RND ? m22 : sc22, MIXED && RND ? mh2 : nh2), p0, p1);
                p0 = ex2_approx(p0); p1 = ex2_approx(p1);
                wp[x] = pack_bf16(p0, p1);
                if (RND) {
                  wp[x] = times_factor(wp[x], f_hi, f_lo);
                  p0 = bf16_lo(wp[x]);
                  p1 = bf16_hi(wp[x]);
                }
                unpack2(mul2(pack2(p0, p1), fma2(pack2(gv[c], gv[c + 1]), scale2, nds2)), d0, d1);
                wd[x] = pack_bf16(d0, d1);
                if (SUB && !live) { wp[x] = 0u; wd[x] = 0u; }
              }
              const uint32_t off = (uint32_t)(((g * 4 + cc) ^ (row & 7)) << 4);
              st_shared_v4(tds + off, wd);
              if (SIDE == COL) st_shared_v4(tds + 2 * VT_BYTES + off, wp);
            };
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) piece(cc);
          }
        }
      };
      // a form of its own for pairs with a block whose keys have different penalties: as a branch in the other it costs every pair 8 %
      if (KP && __any_sync(0xffffffffu, (flags & 3) != 0)) tiles(std::true_type{});
      else tiles(std::false_type{});
      fence_proxy_async();                                            // tiles -> visible to the MMAs
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready + 8 * ps);
      if (pend) ok = flush();                                         // an earlier unit: its last products have long been issued
      if (flags & PF_LAST) {                                          // this group worked on the unit's last pair: it writes the rows
        pend = true;
        pend_acc = (flags >> 4) & 3;
        const OpPos pos = op_pos(bh, a.L, a.heads, D);
        pend_off = (size_t)(pos.row0 + line * BS + orow) * pos.ld + pos.x0;
      }
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

// 32-wide masks: super rows (two block rows) from the longest to the shortest, with the 32-wide blocks that one of their rows selects in ascending order, two
// to a tile, two tiles to a pair.  rec[x] = {super row, index of its first pair, pairs, tiles};  pair[p] = {block | block << 16 of tile 0, of tile 1,
// selected quarters of tile 0 (2 * row + block), of tile 1}.  A tile without a second block has its first one again, nothing of it selected.  One CTA.
__global__ void __launch_bounds__(512) k_gather_recs(const uint8_t* __restrict__ mat, int nb, int4* __restrict__ rec, int4* __restrict__ pair) {
  __shared__ int s_n[SPION_MAX_NB / 2], s_order[SPION_MAX_NB / 2], s_first[SPION_MAX_NB / 2];
  const int lines = nb >> 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int x = warp; x < lines; x += warps) {
    const uint8_t* m = mat + (size_t)2 * x * nb;
    int n = 0;
    for (int c0 = 0; c0 < nb; c0 += 32) {
      const int c = c0 + lane;
      n += __popc(__ballot_sync(0xffffffffu, c < nb && (m[c] | m[nb + c]) != 0));
    }
    if (lane == 0) s_n[x] = (n + 1) >> 1;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < lines; x += blockDim.x) {
    const int n = s_n[x];
    int rank = 0;
    for (int o = 0; o < lines; ++o) rank += (s_n[o] > n) || (s_n[o] == n && o < x);
    s_order[rank] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int x = 0; x < lines; ++x) { s_first[x] = acc; acc += (s_n[s_order[x]] + 1) >> 1; }
  }
  __syncthreads();
  for (int x = warp; x < lines; x += warps) {
    const int line = s_order[x], tiles = s_n[line], np = (tiles + 1) >> 1;
    int4* out = pair + s_first[x];
    if (lane == 0) rec[x] = make_int4(line, s_first[x], np, tiles);
    const uint8_t* m = mat + (size_t)2 * line * nb;
    int n = 0;
    for (int c0 = 0; c0 < nb; c0 += 32) {
      const int c = c0 + lane;
      const int r0 = c < nb && m[c] != 0, r1 = c < nb && m[nb + c] != 0;
      const uint32_t b = __ballot_sync(0xffffffffu, r0 | r1);
      // the blocks of this step, an even one with the one after it: of this step, of the next (lane 31's turn then), or none
      if (r0 | r1) {
        const int e = n + __popc(b & ((1u << lane) - 1u)), p = e >> 2, t = (e >> 1) & 1, half = e & 1;
        uint16_t* ids = reinterpret_cast<uint16_t*>(out + p) + 2 * t + half;
        uint8_t* sub = reinterpret_cast<uint8_t*>(out + p) + 8 + 4 * t;
        *ids = (uint16_t)c;
        sub[1 + half] = (uint8_t)((r0 << half) | (r1 << (2 + half)));
      }
      n += __popc(b);
    }
    __syncwarp();
    for (int t = lane; t < 2 * np; t += 32) {             // quarters of both blocks together; what a tile does not have
      uint16_t* ids = reinterpret_cast<uint16_t*>(out + (t >> 1)) + 2 * (t & 1);
      uint8_t* sub = reinterpret_cast<uint8_t*>(out + (t >> 1)) + 8 + 4 * (t & 1);
      if (2 * t + 1 >= n) ids[1] = 2 * t < n ? ids[0] : 0;
      if (2 * t >= n) ids[0] = 0;
      const int q = (2 * t < n ? sub[1] : 0) | (2 * t + 1 < n ? sub[2] : 0);
      *reinterpret_cast<int*>(sub) = q;
    }
  }
}

}  // namespace

namespace tc {

template <int D, int SIDE, bool SUB, bool KP, bool RND>
static int bw_launch_one(spion_ctx* c, TcState* s, const CUtensorMap& a0, const CUtensorMap& a1, const CUtensorMap& f0, const CUtensorMap& f1,
                     const BwArgs& a) {
  using C = Bw<D, SIDE>;
  static_assert(C::SMEM <= 227 * 1024, "shared memory");
  constexpr auto k = k_bwd_stream<D, SIDE, SUB, KP, RND>;
  int rc = allow_smem<k>(c->device, C::SMEM);
  if (rc) return rc;
  const long long total = (long long)c->BH * a.nb;
  const int grid = (int)(total < (long long)s->sms ? total : (long long)s->sms);       // one CTA per SM (all 512 TMEM columns)
  if (SIDE == COL) SPION_CUDA_TRY(launch_after(k, dim3(grid), dim3(BW_THREADS), C::SMEM, c->stream, a0, a1, f0, f1, a));     // after the rows
  else k<<<grid, BW_THREADS, C::SMEM, c->stream>>>(a0, a1, f0, f1, a);
  SPION_LAUNCH_CHECK();
  c->launches += 1;
  return SPION_OK;
}

template <int D, int SIDE>
static int bw_launch(spion_ctx* c, TcState* s, const CUtensorMap& a0, const CUtensorMap& a1, const CUtensorMap& f0, const CUtensorMap& f1,
                     const BwArgs& a) {
  if (a.factor) return a.keypad ? bw_launch_one<D, SIDE, false, true, true>(c, s, a0, a1, f0, f1, a) : bw_launch_one<D, SIDE, false, false, true>(c, s, a0, a1, f0, f1, a);
  if (a.submask)
    return a.keypad ? bw_launch_one<D, SIDE, true, true, false>(c, s, a0, a1, f0, f1, a) : bw_launch_one<D, SIDE, true, false, false>(c, s, a0, a1, f0, f1, a);
  return a.keypad ? bw_launch_one<D, SIDE, false, true, false>(c, s, a0, a1, f0, f1, a) : bw_launch_one<D, SIDE, false, false, false>(c, s, a0, a1, f0, f1, a);
}

template <int D, bool SUB, bool KP, bool RND>
static int bw_attrs(int device) {
  const int rc = allow_smem<k_bwd_stream<D, ROW, SUB, KP, RND>>(device, Bw<D, ROW>::SMEM);
  return rc ? rc : allow_smem<k_bwd_stream<D, COL, SUB, KP, RND>>(device, Bw<D, COL>::SMEM);
}
template <int D, bool KP>
static int bw_attrs_of(const spion_ctx* c) {
  if (c->bs == 32) return bw_attrs<D, true, KP, false>(c->device);
  const int rc = bw_attrs<D, false, KP, false>(c->device);
  return rc ? rc : bw_attrs<D, false, KP, true>(c->device);
}
int stream_backward_set_attrs(const spion_ctx* c) {
  const bool kp = c->kind == SPION_KIND_BLOCK_KPM;
  if (c->d == 64) return kp ? bw_attrs_of<64, true>(c) : bw_attrs_of<64, false>(c);
  return kp ? bw_attrs_of<32, true>(c) : bw_attrs_of<32, false>(c);
}

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
  if (s->super) {                                                   // at most one pair per block
    if (!s->gather_rec && device_alloc((void**)&s->gather_rec, (SPION_MAX_NB / 2) * sizeof(int4)) != SPION_OK) return SPION_ERR_ALLOC;
    if ((size_t)c->nnzb > s->gather_cap) {
      device_free(s->gather_pair);
      s->gather_pair = nullptr;
      s->gather_cap = 0;
      if (device_alloc((void**)&s->gather_pair, (size_t)c->nnzb * sizeof(int4)) != SPION_OK) return SPION_ERR_ALLOC;
      s->gather_cap = (size_t)c->nnzb;
    }
    k_gather_recs<<<1, 512, 0, c->stream>>>(c->mat, c->nb, s->gather_rec, s->gather_pair);
    SPION_LAUNCH_CHECK();
    c->launches += 1;
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
                      const float* keypad, void* dQ, void* dK, void* dV, bool rounded) {
  const TcView vw = tc_view(c, s);
  CUtensorMap mq, mk, mv, mdo;
  int rc;
  if ((rc = make_operand_map(c, s, &mq, Q, D)) || (rc = make_operand_map(c, s, &mk, K, D)) || (rc = make_operand_map(c, s, &mv, V, D)) ||
      (rc = make_operand_map(c, s, &mdo, dO, D)))
    return rc;
  BwArgs a;
  a.lse = lse; a.keypad = keypad;
  a.factor = rounded ? lse + (size_t)c->BH * c->L : nullptr;
  a.delta = a.delta_out = s->delta_ws;
  a.O = (const __nv_bfloat16*)O; a.dO = (const __nv_bfloat16*)dO;
  a.submask = vw.submask;
  a.L = c->L; a.BH = c->BH; a.nb = vw.nb; a.heads = c->heads; a.by_rank = order_by_rank(c);
  a.scale = c->scale; a.status = c->status_dev;
  prof_mark(c, -1);
  a.rec = s->line_rec + SPION_MAX_NB; a.pair = s->line_pair + s->line_pair_cap;
  a.out0 = (__nv_bfloat16*)dQ; a.out1 = nullptr;
  rc = bw_launch<D, ROW>(c, s, mk, mv, mq, mdo, a);
  if (rc) return rc;
  prof_mark(c, SPION_STAGE_BWD_ROW_RC);
  a.rec = s->line_rec; a.pair = s->line_pair;
  a.out0 = (__nv_bfloat16*)dK; a.out1 = (__nv_bfloat16*)dV;
  rc = bw_launch<D, COL>(c, s, mq, mdo, mk, mv, a);
  if (rc) return rc;
  prof_mark(c, SPION_STAGE_BWD_COL_RC);
  return SPION_OK;
}

int recompute_backward(spion_ctx* c, TcState* s, const void* Q, const void* K, const void* V, const void* O, const void* dO, const float* lse,
                       const float* keypad, void* dQ, void* dK, void* dV, bool rounded) {
  return c->d == 64 ? bwd_stream<64>(c, s, Q, K, V, O, dO, lse, keypad, dQ, dK, dV, rounded)
                    : bwd_stream<32>(c, s, Q, K, V, O, dO, lse, keypad, dQ, dK, dV, rounded);
}

}  // namespace tc
