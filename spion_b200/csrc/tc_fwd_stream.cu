// Forward of the block-sparse attention as a streaming pipeline (sm_100a, bf16, 64 x 64 blocks, no stored P): O and one fp32
// log-sum-exp per row (models/block_attn.cu:453-487 fused; softmax semantics as in tc_fused.cu).
//
// One persistent CTA per SM with four groups (three at head_dim 64: tensor memory).  A group has four arithmetic warps (one per tensor-memory
// quadrant), a warp that issues its MMAs and one that loads its tiles, and walks block rows of its own, two blocks ("a pair") at a time:
//     S = Q K_e^T   (M = 64, the second block at lane offset 16: query rows along the lanes, a row owned by lanes l and l + 16)
//     P = exp2(S scale log2e - m), unnormalised, bf16 into tensor memory, in the lanes of S
//     O += P V_e    (M = 64, P from tensor memory: the products of first and of second blocks in lanes of their own, added when the rows are written)
// S of pair j + 1 is computed while pair j is in the arithmetic (its 64 values per lane are in registers), and the rows of a
// finished unit are written before the first product of the next one.  Nothing is exchanged between the groups: they only fill each
// other's waits.
//
// One pass over a row: m is the maximum of its first pair and is only moved (O and the running sum rescaled) when a later
// score exceeds it by more than 2^8 (the conditional rescaling published with FlashAttention-4), so that almost no row is ever
// rescaled; the result is divided by the sum against the true maximum at the end.  P <= 2^8 loses nothing in bf16 or in the fp32 sums.
//
// What bounds it: per pair the exponentials, 8192 at 16 per cycle and SM = 512 cycles, and at head_dim 64 sixteen MMAs of 32 cycles (M = 64 runs
// at half rate) and 640 cycles of shared memory at 128 bytes (tiles in 256, operands out 384; with P there too, as before, 912 of the 950
// that a pair took).  What it takes beside those, 890 (head_dim 64) and 750, is the chain of a pair: one warp that did the loads and
// the MMAs of a group took as long for them as a pair does, so they are two, and the MMAs are issued by one thread that does nothing else.
// Measured, forward alone, first form (one unit per CTA, two passes over a row), P in shared memory, now: 64 matrices, L = 16384, d 64, 5 % 847,
// 368, 345 us, d 32 -, 312, 292; 256 matrices, L = 4096, d 32, 10 %, padded keys 585, 200, 185; 64 matrices, L = 4096, d 64, 5 % 62, 43.5, 43.
//
// SUB: masks of 32-wide blocks.  A unit is two block rows, a tile two key blocks of 32 that one of them selects, wherever they lie (two copies
// of 32 rows each); quarters that are not selected are left out of the sums, and rows that
// an infinity or a NaN in their values reaches are formed again at the end (redo_rows).  Random masks fill half of such tiles, a third to a quarter of tiles of 64 keys in
// a row.  Us, forward, before (head_dim 64 the mask's own blocks in transposed products, k_b32; 32 such tiles) and now: 64 matrices, L = 4096, d 64, 2 %
// 45, 39; 5 % 122, 70; 10 % 208, 119; 30 % 528, 280; 16 matrices, 5 %, padded keys 40, 29; d 32, 5 % 74, 52; 32 matrices, 15 %, padded keys 107, 73.
// Masks that run on their own blocks (head_dim 64): the reference follows every new maximum, as the kernel before had it: the largest P of a row is 1,
// which bf16 has without rounding.  Moved by 2^8 only, O is 3 % further from fp64 (2.26e-3 instead of 2.14e-3, before 2.18e-3) and the first three
// figures 39, 63, 101.  On derived super-blocks it moves by 2^8, as it did there: 64 matrices, L = 4096, d 64, tiles of 64 keys, every maximum, now: 5 %
// 105, 83, 72; 95 % 415, 510, 424; whole 64 x 64 blocks 5 % 54, 63, 55.
//
// Every wait is bounded; on a time-out the waiting warp records a code in the status word and the CTA winds down.
#include "tc_stream.cuh"

using namespace tc;

namespace {

constexpr float MOVE = 8.0f;                                      // log2 units by which a score may exceed m

template <int D> struct Fs {
  using T = OpTile<D>;
  static constexpr int NG = D == 64 ? 3 : 4;                      // groups: as many as tensor memory holds
  // Warps: four arithmetic ones per group, then one per group that issues its MMAs, one per group that loads its tiles, and idle ones up to two
  // whole warpgroups, so that the arithmetic warps can take registers of the others (setmaxnreg).
  static constexpr int THREADS = 32 * (4 * NG + 8);
  static constexpr int REGS = NG == 4 ? 80 : 96, REGS_A = NG == 4 ? 96 : 120, REGS_S = NG == 4 ? 48 : 56;         // at launch, arithmetic, others
  static_assert(4 * NG * REGS_A + 8 * REGS_S <= (4 * NG + 8) * REGS, "setmaxnreg would wait for ever");
  static constexpr int KB = D == 64 ? 1 : 2;                      // buffers for the K tiles of a pair
  static constexpr uint32_t O_Q = 0, O_K = 2 * T::BYTES, O_V = O_K + 2 * KB * T::BYTES, GROUP = O_V + 4 * T::BYTES;      // Q of two units, V of two pairs
  static constexpr uint32_t O_BAR = NG * GROUP;
  static constexpr uint32_t GBAR = 128;                           // barriers of a group
  static constexpr uint32_t O_INFO = O_BAR + NG * GBAR + 16;      // of a group: records of eight pairs, flags of four
  static constexpr size_t SMEM = O_INFO + NG * 256;
  static constexpr uint32_t T_P = 64, T_O = 96, COLS = 96 + D;    // tensor-memory columns of a group: S, P, O
};

constexpr int PR_TWO = 1, PR_FIRST = 2, PR_END = 4;               // two blocks; first pair of a unit; no pair

struct FsArgs {
  const __nv_bfloat16 *Q, *K, *V;                                 // SUB: for the rows that are formed again
  __nv_bfloat16* O;
  float* lse;
  const float* keypad;
  const int4 *rec, *pair;                                         // block rows and their pairs (k_line_recs; SUB: k_gather_recs)
  int L, BH, nb, heads, by_rank;
  float scale, floor_v, move_by;                                  // move_by: D == 64 and SUB only
  int* status;
};

// SUB: the rows of one arithmetic warp (quadrant q) that are not finite, from the blocks that they select alone.  A tile also holds blocks that only
// the other row of the pair selects, and P = 0 times an infinity or a NaN in their values is a NaN.  The log-sum-exp is right already: scores
// that a row does not select are left out, not multiplied.  Plain fp32 by the lanes that own the columns; a call whose values are finite only pays for
// the test of its outputs.  Rows that are NaN whatever the others hold, by their log-sum-exp or by a NaN of their own in every column that is not finite, stay.
// A lane walks its row's keys alone: one infinity in 8 matrices, L = 16384, 30 %, d 64 makes 0.5 ms of the call 18; NaN everywhere 0.4.
template <int D, bool KP>
__device__ __noinline__ void redo_rows(const FsArgs& a, int first, int step, int total, int q) {
  const int hf = (threadIdx.x >> 4) & 1, row = q * 16 + (threadIdx.x & 15);
  Walk u;
  u.init(UnitMap{a.nb, a.BH, a.by_rank}, a.rec, first, step, total);
#pragma unroll 1
  for (; u.valid(); u.shift()) {
    const int n = u.cur.w;
    const OpPos pos = op_pos(u.bh, a.L, a.heads, D);
    auto at = [&](int r) { return (size_t)(pos.row0 + r) * pos.ld + pos.x0; };
    __nv_bfloat16* dst = a.O + at(u.cur.x * BS + row) + hf * 16;          // columns 32 i + 16 hf ..
    uint32_t bad = 0;
    for (int x = 0; x < D / 2; ++x) bad |= !isfinite(__bfloat162float(dst[(x >> 4) * 32 + (x & 15)])) ? 1u << x : 0u;
    const float lse = a.lse[(size_t)u.bh * a.L + u.cur.x * BS + row];
    if (n == 0 || !bad || isnan(lse)) continue;                   // (an infinity: every P of the row is zero)
    // f of the keys that the row selects, while it returns true
    auto keys = [&](auto f) {
#pragma unroll 1
      for (int t = 0; t < 2 * n; ++t) {                           // halves of the tiles: blocks of 32 keys
        const int4 pr = a.pair[u.cur.y + (t >> 2)];
        const int cols = t & 2 ? pr.y : pr.x, bits = (t & 2 ? pr.w : pr.z) >> ((q >> 1) * 2);
        if (!((bits >> (t & 1)) & 1)) continue;
        const int key0 = ((cols >> (16 * (t & 1))) & 0xffff) * 32;
#pragma unroll 1
        for (int key = key0; key < key0 + 32; ++key)
          if (!f(key)) return;
      }
    };
    auto values = [&](int key, auto f) {                          // this lane's columns of a key, two at a time
      const __nv_bfloat16* vr = a.V + at(key) + hf * 16;
#pragma unroll
      for (int i = 0; i < D / 16; ++i) {
        const uint4 y = *reinterpret_cast<const uint4*>(vr + (i >> 1) * 32 + (i & 1) * 8);
        const uint32_t ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) f(8 * i + 2 * e, bf16_lo(ys[e]), bf16_hi(ys[e]));
      }
    };
    keys([&](int key) {
      values(key, [&](int x, float lo, float hi) { bad &= ~((isnan(lo) ? 1u << x : 0u) | (isnan(hi) ? 2u << x : 0u)); });
      return bad != 0;
    });
    if (!bad) continue;
    const uint4* qr = reinterpret_cast<const uint4*>(a.Q + at(u.cur.x * BS + row));
    const float sc2 = a.scale * LOG2E;
    float o[D / 2];
#pragma unroll
    for (int x = 0; x < D / 2; ++x) o[x] = 0.f;
    keys([&](int key) {
      const uint4* kr = reinterpret_cast<const uint4*>(a.K + at(key));
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        const uint4 x = qr[i], y = kr[i];
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) s = fmaf(bf16_hi(xs[e]), bf16_hi(ys[e]), fmaf(bf16_lo(xs[e]), bf16_lo(ys[e]), s));
      }
      const float pen = KP ? a.keypad[(size_t)u.bh * a.L + key] * LOG2E : 0.f, p = exp2f(fmaf(s, sc2, -pen) - lse);
      values(key, [&](int x, float lo, float hi) { o[x] = fmaf(p, lo, o[x]); o[x + 1] = fmaf(p, hi, o[x + 1]); });
      return true;
    });
#pragma unroll
    for (int i = 0; i < D / 16; ++i)
      *reinterpret_cast<uint4*>(dst + (i >> 1) * 32 + (i & 1) * 8) =
          make_uint4(pack_bf16(o[8 * i], o[8 * i + 1]), pack_bf16(o[8 * i + 2], o[8 * i + 3]), pack_bf16(o[8 * i + 4], o[8 * i + 5]),
                     pack_bf16(o[8 * i + 6], o[8 * i + 7]));
  }
}

template <int D, bool KP, bool SUB>
__global__ void __launch_bounds__(Fs<D>::THREADS, 1) k_fwd_stream(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ FsArgs a) {
  using C = Fs<D>;
  using T = OpTile<D>;
  constexpr int NG = C::NG;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);                      // must be 1024-aligned (checked below)
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int grp = warp < 4 * NG ? warp >> 2 : (warp - 4 * NG) & 3;          // arithmetic warps, four for MMAs, four for loads
  const uint32_t gb = sbase + grp * C::GROUP, bars = sbase + C::O_BAR + grp * C::GBAR;
  // k_full[KB]: K tiles of a pair, Q with the first of a unit, and the pair's record; k_free[KB]: S of that pair complete; v_full[2]: V tiles
  // landed; v_free[2]: product of that pair complete; s_ready: S of a pair complete; s_free: read out (4 warps); p_ready: P of a pair written
  // (4 warps); pv_done: O += P V of a pair complete; pi_full[4]: flags of a pair written.  A parity tells two phases apart.  Every waiter waits
  // for each phase, and the next one needs something that comes after that wait: S of pair j + 1 the four arrivals on s_free for pair j, the
  // product of pair j + 1 those on p_ready, which follow the warps' wait for the product of pair j, tiles a buffer that the loader saw free.
  // Records and flags of pair j are written when S of pair j - KB is complete, so the arithmetic of pair j - 3 has read its own.
  constexpr uint32_t B_KFULL = 0, B_KFREE = 16, B_VFULL = 32, B_VFREE = 48, B_SREADY = 64, B_SFREE = 72, B_PREADY = 80, B_PV = 88, B_PI = 96;
  const uint32_t k_full = bars + B_KFULL, k_free = bars + B_KFREE, v_full = bars + B_VFULL, v_free = bars + B_VFREE, s_ready = bars + B_SREADY,
                 s_free = bars + B_SFREE, p_ready = bars + B_PREADY, pv_done = bars + B_PV, pi_full = bars + B_PI;
  constexpr int KB = C::KB;
  const uint32_t slot = sbase + C::O_BAR + NG * C::GBAR, abort_w = slot + 4;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - sbase));
  volatile int* abort_ptr = reinterpret_cast<volatile int*>(smem_raw + (abort_w - sbase));
  // records [8]: {PR_*| (b,h) << 4, block columns c0 | c1 << 16, CSR block ids};  flags [4][8]: which blocks have different penalties and
  // which quarters are selected, block columns, -, one penalty per block in base-2 units
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
  const uint32_t tmem = *slot_ptr, tS = tmem + grp * C::COLS, tP = tS + C::T_P, tO = tS + C::T_O;
  auto wait_all = [&](uint32_t bar, uint32_t parity, int code) -> bool { return warp_wait(bar, parity & 1u, a.status, code); };
  const UnitMap um{a.nb, a.BH, a.by_rank};
  // group g of CTA b walks units b + g G, + NG G, ...
  const int first = (int)blockIdx.x + grp * (int)gridDim.x, step = NG * (int)gridDim.x, total = a.nb * a.BH;

  auto wait_one = [&](uint32_t bar, uint32_t parity, int code) -> bool {           // one thread
    if (mbar_wait(bar, parity & 1u)) return true;
    report(a.status, code);
    return false;
  };
  if (warp < 4 * NG) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REGS_A));
  else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REGS_S));

  if (warp >= 4 * NG + 4) {
    // ================================================================== loads of a group
    Walk w;
    w.init(um, a.rec, first, step, grp < NG ? total : 0);
    w.skip();
    int4 pr = w.valid() ? a.pair[w.cur.y] : make_int4(0, -1, 0, 0), nx = pr;       // records of pairs j, j + 1
    int units = 0;
    for (int j = 0; grp < NG; ++j) {
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
      const bool two = w.cnt() == 2, with_q = w.k == 0;
      const OpPos pos = op_pos(w.bh, a.L, a.heads, D);
      const int bh = w.bh, line = w.cur.x;
      // SUB: lanes 0 to 3 copy a quarter of a pair's tiles each
      const int piece = (lane & 2 ? pr.y : pr.x) >> ((lane & 1) * 16) & 0xffff;
      const bool mine = SUB && lane < (two ? 4 : 2);
      if (elect_one()) {
        ring[j & 7] = make_int4((two ? PR_TWO : 0) | (with_q ? PR_FIRST : 0), 0, 0, 0);
        mbar_expect_tx(kb, ((two ? 2 : 1) + (with_q ? 1 : 0)) * T::BYTES);
        const uint32_t dst = gb + C::O_K + (j % KB) * 2 * T::BYTES;
        if (!SUB) {
          tma_load_2d(dst, &tmK, kb, pos.x0, pos.row0 + pr.x * BS);
          if (two) tma_load_2d(dst + T::BYTES, &tmK, kb, pos.x0, pos.row0 + pr.y * BS);
        }
        // the Q buffer was read by the unit before the last, whose last pair is not after the one k_free was for
        if (with_q) tma_load_2d(gb + C::O_Q + (units & 1) * T::BYTES, &tmQ, kb, pos.x0, pos.row0 + line * BS);
      }
      __syncwarp();
      if (mine) tma_load_2d(gb + C::O_K + (j % KB) * 2 * T::BYTES + lane * (T::BYTES / 2), &tmK, kb, pos.x0, pos.row0 + piece * 32);
      if (w.last()) ++units;
      w.next();
      if (w.valid()) nx = a.pair[w.cur.y + w.k];
      if (KP || SUB) {
        const int e = lane >> 4, o = e ? pr.y : pr.x;
        const bool here = !e || two;
        uint32_t mixed = 0u;
        float pen = 0.f, pen1 = 0.f;
        if (KP) {
          Pen4 p = {};
          const float* kp = a.keypad + (size_t)bh * a.L;
          if (here && SUB) pen_load(p, kp + (o & 0xffff) * 32, kp + (o >> 16) * 32);
          else if (here) pen_load(p, kp + o * BS);
          pen = pen_of(p, mixed) * LOG2E;
          pen1 = __shfl_sync(0xffffffffu, pen, 16);
        }
        const int sub_l = SUB && here ? (e ? pr.w : pr.z) : 0;
        const int s1 = SUB ? __shfl_sync(0xffffffffu, sub_l, 16) : 0xff;
        if (lane == 0) {
          int* x = info + 8 * (j & 3);
          x[0] = (int)mixed | ((SUB ? sub_l : 0xff) << 8) | (s1 << 16);
          x[1] = pr.x; x[2] = pr.y;
          if (KP) { x[4] = __float_as_int(pen); x[5] = __float_as_int(pen1); }
          mbar_arrive(pi_full + 8 * (j & 3));
        }
        __syncwarp();
      }
      if (j >= 2 && !wait_all(v_free + 8 * (j & 1), (uint32_t)(j >> 1) - 1u, ERR_MMA2_WAIT)) break;
      if (elect_one()) {
        const uint32_t vb = v_full + 8 * (j & 1), dst = gb + C::O_V + (j & 1) * 2 * T::BYTES;
        mbar_expect_tx(vb, (two ? 2 : 1) * T::BYTES);
        if (!SUB) {
          tma_load_2d(dst, &tmV, vb, pos.x0, pos.row0 + pr.x * BS);
          if (two) tma_load_2d(dst + T::BYTES, &tmV, vb, pos.x0, pos.row0 + pr.y * BS);
        }
      }
      __syncwarp();
      if (mine) tma_load_2d(gb + C::O_V + (j & 1) * 2 * T::BYTES + lane * (T::BYTES / 2), &tmV, v_full + 8 * (j & 1), pos.x0, pos.row0 + piece * 32);
      pr = nx;
    }
  } else if (warp >= 4 * NG) {
    // ================================================================== MMAs of a group: one thread
    if (grp < NG && elect_one()) {
      constexpr uint32_t IDESC_S = make_idesc_bf16(64, 64, 0, 0), IDESC_O = make_idesc_bf16(64, D, 0, 1);
      const uint64_t dQ = T::kmajor(gb + C::O_Q, 0), dK = T::kmajor(gb + C::O_K, 0), dV = T::mnmajor(gb + C::O_V, 0);
      int units = 0;                                              // units up to the one of pair j
      int prev = 0;                                               // record of pair j - 1
      for (int j = 0;; ++j) {
        if (!wait_one(k_full + 8 * (j % KB), (uint32_t)(j / KB), ERR_LOAD_WAIT)) break;
        const int now = ring[j & 7].x;
        if (!(now & PR_END)) {                                    // S of pair j
          if (now & PR_FIRST) ++units;
          if (j >= 1 && !wait_one(s_free, (uint32_t)(j - 1), ERR_MMA_WAIT)) break;
          tc_fence_after();
          const uint64_t q = desc_advance(dQ, ((units - 1) & 1) * T::BYTES), k = desc_advance(dK, (j % KB) * 2 * T::BYTES);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_bf16(tS, desc_advance(q, kk * T::K_STEP), desc_advance(k, kk * T::K_STEP), IDESC_S, kk > 0);
          if (now & PR_TWO) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              mma_bf16(tS + (16u << 16), desc_advance(q, kk * T::K_STEP), desc_advance(k, T::BYTES + kk * T::K_STEP), IDESC_S, kk > 0);
          }
          mma_commit(s_ready);
          mma_commit(k_free + 8 * (j % KB));
        }
        if (j >= 1) {                                             // O += P V of pair j - 1
          const int jp = j - 1;
          if (!wait_one(v_full + 8 * (jp & 1), (uint32_t)(jp >> 1), ERR_LOAD_WAIT)) break;
          if (!wait_one(p_ready, (uint32_t)jp, ERR_MMA_WAIT)) break;
          tc_fence_after();
          const uint32_t more = (prev & PR_FIRST) ? 0u : 1u;      // not the first product of its unit
          const uint64_t v = desc_advance(dV, (jp & 1) * 2 * T::BYTES);
#pragma unroll
          for (int kk = 0; kk < BS / 16; ++kk) mma_bf16_ts(tO, tP + kk * 8u, desc_advance(v, kk * T::MN_STEP), IDESC_O, kk > 0 ? 1u : more);
          if (prev & PR_TWO) {
#pragma unroll
            for (int kk = 0; kk < BS / 16; ++kk)
              mma_bf16_ts(tO + (16u << 16), tP + (16u << 16) + kk * 8u, desc_advance(v, T::BYTES + kk * T::MN_STEP), IDESC_O, kk > 0 ? 1u : more);
          }
          mma_commit(pv_done);
          mma_commit(v_free + 8 * (jp & 1));
        }
        if (now & PR_END) break;
        prev = now;
      }
    }
    __syncwarp();
  } else {
    // ================================================================== arithmetic warps of a group
    const int q = warp & 3, hf = lane >> 4, row = q * 16 + (lane & 15);
    const uint32_t lS = tS + ((uint32_t)(q * 32) << 16), lP = lS + C::T_P, lO = lS + C::T_O;
    const float sc2 = a.scale * LOG2E, floor2 = a.floor_v * LOG2E, inv_scale = 1.0f / a.scale;
    const float move_by = SUB && D == 64 ? a.move_by : MOVE;
    bool ok = true;
    // The finished unit whose rows are still in tensor memory: the products of first entries in lanes 0-15 of every quadrant, of second ones
    // in lanes 16-31.  Lane l gives half of its columns to lane l ^ 16 and takes the other half's from there.
    bool pend = false, pend_two = false;
    bool redo = false;                                            // SUB: something of this lane's is not finite
    float pend_inv = 0.f;
    __nv_bfloat16* pend_dst = nullptr;
    auto put = [&](__nv_bfloat16* dst, const float (&v)[16]) {
#pragma unroll
      for (int x = 0; x < 16; x += 8)
        *reinterpret_cast<uint4*>(dst + x) = make_uint4(pack_bf16(v[x], v[x + 1]), pack_bf16(v[x + 2], v[x + 3]), pack_bf16(v[x + 4], v[x + 5]),
                                                        pack_bf16(v[x + 6], v[x + 7]));
    };
    auto flush = [&]() {                                          // its last product is complete
#pragma unroll
      for (int h = 0; h < D / 32; ++h) {
        uint32_t v[32];
        tmem_ld32(lO + h * 32, v);
        tmem_ld_wait();
        float o[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) {
          const float keep = __uint_as_float(hf ? v[16 + x] : v[x]), give = __uint_as_float(hf ? v[x] : v[16 + x]);
          const float take = __shfl_xor_sync(0xffffffffu, give, 16);
          // one entry: what lanes 16-31 hold was never written
          o[x] = (pend_two ? keep + take : hf ? take : keep) * pend_inv;
        }
        if (SUB) {
          float probe = 0.f;
#pragma unroll
          for (int x = 0; x < 16; ++x) probe = fmaf(o[x], 0.f, probe);
          redo |= !(probe == 0.f);
        }
        put(pend_dst + h * 32 + hf * 16, o);
      }
      pend = false;
    };
    Walk u;
    u.init(um, a.rec, first, step, total);
    int j = 0;
    for (; u.valid() && ok; u.shift()) {
      const int n = u.cur.w;
      const OpPos pos = op_pos(u.bh, a.L, a.heads, D);
      __nv_bfloat16* dst = a.O + (size_t)(pos.row0 + u.cur.x * BS + row) * pos.ld + pos.x0;
      float* lse = a.lse + (size_t)u.bh * a.L + u.cur.x * BS + row;
      if (n == 0) {                                               // a row without blocks: every key counts as score 0
        const float m0 = fmaxf(floor2, -INFINITY);
        if (hf == 0) *lse = m0 + log2f((float)a.L * exp2f(-m0));
        const float zero[16] = {};
        for (int h = 0; h < D; h += 32) put(dst + h + hf * 16, zero);
        continue;
      }
      const float* kpu = KP ? a.keypad + (size_t)u.bh * a.L : nullptr;
      float m = floor2, mx = floor2, l = 0.f;                     // reference exponent, true maximum, sum
      int n_sel = 0;
      const int np = u.pairs();
      for (int k = 0; k < np && ok; ++k, ++j) {
        const bool mine = 2 * k + hf < n;
        const float *kp = nullptr, *kp_hi = nullptr;
        float pen = 0.f;
        bool live0 = mine, live1 = mine;
        if (KP || SUB) {
          if (!wait_all(pi_full + 8 * (j & 3), (uint32_t)(j >> 2), ERR_MMA_WAIT)) { ok = false; break; }
          const int* x = info + 8 * (j & 3);
          const int f = x[0];
          if (KP) {
            const bool mixed = (f >> hf) & 1;
            pen = mixed ? 0.f : __int_as_float(x[4 + hf]);
            if (mixed) {
              kp = SUB ? kpu + (x[1 + hf] & 0xffff) * 32 : kpu + x[1 + hf] * BS;
              kp_hi = SUB ? kpu + (x[1 + hf] >> 16) * 32 : kp + 32;
            }
          }
          if (SUB) {
            const int bits = (f >> (8 + 8 * hf + (q >> 1) * 2)) & 3;
            live0 = mine && (bits & 1);
            live1 = mine && (bits & 2);
            n_sel += mine ? 32 * __popc(bits) : 0;
          }
        }
        if (!SUB) n_sel += mine ? BS : 0;
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
          take_penalty(v1, kp_hi, inv_scale);
        }
        float cm = -INFINITY;
        {                                                         // the scale is positive: compare raw scores
          float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            m0 = max3(m0, __uint_as_float(v0[x]), __uint_as_float(v0[x + 1]));
            m1 = max3(m1, __uint_as_float(v0[x + 2]), __uint_as_float(v0[x + 3]));
            m2 = max3(m2, __uint_as_float(v1[x]), __uint_as_float(v1[x + 1]));
            m3 = max3(m3, __uint_as_float(v1[x + 2]), __uint_as_float(v1[x + 3]));
          }
          if (live0) cm = fmaf(fmaxf(m0, m1), sc2, -pen);
          if (live1) cm = fmaxf(cm, fmaf(fmaxf(m2, m3), sc2, -pen));
        }
        cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, 16));     // both owners of a row agree
        mx = fmaxf(mx, cm);
        if (k == 0) {
          m = mx;
        } else if (__any_sync(0xffffffffu, mx > m + move_by)) {      // rare: move the reference, rescale what has been summed
          const float m_new = mx > m + move_by ? mx : m, f = exp2f(m - m_new);
          l *= f;
          m = m_new;
          if (!wait_all(pv_done, (uint32_t)(j - 1), ERR_MMA2_WAIT)) { ok = false; break; }
          tc_fence_after();
#pragma unroll 1
          for (int h = 0; h < D; h += 8) {
            uint32_t o[8];
            tmem_ld8(lO + h, o);
            tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 8; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * f);
            tmem_st8(lO + h, o);
          }
          tmem_st_wait();
        }
        uint64_t l2 = 0ull;
        const uint64_t sc22 = pack2(sc2, sc2), nm2 = pack2(-(m + pen), -(m + pen));
        // P of 32 keys, two per register
        auto half_row = [&](uint32_t (&v)[32], bool live) {
          uint64_t sum = 0ull;
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            float e0, e1;
            unpack2(fma2(pack2(v[2 * x], v[2 * x + 1]), sc22, nm2), e0, e1);
            e0 = ex2_approx(e0); e1 = ex2_approx(e1);
            sum = add2(sum, pack2(e0, e1));
            v[x] = pack_bf16(e0, e1);
          }
          if (!live) {
            sum = 0ull;
#pragma unroll
            for (int x = 0; x < 16; ++x) v[x] = 0u;
          }
          l2 = add2(l2, sum);
        };
        half_row(v0, live0);
        // P and O of the pair before: by now its product has long been issued
        if (j >= 1 && !wait_all(pv_done, (uint32_t)(j - 1), ERR_MMA2_WAIT)) { ok = false; break; }
        tc_fence_after();
        tmem_st16(lP, v0);
        half_row(v1, live1);
        tmem_st16(lP + 16u, v1);
        float la, lb;
        unpack2(l2, la, lb);
        l += la + lb;
        if (pend) flush();                                        // the previous unit, before this one's first product
        tmem_st_wait();
        tc_fence_before();                                        // P -> visible to the MMA
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready);
      }
      if (!ok) break;
      n_sel += __shfl_xor_sync(0xffffffffu, n_sel, 16);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      const float f = exp2f(m - mx), z = l * f + (float)(a.L - n_sel) * exp2f(-mx);
      if (hf == 0) *lse = mx + log2f(z);
      pend = true; pend_two = n > 1; pend_inv = f / z; pend_dst = dst;
    }
    if (ok && pend && wait_all(pv_done, (uint32_t)(j - 1), ERR_MMA2_WAIT)) {
      tc_fence_after();
      flush();
      if (SUB && __any_sync(0xffffffffu, redo)) {
        __syncwarp();                                             // the rows' sums are one half-warp's
        redo_rows<D, KP>(a, first, step, total, q);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512u);
}

}  // namespace

namespace tc {

template <int D, bool KP, bool SUB>
static int fs_launch(spion_ctx* c, TcState* s, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const FsArgs& a) {
  using C = Fs<D>;
  static_assert(C::SMEM <= 227 * 1024 && C::NG * C::COLS <= 512, "shared or tensor memory");
  constexpr auto k = k_fwd_stream<D, KP, SUB>;
  int rc = allow_smem<k>(c->device, C::SMEM);
  if (rc) return rc;
  const long long total = (long long)c->BH * a.nb;
  const int grid = (int)(total < (long long)s->sms ? total : (long long)s->sms);       // one CTA per SM (all 512 TMEM columns)
  k<<<grid, C::THREADS, C::SMEM, c->stream>>>(mq, mk, mv, a);
  SPION_LAUNCH_CHECK();
  c->launches += 1;
  return SPION_OK;
}

template <int D>
static int fs_forward(spion_ctx* c, TcState* s, const void* Q, const void* K, const void* V, const float* keypad, void* O, float* lse) {
  const TcView vw = tc_view(c, s);
  const int rows = vw.submask ? 32 : BS;
  CUtensorMap mq, mk, mv;
  int rc;
  if ((rc = make_operand_map(c, s, &mq, Q, D)) || (rc = make_operand_map(c, s, &mk, K, D, rows)) || (rc = make_operand_map(c, s, &mv, V, D, rows))) return rc;
  FsArgs a;
  a.Q = (const __nv_bfloat16*)Q; a.K = (const __nv_bfloat16*)K; a.V = (const __nv_bfloat16*)V;
  a.O = (__nv_bfloat16*)O; a.lse = lse; a.keypad = keypad;
  a.rec = vw.submask ? s->gather_rec : s->line_rec + SPION_MAX_NB;
  a.pair = vw.submask ? s->gather_pair : s->line_pair + s->line_pair_cap;
  a.L = c->L; a.BH = c->BH; a.nb = vw.nb; a.heads = c->heads; a.by_rank = order_by_rank(c);
  a.scale = c->scale; a.floor_v = keypad ? 0.0f : -100.0f; a.status = c->status_dev;
  a.move_by = s->b32 && s->b32_use ? 0.f : MOVE;
  if (keypad) return vw.submask ? fs_launch<D, true, true>(c, s, mq, mk, mv, a) : fs_launch<D, true, false>(c, s, mq, mk, mv, a);
  return vw.submask ? fs_launch<D, false, true>(c, s, mq, mk, mv, a) : fs_launch<D, false, false>(c, s, mq, mk, mv, a);
}

template <int D>
static int fs_attrs(const spion_ctx* c) {
  if (c->kind == SPION_KIND_BLOCK_KPM)
    return c->bs == 32 ? allow_smem<k_fwd_stream<D, true, true>>(c->device, Fs<D>::SMEM) : allow_smem<k_fwd_stream<D, true, false>>(c->device, Fs<D>::SMEM);
  return c->bs == 32 ? allow_smem<k_fwd_stream<D, false, true>>(c->device, Fs<D>::SMEM) : allow_smem<k_fwd_stream<D, false, false>>(c->device, Fs<D>::SMEM);
}
int stream_forward_set_attrs(const spion_ctx* c) { return c->d == 64 ? fs_attrs<64>(c) : fs_attrs<32>(c); }

int stream_forward(spion_ctx* c, TcState* s, const void* Q, const void* K, const void* V, const float* keypad, void* O, float* lse) {
  return c->d == 64 ? fs_forward<64>(c, s, Q, K, V, keypad, O, lse) : fs_forward<32>(c, s, Q, K, V, keypad, O, lse);
}

}  // namespace tc
