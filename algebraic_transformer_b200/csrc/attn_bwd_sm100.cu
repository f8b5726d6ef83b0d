// Asinh-power attention backward on tcgen05 tensor cores (the throughput path of alg_attn_bwd).
//
// Same mathematics as attn_bwd_mma.cu (reference: the custom VJP of
// src/algebraic/kernels/flash.py:333-727): with x = q.k / (sqrt(D) c), p rebuilt from the saved
// statistic, delta_i = dO_i . o_i and dP = dO V^T,
//   dS = n p (dP - delta) / sqrt(1 + x^2) / (sqrt(D) c),  dQ = dS K,  dK = dS^T Q,  dV = P^T dO.
// bf16, causal self-attention of any length, head_dim 64 or 128; non-causal and cross-attention shapes
// stay on the mma.sync kernels.
//
// One launch, two kinds of CTA, each for a resident block of 128 rows of one (batch, head):
//   MODE 0 (dQ, dsink)  rows = queries.  Resident: Q, dO.  Streamed: BS keys (K, V) at a time up to
//                       the diagonal.  S = Q K^T, dP = dO V^T, dQ += dS K.
//   MODE 1 (dK, dV)     rows = keys.  Resident: K, V.  Streamed: BS queries (Q, dO) at a time from the
//                       diagonal on.  S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q.
// S is evaluated in both; in exchange there are no atomics on dQ, no fp32 copy of it and no second pass
// that rounds it, and the results repeat bit for bit.
// Roles: warp 0 TMA producer (and, in MODE 1, the streamed queries' statistic and delta into shared
// memory), warp 1 tcgen05.mma issuer, the others the element-wise stage: four warps (one thread = one
// row) per 32 streamed columns.  Tensor memory: the two score tiles (BS columns each), one or two
// D-column accumulators and, where it fits, a second S buffer; the bf16 operands of the second
// products (P^T, dS) are written back over the columns their own thread has already read - columns
// [32 g, 32 g + 32) of scores become [32 g, 32 g + 16) of packed weights - and fed to the tensor core
// from tensor memory (TS form) with the streamed tile as an MN-major B operand, so nothing is
// transposed or staged.  A step has two element-wise phases and the tensor core works on one region
// while the threads work on the other:
//   phase 1  reads S, forms p (MODE 1 writes P^T over S) and keeps p / sqrt(1+x^2) in registers;
//            meanwhile: dK/dQ product of the previous step, then dP of this step;
//   phase 2  reads dP, writes dS = (kept factor) (dP - delta) over it;
//            meanwhile: dV product of this step (MODE 1), then S of the next step.
//
// What bounds it is the chain S -> phase 1 -> phase 2 -> product of a step (tensor-memory latency,
// barrier, arithmetic), not a pipe, so the tile is chosen for the number of independent warps:
//   head_dim 128  BS = 128 and 16 element-wise warps of 32 columns each (tensor memory is full with one
//                 CTA);
//   head_dim 64   BS = 64: a CTA then needs 256 tensor-memory columns and 98 KB of shared memory, and TWO
//                 CTAs share an SM, so one computes while the other waits, loads or stores.  The 64-wide
//                 score products take nearly as long as 128-wide ones; the overlap is worth more.
// Measured (CUDA-graph replay over several sets of inputs, delta kernel included; before = 128-wide steps, 8 warps of 64
// columns, one launch per kind, mma.sync kernels for lengths off 128): (16,12,1024,64) 317 -> 181 us, (8,16,2048,64) 578 -> 384,
// (1,16,8192,64) 808 -> 620, (1,16,8192,128) 1017 -> 900-920, (2,16,1837,128) 591 -> 142, (5,12,489,64) 102 -> 35.
// Other forms of this one, where (16,12,1024,64) took 174 us and (8,16,2048,64) 366 on one set of inputs: BS = 128 with one CTA at
// head_dim 64 245 / 496 us; two warp sets on alternate 64-wide steps in one CTA 257 us (head_dim 128: 1036 against 960), since
// 64-wide score products cost the tensor pipe what 128-wide ones do.
//
// Lengths off the tile: TMA fills rows past the end with zeros.  Keys past the end lie above the
// diagonal of every real query; queries past the end get statistic and delta 0, hence weight 0; rows past
// the end are computed and not stored.
// Every mbarrier wait is bounded; a wait that runs out reports ALG_DEV_TIMEOUT.
#include "common.cuh"
#include "launchers.h"
#include "sm100_ptx.cuh"

#include <type_traits>

namespace alg {
namespace {

using namespace sm100;

constexpr int BT = 128;                          // resident rows of a CTA
constexpr int RES_PANEL = BT * 128;              // one 64-column panel of a resident tile
constexpr int MAX_STEPS = 4;

template <int D, int BS, int CTAS> struct Cfg {
  static constexpr int PANELS = D / 64;
  static constexpr int RES_BYTES = PANELS * RES_PANEL;
  static constexpr int STR_PANEL = BS * 128, STR_BYTES = PANELS * STR_PANEL;
  static constexpr int NS = (D == 128) ? 2 : 4;                 // ring depth in steps (two streamed tiles per step)
  static constexpr int NG = BS / 32;                            // column groups of the element-wise stage
  static constexpr int EW_WARPS = 4 * NG, NTHREADS = 64 + 32 * EW_WARPS;
  static constexpr int RING_OFF = 2 * RES_BYTES;
  static constexpr int VEC_OFF = RING_OFF + NS * 2 * STR_BYTES; // MODE 1: per ring slot BS statistics, BS negated deltas
  static constexpr int CTL_OFF = VEC_OFF + NS * 2 * BS * 4;
  static constexpr uint32_t TMEM_COLS = 512 / CTAS;
  static constexpr uint32_t S_COL = 0, DP_COL = BS, ACC0_COL = 2 * BS, ACC1_COL = 2 * BS + D;
  static constexpr uint32_t s1_col(int mode) { return 2 * BS + (mode + 1) * D; }
  // a second S buffer where tensor memory has room for it: S of step j + 1 is then computed while the threads
  // are still reading S of step j
  static constexpr bool double_s(int mode) { return s1_col(mode) + BS <= TMEM_COLS; }
  static constexpr uint32_t IDESC_S = make_idesc_bf16(BT, BS, 0, 0);
  static constexpr uint32_t IDESC_TS = make_idesc_bf16(BT, D, 0, 1);
};

struct __align__(16) Control {
  uint64_t res_full, full[MAX_STEPS], empty[MAX_STEPS], vec_full[MAX_STEPS], s_full[2], dp_full, p_done[2], ds_done, acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

template <class C> constexpr size_t smem_bytes() { return size_t(C::CTL_OFF) + sizeof(Control) + 1024; }

// 16 scores of this thread's row -> the weights p (packed bf16 pairs in pw) and the factor
// p / sqrt(1 + x^2) that phase 2 multiplies (dP - delta) by.  Packed fp32 pairs throughout.
//
// Unshifted statistic (1 / l): with y the raw score, s = 1 / (sqrt(D) c) and kappa = 1 / s^2,
//   p = (s (y + sqrt(kappa + y^2)))^n / l  and  1 / sqrt(1 + x^2) = rsqrt(kappa + y^2) / s;
// the constant 1 / s joins the factors n s that the epilogue applies.  The statistic multiplies the finished power: as
// s l^(-1/n) ahead of it, one multiplication less, its own rounding came out of the power n times as large, and the
// kernel was hardly faster for it ((16,12,1024,64) 182.0 us against 180.9, (8,16,2048,64) 383 and 384, (1,16,8192,64) 608
// against 622, (2,16,1837,128) 143 and 142).
// Shifted statistic (rho(-m) l^(-1/n)): p = (rho(x) a)^n with the cancellation-free rho and a = the statistic.
// `a` comes by row (MODE 0: a2[0]) or by column (MODE 1: a2[0..7]).
template <bool SHIFTED, bool BY_COLUMN, int LOG2N, bool MASK>
__device__ __forceinline__ void weights16(const uint32_t* s, float2* slope, uint32_t* pw, const float2* a2, float scale,
                                          float kappa, int log2n, int row, int col0) {
  const float2 kp = make_float2(kappa, kappa), sc = make_float2(scale, scale), one = make_float2(1.f, 1.f);
  float2 t[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float2 y = make_float2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
    if (SHIFTED) {
      y = __fmul2_rn(y, sc);
      const float2 rad = __ffma2_rn(y, y, one);
      slope[i] = make_float2(rsqrt_approx(rad.x), rsqrt_approx(rad.y));
      t[i] = make_float2(rho_stable(y.x), rho_stable(y.y));
    } else {
      const float2 rad = __ffma2_rn(y, y, kp);
      slope[i] = make_float2(rsqrt_approx(rad.x), rsqrt_approx(rad.y));
      t[i] = __ffma2_rn(rad, slope[i], y);
    }
    t[i] = __fmul2_rn(t[i], !SHIFTED ? sc : BY_COLUMN ? a2[i] : a2[0]);
  }
  // the power as passes over the eight pairs, so that every pass has independent multiplications
  if (LOG2N > 0) {
#pragma unroll
    for (int it = 0; it < LOG2N; ++it)
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = __fmul2_rn(t[i], t[i]);
  } else {
    for (int it = 0; it < log2n; ++it)
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = __fmul2_rn(t[i], t[i]);
  }
  if (!SHIFTED) {
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = __fmul2_rn(t[i], BY_COLUMN ? a2[i] : a2[0]);
  }
  if (MASK) {   // causal, key <= query: rows are keys where the factors come by column, else queries
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = col0 + 2 * i;
      if (BY_COLUMN ? (c < row) : (c > row)) t[i].x = 0.f;
      if (BY_COLUMN ? (c + 1 < row) : (c + 1 > row)) t[i].y = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    slope[i] = __fmul2_rn(slope[i], t[i]);
    if (BY_COLUMN) pw[i] = pack_bf16(t[i].x, t[i].y);
  }
}

// Phase 1 on this thread's 32 scores at tensor-memory address s_t; `vec`: the columns' statistics in shared memory
// (MODE 1).  MODE 1 leaves the packed weights over the columns read.
template <int MODE, bool SHIFTED, int LOG2N, bool MASK>
__device__ __forceinline__ void phase1(uint32_t s_t, float2* slope, const float* vec, float2 a_row, float scale, float kappa,
                                       int log2n, int row, int col0) {
  uint32_t s0[16], s1[16];
  tmem_ld_32x16(s_t, s0);
  tmem_ld_wait_for16(s0);
  tmem_ld_32x16(s_t + 16, s1);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t pw[8];
    float2 a2[8];
    if (MODE == 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(vec + c * 16 + 4 * i);
        a2[2 * i] = make_float2(v.x, v.y);
        a2[2 * i + 1] = make_float2(v.z, v.w);
      }
    } else {
      a2[0] = a_row;
    }
    if (c == 1) tmem_ld_wait_for16(s1);
    weights16<SHIFTED, MODE == 1, LOG2N, MASK>(c == 0 ? s0 : s1, slope + 8 * c, pw, a2, scale, kappa, log2n, row, col0 + c * 16);
    if (MODE == 1) tmem_st_32x8(s_t + c * 8, pw);
  }
}

template <class C, int D, int BS, int MODE>
__device__ __forceinline__ void bwd_block(unsigned char* smem, Control* ctl, const CUtensorMap* tm_q, const CUtensorMap* tm_k,
                                          const CUtensorMap* tm_v, const CUtensorMap* tm_do, const AttnBwdParams& p, int tile) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem_base = ctl->tmem_base;
  const BoundedWait bw{&ctl->abort_flag, 1000000000ull};
  constexpr bool DB = C::double_s(MODE);
  auto sbuf = [](int j) { return DB ? (j & 1) : 0; };
  auto sphase = [](int j) -> uint32_t { return DB ? ((j >> 1) & 1u) : (j & 1u); };
  auto s_col = [](int j) -> uint32_t { return (DB && (j & 1)) ? C::s1_col(MODE) : C::S_COL; };

  const int h = blockIdx.x, b = blockIdx.y;
  const int row0 = tile * BT;
  const int first = (MODE == 0) ? 0 : row0;                  // first streamed row
  const int end = (MODE == 0) ? min(row0 + BT, p.Tq) : p.Tq; // one past the last
  const int nsteps = (end - first + BS - 1) / BS;
  const bool shifted = *p.stat_kind == ALG_VARIANT_SHIFT;
  const int64_t bh = int64_t(b) * p.H + h;

  if (warp == 0) {
    const CUtensorMap* res0 = (MODE == 0) ? tm_q : tm_k;     // A operand of the first score product
    const CUtensorMap* res1 = (MODE == 0) ? tm_do : tm_v;    // A operand of the second
    const CUtensorMap* str0 = (MODE == 0) ? tm_k : tm_q;     // their streamed B operands
    const CUtensorMap* str1 = (MODE == 0) ? tm_v : tm_do;
    if (lane == 0) {
      mbar_arrive_expect_tx(&ctl->res_full, 2 * C::RES_BYTES);
      for (int pn = 0; pn < C::PANELS; ++pn)
        for (int r = 0; r < BT; r += BS) {                   // boxes are BS rows high
          tma_load_4d(smem + pn * RES_PANEL + r * 128, res0, &ctl->res_full, pn * 64, row0 + r, h, b);
          tma_load_4d(smem + C::RES_BYTES + pn * RES_PANEL + r * 128, res1, &ctl->res_full, pn * 64, row0 + r, h, b);
        }
    }
    // MODE 1: statistic and delta of the next step's queries, fetched one step ahead
    constexpr int VPL = BS / 32;
    float st[VPL], dl[VPL];
    auto fetch = [&](int j) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int t = first + j * BS + i * 32 + lane;
        const bool in = t < p.Tq;
        st[i] = in ? __ldg(p.stat + bh * p.Tq + t) : 0.f;
        dl[i] = in ? __ldg(p.delta + bh * p.Tq + t) : 0.f;
      }
    };
    if (MODE == 1) fetch(0);
    for (int j = 0; j < nsteps; ++j) {
      const int slot = j % C::NS;
      if (__any_sync(0xffffffffu, !bw.wait(&ctl->empty[slot], ((j / C::NS) & 1u) ^ 1u))) break;
      if (lane == 0) {
        unsigned char* dst = smem + C::RING_OFF + slot * 2 * C::STR_BYTES;
        mbar_arrive_expect_tx(&ctl->full[slot], 2 * C::STR_BYTES);
        for (int pn = 0; pn < C::PANELS; ++pn) {
          tma_load_4d(dst + pn * C::STR_PANEL, str0, &ctl->full[slot], pn * 64, first + j * BS, h, b);
          tma_load_4d(dst + C::STR_BYTES + pn * C::STR_PANEL, str1, &ctl->full[slot], pn * 64, first + j * BS, h, b);
        }
      }
      if (MODE == 1) {
        float* vec = reinterpret_cast<float*>(smem + C::VEC_OFF) + slot * 2 * BS;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
          vec[i * 32 + lane] = st[i];
          vec[BS + i * 32 + lane] = -dl[i];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->vec_full[slot]);
        if (j + 1 < nsteps) fetch(j + 1);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // the whole warp runs the loop and one elected lane issues (cheaper per issue than a lane-0 branch)
    auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, bw.wait(bar, parity)) != 0; };
    const uint32_t res_addr = smem_u32(smem), ring_addr = smem_u32(smem + C::RING_OFF);
    const uint32_t a0_lo = sw128_desc_lo(res_addr, 16), a1_lo = sw128_desc_lo(res_addr + C::RES_BYTES, 16);
    // S-like product: d = A . B^T, both K-major tiles of D columns
    auto issue_scores = [&](uint32_t d_tmem, uint32_t a_lo, uint32_t b_addr) {
      const uint32_t b_lo = sw128_desc_lo(b_addr, 16);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const uint32_t a_off = ((ks >> 2) * RES_PANEL + (ks & 3) * 32) >> 4, b_off = ((ks >> 2) * C::STR_PANEL + (ks & 3) * 32) >> 4;
        umma_f16_ss_parts(d_tmem, a_lo + a_off, SW128_DESC_HI, b_lo + b_off, SW128_DESC_HI, C::IDESC_S, ks != 0 ? 1u : 0u);
      }
    };
    // acc += W . B: W = packed bf16 in tensor memory (see the head of the file), B = a streamed [row][D] tile read
    // as an MN-major operand
    auto issue_product = [&](uint32_t d_tmem, uint32_t w_tmem, uint32_t b_addr, bool first_step) {
      const uint32_t b_lo = sw128_desc_lo(b_addr, C::STR_PANEL);
#pragma unroll
      for (int ks = 0; ks < BS / 16; ++ks)
        umma_f16_ts_parts(d_tmem, w_tmem + (ks >> 1) * 32 + (ks & 1) * 8, b_lo + ks * (2048 >> 4), SW128_DESC_HI, C::IDESC_TS,
                          (first_step && ks == 0) ? 0u : 1u);
    };
    auto tile0 = [&](int j) { return ring_addr + (j % C::NS) * 2 * C::STR_BYTES; };
    auto score_s = [&](int j) -> bool {                      // waits for step j's tiles, then S (or S^T) of step j
      if (!wait_all(&ctl->full[j % C::NS], (j / C::NS) & 1u)) return false;
      tc_fence_after();
      if (elect_one()) {
        issue_scores(tmem_base + s_col(j), a0_lo, tile0(j));
        umma_commit(&ctl->s_full[sbuf(j)]);
      }
      __syncwarp();
      return true;
    };
    auto score_dp = [&](int j) {                             // dP (or dP^T) of step j, whose tiles score_s(j) has waited for
      if (elect_one()) {
        issue_scores(tmem_base + C::DP_COL, a1_lo, tile0(j) + C::STR_BYTES);
        umma_commit(&ctl->dp_full);
      }
      __syncwarp();
    };
    bool ok = wait_all(&ctl->res_full, 0) && score_s(0);
    if (ok) {
      score_dp(0);
      if (DB && nsteps > 1) ok = score_s(1);
    }
    for (int j = 0; j < nsteps && ok; ++j) {
      const bool has_next = j + 1 < nsteps;
      const uint32_t t0 = tile0(j), t1 = t0 + C::STR_BYTES;
      // phase 1 is over: S has been read (MODE 1: P^T stands in its place)
      if (!wait_all(&ctl->p_done[sbuf(j)], sphase(j))) { ok = false; break; }
      tc_fence_after();
      if (MODE == 1) {
        if (elect_one()) issue_product(tmem_base + C::ACC0_COL, tmem_base + s_col(j), t1, j == 0);     // dV += P^T dO
        __syncwarp();
      }
      if (!DB && has_next && !score_s(j + 1)) { ok = false; break; }     // after the dV product: may overwrite P^T
      // phase 2 is over: dS stands in place of dP
      if (!wait_all(&ctl->ds_done, j & 1u)) { ok = false; break; }
      tc_fence_after();
      if (elect_one()) {
        issue_product(tmem_base + (MODE == 0 ? C::ACC0_COL : C::ACC1_COL), tmem_base + C::DP_COL, t0, j == 0);   // dQ += dS K / dK += dS^T Q
        umma_commit(&ctl->empty[j % C::NS]);
      }
      __syncwarp();
      if (has_next) score_dp(j + 1);                         // after that product: may overwrite dS
      if (DB && j + 2 < nsteps && !score_s(j + 2)) { ok = false; break; }   // into the buffer phase 1 of step j has left
    }
    if (ok && elect_one()) umma_commit(&ctl->acc_full);
  } else {
    const int quarter = warp & 3, group = (warp - 2) >> 2;
    const int r = quarter * 32 + lane, row = row0 + r;
    const int wrow0 = row0 + quarter * 32;                    // this warp's first row
    const uint32_t lane_sel = uint32_t(quarter * 32) << 16;
    const float kappa = 1.0f / (p.scale * p.scale);
    float2 a_row = make_float2(0.f, 0.f), delta_row = make_float2(0.f, 0.f);
    if (MODE == 0 && row < p.Tq) {
      const float a = p.stat[bh * p.Tq + row], d = -p.delta[bh * p.Tq + row];
      a_row = make_float2(a, a);
      delta_row = make_float2(d, d);
    }
    const uint32_t dp_t = tmem_base + lane_sel + C::DP_COL + group * 32;
    // one instance per form of the weight, so that nothing is decided per score block but what the mask needs
    auto steps = [&](auto form, auto power) -> bool {
      constexpr bool SHIFTED = decltype(form)::value;
      constexpr int LOG2N = decltype(power)::value;
      int slot = 0;
      uint32_t ring = 0;                                      // ring position and phase
      for (int j = 0; j < nsteps; ++j) {
        const int col0 = first + j * BS + group * 32;         // first streamed row of this thread's 32 columns
        const float* vec = reinterpret_cast<const float*>(smem + C::VEC_OFF) + slot * 2 * BS + group * 32;
        float2 slope[16];
        // ---- phase 1: scores -> weights
        const uint32_t s_t = tmem_base + lane_sel + s_col(j) + group * 32;
        if (MODE == 1 && !bw.wait(&ctl->vec_full[slot], ring)) return false;
        if (++slot == C::NS) { slot = 0; ring ^= 1u; }
        if (!bw.wait(&ctl->s_full[sbuf(j)], sphase(j))) return false;
        tc_fence_after();
        // the causal mask removes none, some or all of a 32 x 32 block (warp-uniform)
        const int ahead = (MODE == 0) ? col0 - wrow0 : wrow0 - col0;      // > -32: some, >= 32: all
        if (ahead <= -32) {
          phase1<MODE, SHIFTED, LOG2N, false>(s_t, slope, vec, a_row, p.scale, kappa, p.log2n, row, col0);
        } else if (ahead < 32) {
          phase1<MODE, SHIFTED, LOG2N, true>(s_t, slope, vec, a_row, p.scale, kappa, p.log2n, row, col0);
        } else {
          uint32_t zero[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) { slope[i] = make_float2(0.f, 0.f); zero[i] = 0u; }
          if (MODE == 1) tmem_st_32x16(s_t, zero);
        }
        if (MODE == 1) tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->p_done[sbuf(j)]);
        // ---- phase 2: dP -> dS = slope (dP - delta)
        if (!bw.wait(&ctl->dp_full, j & 1u)) return false;
        tc_fence_after();
        uint32_t d0[16], d1[16];
        tmem_ld_32x16(dp_t, d0);
        tmem_ld_wait_for16(d0);
        tmem_ld_32x16(dp_t + 16, d1);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float2 nd[8];
          if (MODE == 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 v = *reinterpret_cast<const float4*>(vec + BS + c * 16 + 4 * i);
              nd[2 * i] = make_float2(v.x, v.y);
              nd[2 * i + 1] = make_float2(v.z, v.w);
            }
          }
          if (c == 1) tmem_ld_wait_for16(d1);
          const uint32_t* dp = c == 0 ? d0 : d1;
          uint32_t ds[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float2 d = make_float2(__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1]));
            const float2 v = __fmul2_rn(slope[8 * c + i], __fadd2_rn(d, MODE == 1 ? nd[i] : delta_row));
            ds[i] = pack_bf16(v.x, v.y);
          }
          tmem_st_32x8(dp_t + c * 8, ds);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->ds_done);
      }
      return true;
    };
    using std::integral_constant;
    bool ok;
    if (shifted) ok = steps(integral_constant<bool, true>{}, integral_constant<int, 0>{});
    else if (p.log2n == 4) ok = steps(integral_constant<bool, false>{}, integral_constant<int, 4>{});
    else ok = steps(integral_constant<bool, false>{}, integral_constant<int, 0>{});
    if (ok && bw.wait(&ctl->acc_full, 0)) {
      tc_fence_after();
      constexpr int CPT = D / C::NG;                           // accumulator columns per thread
      __nv_bfloat16* out0 = ((MODE == 0) ? p.dq + b * p.qs.b + h * p.qs.h + int64_t(row) * p.qs.t
                                         : p.dv + b * p.vs.b + h * p.vs.h + int64_t(row) * p.vs.t) + group * CPT;
      __nv_bfloat16* out1 = (MODE == 1) ? p.dk + b * p.ks.b + h * p.ks.h + int64_t(row) * p.ks.t + group * CPT : nullptr;
      // the constant factors the element-wise stage left out (see weights16); dV carries none
      const float n_fac = shifted ? p.n_scale : p.n_f;
#pragma unroll 1
      for (int which = 0; which < (MODE == 0 ? 1 : 2); ++which) {
        const uint32_t acc_t = tmem_base + lane_sel + (which == 0 ? C::ACC0_COL : C::ACC1_COL) + group * CPT;
        __nv_bfloat16* dst = which == 0 ? out0 : out1;
        const float fac = (MODE == 0 || which == 1) ? n_fac : 1.0f;
#pragma unroll 1
        for (int c = 0; c < CPT / 16; ++c) {
          uint32_t a[16];
          tmem_ld_32x16(acc_t + c * 16, a);
          tmem_ld_wait_for16(a);
          if (row < p.Tq) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
              *reinterpret_cast<uint4*>(dst + c * 16 + i * 8) =
                  make_uint4(pack_bf16(__uint_as_float(a[8 * i]) * fac, __uint_as_float(a[8 * i + 1]) * fac),
                             pack_bf16(__uint_as_float(a[8 * i + 2]) * fac, __uint_as_float(a[8 * i + 3]) * fac),
                             pack_bf16(__uint_as_float(a[8 * i + 4]) * fac, __uint_as_float(a[8 * i + 5]) * fac),
                             pack_bf16(__uint_as_float(a[8 * i + 6]) * fac, __uint_as_float(a[8 * i + 7]) * fac));
          }
        }
      }
    }
    // dsink: -sum_i delta_i p_sink,i n / (c sqrt(1 + (b/c)^2)), one atomic per warp of the first column group
    if (MODE == 0 && p.sink != nullptr && p.dsink != nullptr && group == 0) {
      const float bs = p.sink[h] * p.inv_c;
      const float ps = shifted ? pow2n_rt(rho_stable(bs) * a_row.x, p.log2n) : pow2n_rt(rho_stable(bs), p.log2n) * a_row.x;
      float part = delta_row.x * ps * p.n_f * p.inv_c * rsqrtf(fmaf(bs, bs, 1.0f));
      part = warp_sum(part);
      if (lane == 0) atomicAdd(p.dsink + h, part);
    }
  }
}

template <int D, int BS, int CTAS>
__global__ void __launch_bounds__(Cfg<D, BS, CTAS>::NTHREADS, CTAS)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ AttnBwdParams p) {
  using C = Cfg<D, BS, CTAS>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Control* ctl = reinterpret_cast<Control*>(smem + C::CTL_OFF);
  const int warp = threadIdx.x >> 5;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_do);
    mbar_init(&ctl->res_full, 1);
    for (int i = 0; i < C::NS; ++i) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], 1); mbar_init(&ctl->vec_full[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&ctl->s_full[i], 1); mbar_init(&ctl->p_done[i], C::EW_WARPS); }
    mbar_init(&ctl->dp_full, 1);
    mbar_init(&ctl->ds_done, C::EW_WARPS);
    mbar_init(&ctl->acc_full, 1);
    ctl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_wait();                               // delta (and a zeroed dsink) come from the kernel ahead in the stream

  // heavy blocks first over all heads: early key blocks are seen by many queries, late query blocks see many
  // keys; the dK/dV blocks, the dearer kind, before the dQ blocks
  const int nt = int(gridDim.z) / 2, z = int(blockIdx.z);
  if (z < nt) bwd_block<C, D, BS, 1>(smem, ctl, &tm_q, &tm_k, &tm_v, &tm_do, p, z);
  else bwd_block<C, D, BS, 0>(smem, ctl, &tm_q, &tm_k, &tm_v, &tm_do, p, 2 * nt - 1 - z);

  tc_fence_before();
  __syncthreads();
  if (ctl->abort_flag != 0) {
    if (threadIdx.x == 0) {
      if (p.status != nullptr) atomicExch(p.status, ALG_DEV_TIMEOUT);
      const uint64_t t0 = global_timer_ns();                 // let issued loads land before shared memory is released
      while (global_timer_ns() - t0 < 200000ull) { }
    }
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(ctl->tmem_base, C::TMEM_COLS);
  }
}

// delta_i = dO_i . o_i, one row per LPR lanes, ROWS of them in flight per lane; the first block also zeroes dsink.
template <int D>
__global__ void __launch_bounds__(256) attn_delta_kernel(const AttnBwdParams p) {
  constexpr int LPR = D / 8, RPW = 32 / LPR, ROWS = 4;
  griddep_wait();
  if (blockIdx.x == 0 && p.dsink != nullptr)
    for (int i = threadIdx.x; i < p.H; i += blockDim.x) p.dsink[i] = 0.f;
  const int lane = threadIdx.x & 31, lir = lane % LPR, sub = lane / LPR;
  const int64_t rows = int64_t(p.B) * p.H * p.Tq;
  const int64_t warp_global = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps_total = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r0 = warp_global * (RPW * ROWS); r0 < rows; r0 += warps_total * (RPW * ROWS)) {
    uint4 a[ROWS], c[ROWS];
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const int64_t row = min(r0 + u * RPW + sub, rows - 1);
      const int t = int(row % p.Tq);
      const int64_t bh = row / p.Tq;
      const int h = int(bh % p.H);
      const int64_t b = bh / p.H;
      a[u] = __ldg(reinterpret_cast<const uint4*>(p.o + b * p.os.b + h * p.os.h + int64_t(t) * p.os.t + lir * 8));
      c[u] = __ldg(reinterpret_cast<const uint4*>(p.d_o + b * p.gs.b + h * p.gs.h + int64_t(t) * p.gs.t + lir * 8));
    }
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a[u]);
      const __nv_bfloat162* c2 = reinterpret_cast<const __nv_bfloat162*>(&c[u]);
      float d = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 fa = __bfloat1622float2(a2[i]), fc = __bfloat1622float2(c2[i]);
        d = fmaf(fa.x, fc.x, d);
        d = fmaf(fa.y, fc.y, d);
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      const int64_t row = r0 + u * RPW + sub;
      if (lir == 0 && row < rows) p.delta[row] = d;
    }
  }
}

int make_map(CUtensorMap* tm, const void* base, const Strides3& s, int B, int H, int T, int D, int box_rows) {
  const uint64_t dims[4] = {uint64_t(D), uint64_t(T), uint64_t(H), uint64_t(B)};
  const uint64_t strides[3] = {uint64_t(s.t), uint64_t(s.h), uint64_t(s.b)};
  const uint32_t box[4] = {64, uint32_t(box_rows), 1, 1};
  return make_tmap_bf16(tm, base, 4, dims, strides, box, true);
}

template <int D, int BS, int CTAS>
int launch_d(const AttnBwdParams& p, cudaStream_t stream) {
  using C = Cfg<D, BS, CTAS>;
  static_assert(CTAS * smem_bytes<C>() <= 232448 - CTAS * 1024, "shared memory budget of an SM");
  static_assert(C::ACC1_COL + D <= C::TMEM_COLS, "tensor-memory budget of a CTA");
  CUtensorMap tq, tk, tv, tdo;
  if (int rc = make_map(&tq, p.q, p.qs, p.B, p.H, p.Tq, D, BS)) return rc;
  if (int rc = make_map(&tk, p.k, p.ks, p.B, p.H, p.Tk, D, BS)) return rc;
  if (int rc = make_map(&tv, p.v, p.vs, p.B, p.H, p.Tk, D, BS)) return rc;
  if (int rc = make_map(&tdo, p.d_o, p.gs, p.B, p.H, p.Tq, D, BS)) return rc;
  auto kern = attn_bwd_tc_kernel<D, BS, CTAS>;
  static PerDeviceOnce configured;
  int sms = 0;
  if (int rc = configured.run([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes<C>())); }, &sms))
    return rc;
  const int64_t rows = int64_t(p.B) * p.H * p.Tq;
  int64_t blocks = (rows / (4 * (32 / (D / 8))) + 7) / 8;
  if (blocks > sms * 6) blocks = sms * 6;
  if (blocks < 1) blocks = 1;
  ALG_CUDA_TRY(launch_dependent(attn_delta_kernel<D>, dim3(unsigned(blocks)), dim3(256), 0, stream, p));
  const dim3 grid(p.H, p.B, 2 * ((p.Tq + BT - 1) / BT));
  ALG_CUDA_TRY(launch_dependent(kern, grid, dim3(C::NTHREADS), smem_bytes<C>(), stream, tq, tk, tv, tdo, p));
  count_launch(2);
  return ALG_OK;
}

}  // namespace

bool attn_bwd_tcgen05_supports(const AttnBwdParams& p) {
  const bool strides_fit = p.qs.t > 0 && p.ks.t > 0 && p.vs.t > 0 && p.os.t > 0 && p.gs.t > 0 && p.qs.h >= 0 && p.qs.b >= 0 &&
                           p.ks.h >= 0 && p.ks.b >= 0 && p.vs.h >= 0 && p.vs.b >= 0 && p.gs.h >= 0 && p.gs.b >= 0;
  const bool rows_fit = p.B <= 65535 && 2 * ((p.Tq + BT - 1) / BT) <= 65535;
  return p.causal && p.Tq == p.Tk && (p.D == 64 || p.D == 128) && strides_fit && rows_fit &&
         (p.B == 1 || (p.qs.b > 0 && p.gs.b > 0)) && (p.H == 1 || (p.qs.h > 0 && p.gs.h > 0));
}

int launch_attn_bwd_tcgen05(const AttnBwdParams& p, cudaStream_t stream) {
  return p.D == 64 ? launch_d<64, 64, 2>(p, stream) : launch_d<128, 128, 1>(p, stream);
}

}  // namespace alg
