// All blocks of a prefill as one call: per block the five kernels of the fused form (QKV projection,
// attention, out-projection, gate|up projection, down-projection), then the final norm
// (src/algebraic/model.py:162-208 of the reference).  Host code only - it derives every launch from the
// entry points of the single kernels.  A short prompt is bound by what the host spends between launches:
// issued one operator at a time from the interpreter a block cost about 160 us of host time for about 45 us
// of GPU time (613 tokens of the 125M model); issued here it costs about 20.
#include <stdint.h>

#include "common.cuh"
#include "launchers.h"

using namespace alg;

namespace {

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct Scratch {
  size_t qkv, attn, ff, ss_in, ss_o, ss_d, attn_ws, attn_ws_bytes, total;
  int slots;
};

alg_attn_args attn_args(const alg_prefill_blocks_args* a, unsigned char* base, const Scratch& s) {
  const int64_t hd = int64_t(a->H) * a->D;
  alg_attn_args t{};
  unsigned char* qkv = base + s.qkv;
  t.q = qkv; t.k = qkv + hd * 2; t.v = qkv + 2 * hd * 2;
  t.o = base + s.attn;
  t.B = a->B; t.H = a->H; t.Tq = a->T; t.Tk = a->T; t.D = a->D;
  t.n = a->attn_n; t.c = a->attn_c; t.eps = a->eps;
  t.causal = 1; t.variant = ALG_VARIANT_GUARD; t.dtype = ALG_BF16; t.impl = a->impl;
  int64_t* in[3] = {t.q_stride, t.k_stride, t.v_stride};
  for (int64_t* st : in) { st[0] = a->T * 3 * hd; st[1] = a->D; st[2] = 3 * hd; }
  t.o_stride[0] = a->T * hd; t.o_stride[1] = a->D; t.o_stride[2] = hd;
  return t;
}

Scratch layout(const alg_prefill_blocks_args* a) {
  const size_t M = size_t(a->B) * a->T, hd = size_t(a->H) * a->D;
  Scratch s{};
  size_t at = 0;
  auto take = [&](size_t bytes) { const size_t here = at; at += align256(bytes); return here; };
  s.slots = alg_resid_proj_ss_slots(int(M), a->d);
  s.qkv = take(M * 3 * hd * 2);
  s.attn = take(M * hd * 2);
  s.ff = take(M * a->f * 2);
  s.ss_in = take(M * sizeof(float));
  s.ss_o = take(M * s.slots * sizeof(float));
  s.ss_d = take(M * s.slots * sizeof(float));
  const alg_attn_args t = attn_args(a, nullptr, s);
  s.attn_ws_bytes = alg_attn_workspace_bytes(&t);
  s.attn_ws = take(s.attn_ws_bytes);
  s.total = at;
  return s;
}

bool extents_ok(const alg_prefill_blocks_args* a) {
  return a != nullptr && a->L >= 0 && a->B >= 0 && a->T >= 1 && a->H >= 1 && (a->D == 64 || a->D == 128) && a->d >= 64 &&
         a->d == a->H * a->D && a->f >= 128 && a->f % 128 == 0 && int64_t(a->B) * a->T < (int64_t(1) << 31);
}

}  // namespace

extern "C" {

size_t alg_prefill_blocks_workspace_bytes(const alg_prefill_blocks_args* a) {
  return extents_ok(a) && a->B > 0 ? layout(a).total : 0;
}

int alg_prefill_blocks(const alg_prefill_blocks_args* a, void* stream) {
  if (!extents_ok(a)) {
    set_error("prefill_blocks: head_dim 64 or 128, d = H D, f a multiple of 128, T at least 1");
    return ALG_ERR_INVALID;
  }
  if (a->B == 0) return ALG_OK;
  if (a->x == nullptr || a->out == nullptr || a->w_qkv == nullptr || a->w_o == nullptr || a->w_gu == nullptr ||
      a->w_d == nullptr || a->cos == nullptr || a->sin == nullptr || a->guard == nullptr) {
    set_error("prefill_blocks: null argument");
    return ALG_ERR_INVALID;
  }
  const Scratch s = layout(a);
  if (a->workspace == nullptr || a->workspace_bytes < s.total || (reinterpret_cast<uintptr_t>(a->workspace) & 255) != 0) {
    set_error("prefill_blocks: workspace of %zu bytes (256-byte aligned) required, got %zu", s.total, a->workspace_bytes);
    return ALG_ERR_WORKSPACE;
  }
  unsigned char* base = static_cast<unsigned char*>(a->workspace);
  const int M = a->B * a->T, d = a->d, f = a->f, hd = a->H * a->D;
  auto rows = [](const void* p, int64_t n) { return static_cast<const unsigned char*>(p) + n * 2; };   // n bf16 elements on
  float* ss_in = reinterpret_cast<float*>(base + s.ss_in);
  float* ss_o = reinterpret_cast<float*>(base + s.ss_o);
  float* ss_d = reinterpret_cast<float*>(base + s.ss_d);
  if (int rc = alg_row_sumsq(a->x, M, d, d, ss_in, stream)) return rc;

  alg_qkv_proj_args qkv{};
  qkv.x = a->x; qkv.qkv = base + s.qkv; qkv.cos = a->cos; qkv.sin = a->sin; qkv.eps = a->eps; qkv.M = M; qkv.d = d;
  qkv.H = a->H; qkv.D = a->D; qkv.T = a->T; qkv.ld_x = d; qkv.attn_c = a->attn_c; qkv.status = a->status;
  qkv.row_ss = ss_in; qkv.ss_slots = 1; qkv.row_eps = a->eps; qkv.guard_is_zero = 1;
  alg_attn_args att = attn_args(a, base, s);
  att.workspace = base + s.attn_ws; att.workspace_bytes = s.attn_ws_bytes; att.status = a->status;
  alg_resid_proj_args out{};
  out.x = base + s.attn; out.resid = a->x; out.out = a->x; out.ss_out = ss_o; out.M = M; out.K = hd; out.N = d;
  out.ld_x = hd; out.ld_resid = d; out.ld_out = d; out.status = a->status;
  alg_glu_proj_args glu{};
  glu.x = a->x; glu.out = base + s.ff; glu.M = M; glu.d = d; glu.f = f; glu.ld_x = d; glu.ld_out = f; glu.beta = a->alu_beta;
  glu.status = a->status; glu.row_ss = ss_o; glu.ss_slots = s.slots; glu.row_eps = a->eps;
  alg_resid_proj_args down = out;
  down.x = base + s.ff; down.ss_out = ss_d; down.K = f; down.ld_x = f;
  for (int64_t l = 0; l < a->L; ++l) {
    qkv.w = rows(a->w_qkv, l * 3 * hd * d);
    qkv.q_gain = a->q_gain != nullptr ? a->q_gain + l * a->D : nullptr;
    qkv.k_gain = a->k_gain != nullptr ? a->k_gain + l * a->D : nullptr;
    qkv.guard = static_cast<unsigned char*>(a->guard) + l * 16;
    if (int rc = alg_qkv_proj_fwd(&qkv, stream)) return rc;
    att.guard_words = qkv.guard;
    att.sink = a->sink != nullptr ? a->sink + l * a->H : nullptr;
    if (int rc = alg_attn_fwd(&att, stream)) return rc;
    out.w = rows(a->w_o, l * d * hd);
    if (int rc = alg_resid_proj_fwd(&out, stream)) return rc;
    glu.w = rows(a->w_gu, l * 2 * f * d);
    if (int rc = alg_glu_proj_fwd(&glu, stream)) return rc;
    down.w = rows(a->w_d, l * d * f);
    if (int rc = alg_resid_proj_fwd(&down, stream)) return rc;
    qkv.row_ss = ss_d; qkv.ss_slots = s.slots;
  }
  return alg_rms_norm_fwd(a->x, a->final_gain, a->out, M, d, a->eps, stream);
}

}  // extern "C"
