// C-ABI layer of libkda_b200.so: argument checks, workspace arithmetic, stage launches.
// Interface and the reference entry points it stands in for: include/kda_b200.h.
#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda.h>

#include "../../include/kda_b200.h"
#include "kda_common.cuh"
#include "kda_kernels.h"

static_assert(sizeof(KdaFwdArgs) == 312 && offsetof(KdaFwdArgs, chunk_table) == 288 && offsetof(KdaFwdArgs, Hq) == 308,
              "KdaFwdArgs layout is part of the ABI (bindings mirror it field by field)");

namespace {

thread_local char g_err[512] = "";
thread_local int g_launches = 0;

int fail(int code, const char* fmt, const char* a = "", long long x = 0, long long y = 0) {
  snprintf(g_err, sizeof(g_err), fmt, a, x, y);
  return code;
}

int check_common(const KdaFwdArgs* a) {
  if (a == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: args is NULL%s", "");
  if (a->B <= 0 || a->T <= 0 || a->H <= 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: B, T, H must be positive%s (T=%lld, H=%lld)", "", a->T, a->H);
  if (a->workspace == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: workspace is NULL%s", "");
  if (reinterpret_cast<uintptr_t>(a->workspace) % 256 != 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: workspace must be 256-byte aligned%s", "");
  if (a->Hq < 0 || (a->Hq > 0 && a->H % a->Hq != 0))
    return fail(KDA_ERR_INVALID_ARG, "kda: H%s (%lld) must be a multiple of Hq (%lld)", "", a->H, a->Hq);
  if (a->n_seqs < 0) return fail(KDA_ERR_INVALID_ARG, "kda: n_seqs must not be negative%s", "");
  if (a->n_seqs > 0) {
    if (a->B != 1) return fail(KDA_ERR_INVALID_ARG, "kda: packed sequences need B = 1%s (got %lld)", "", a->B);
    if (a->chunk_table == nullptr || a->seq_table == nullptr || a->n_chunks <= 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: packed sequences need chunk_table, seq_table and n_chunks%s", "");
    if (reinterpret_cast<uintptr_t>(a->chunk_table) % 16 != 0 || reinterpret_cast<uintptr_t>(a->seq_table) % 16 != 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: chunk_table and seq_table must be 16-byte aligned%s", "");
    if (a->g_out != nullptr || a->ainv_out != nullptr)
      return fail(KDA_ERR_INVALID_ARG, "kda: the debug outputs are not available with packed sequences%s", "");
  }
  return KDA_OK;
}

bool row_aligned(const void* p, const int64_t s[3], int elem_bytes) {
  if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
  for (int i = 0; i < 3; ++i)
    if ((s[i] * elem_bytes) % 16 != 0) return false;
  return true;
}

// The fp32 parameters that are read one float at a time: views of larger buffers, so no more than their own alignment is asked for.
bool params_aligned(const KdaFwdArgs* a, bool gate) {
  uintptr_t at = reinterpret_cast<uintptr_t>(a->beta);
  if (gate) at |= reinterpret_cast<uintptr_t>(a->A_log) | reinterpret_cast<uintptr_t>(a->dt_bias);
  return at % sizeof(float) == 0;
}

int check_k1(const KdaFwdArgs* a) {
  if (int rc = check_common(a)) return rc;
  if (!a->q || !a->k || !a->v || !a->g || !a->beta)
    return fail(KDA_ERR_INVALID_ARG, "kda: q, k, v, g and beta are required%s", "");
  if (a->g_dtype != KDA_G_FP32 && a->g_dtype != KDA_G_BF16)
    return fail(KDA_ERR_INVALID_ARG, "kda: g_dtype must be KDA_G_FP32 or KDA_G_BF16%s (got %lld)", "", a->g_dtype);
  if ((a->flags & KDA_FLAG_GATE_IN_KERNEL) && a->A_log == nullptr)
    return fail(KDA_ERR_INVALID_ARG, "kda: the in-kernel gate requires A_log%s", "");
  if ((a->flags & KDA_FLAG_GATE_IN_KERNEL) && !(a->lower_bound > -11.0f && a->lower_bound < 0.0f))
    return fail(KDA_ERR_INVALID_ARG, "kda: lower_bound must be in (-11, 0)%s", "");
  if (!row_aligned(a->q, a->q_stride, 2) || !row_aligned(a->k, a->k_stride, 2) || !row_aligned(a->v, a->v_stride, 2) ||
      !row_aligned(a->g, a->g_stride, a->g_dtype == KDA_G_BF16 ? 2 : 4))
    return fail(KDA_ERR_INVALID_ARG, "kda: q/k/v/g rows must start on 16-byte boundaries%s", "");
  if (!params_aligned(a, (a->flags & KDA_FLAG_GATE_IN_KERNEL) != 0))
    return fail(KDA_ERR_INVALID_ARG, "kda: beta, A_log and dt_bias must be 4-byte aligned%s", "");
  if (reinterpret_cast<uintptr_t>(a->g_out) % 8 != 0 || reinterpret_cast<uintptr_t>(a->ainv_out) % 4 != 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: g_out must be 8-byte and ainv_out 4-byte aligned%s", "");
  // an expanded view (stride 0 on a dimension larger than 1) cannot be described to the TMA unit
  const int hq = a->Hq > 0 ? a->Hq : a->H;
  const struct { const int64_t* s; int heads; const char* name; } views[4] = {
      {a->q_stride, hq, "q"}, {a->k_stride, hq, "k"}, {a->v_stride, a->H, "v"}, {a->g_stride, a->H, "g"}};
  for (const auto& v : views) {
    const int sizes[3] = {a->B, a->T, v.heads};
    for (int i = 0; i < 3; ++i)
      if (sizes[i] > 1 && v.s[i] <= 0)
        return fail(KDA_ERR_INVALID_ARG, "kda: %s has a zero or negative stride on a dimension of size %lld (expanded views are not supported)",
                    v.name, sizes[i]);
  }
  return KDA_OK;
}

int check_k2(const KdaFwdArgs* a, bool state_only) {
  if (int rc = check_common(a)) return rc;
  if (!state_only && a->o == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: o is NULL%s", "");
  if (!state_only && !row_aligned(a->o, a->o_stride, 2))
    return fail(KDA_ERR_INVALID_ARG, "kda: o rows must start on 16-byte boundaries%s", "");
  for (const void* ptr : {static_cast<const void*>(a->h0), static_cast<const void*>(a->ht)})
    if (ptr != nullptr && reinterpret_cast<uintptr_t>(ptr) % 16 != 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: h0 and ht must be 16-byte aligned%s", "");
  const int vs = a->k2_vsplit, var = a->k2_variant;
  if (var < 0 || var > 5 || var == 2)
    return fail(KDA_ERR_INVALID_ARG, "kda: k2_variant must be 0, 1, 3, 4 or 5%s (got %lld)", "", var);
  if (var == 4 && state_only)
    return fail(KDA_ERR_INVALID_ARG, "kda: the tensor-memory K2 (k2_variant 4) has no state-only form%s", "");
  if (var == 4) return KDA_OK;
  if (vs != 0 && vs != 2 && vs != 4 && vs != 8 && vs != 16)
    return fail(KDA_ERR_INVALID_ARG, "kda: k2_vsplit must be 0, 2, 4, 8 or 16%s (got %lld)", "", vs);
  if (vs != 0 && var != 0 && ((var == 1 || var == 5) ? (vs < 4) : (vs > 8)))
    return fail(KDA_ERR_INVALID_ARG, "kda: k2_vsplit %lld%s does not go with k2_variant %lld", "", vs, var);
  return KDA_OK;
}

// How one head's 128x128 state is spread over warps.  The recurrence is a serial chain per head;
// a warp alone on an SM sub-partition cannot overlap its own MMA issue with its other
// instructions, so a step costs about 8 cycles per MMA plus its non-MMA instructions, and every
// warp re-reads the shared operand tiles from shared memory.  Measured on B200, kda_fwd in us, chains x chunks:
//   up to SMs/4 chains the 8-rows-per-warp "n8" form (two warps per SM while chains x 8 CTAs fit the SMs, else four), from
//     there on the 16-rows-per-warp "m16" form with four warps per CTA, which reads half the shared-memory bytes per MMA:
//     n8 / m16  37 x 8 14.4 / 16.3, 37 x 128 115 / 124, 37 x 512 418 / 465;  38 x 8 19.6 / 16.5, 38 x 128 177 / 137,
//     38 x 512 669 / 521.
//   more chains than SMs: the tensor-memory form (one CTA per chain, two per SM, tcgen05) from four chunks per chain on; its
//     set-up (TMEM allocation, the state in and out through registers) costs about as much as two steps:
//     m16 / tc  160 x 2 17.6 / 18.8, 160 x 4 24.7 / 24.7, 160 x 8 38.9 / 37.0;  296 x 2 22.6 / 22.6, 296 x 4 34.9 / 32.8;
//     400 x 4 49.6 / 52.2, 400 x 6 64.4 / 64.1;  592 x 4 68.1 / 64.1.
//   between half as many chains as SMs and as many (where m16 needs two CTAs per chain and so more than one per SM) from 32
//     chunks on.  K2 alone tc is ahead from 12 chunks, but the forward follows late and less the more chains there are:
//     m16 / tc  80 x 8 24.7 / 24.7, 80 x 16 39.4 / 37.8, 80 x 24 55.8 / 52.4, 80 x 32 71.1 / 63.1;  112 x 16 45.6 / 44.3,
//     112 x 24 63.9 / 61.3, 112 x 32 80.5 / 78.6;  148 x 16 51.7 / 50.4, 148 x 24 71.9 / 73.8, 148 x 32 90.8 / 91.3,
//     148 x 48 129.7 / 126.2.  The line is safe for all of them; below it 75 to 130 chains of 16 to 31 chunks give up 2 to 6 %.
//   up to half as many chains as SMs m16 wins at every length (K2 alone, 74 chains x 256 chunks 175 / 229).
// The tensor-memory form has no state-only variant.
void pick_split(const KdaFwdArgs* a, bool state_only, int* vsplit, int* variant, int sms = 0, int chain_mult = 1) {
  if (sms <= 0) {   // the current device's SM count
    int dev = 0;
    sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const long long bh = static_cast<long long>(a->n_seqs > 0 ? a->n_seqs : a->B) * a->H * chain_mult;
  // chunks per chain (the mean, for packed sequences)
  const long long steps = a->n_seqs > 0 ? a->n_chunks / a->n_seqs : (a->T + kda::BT - 1) / kda::BT;
  int var = a->k2_variant;
  int vs = a->k2_vsplit;
  if (var == 0) {
    if (vs == 16) var = 1;
    else if (vs == 2) var = 3;
    else if (!state_only && vs == 0 && ((bh > sms && steps >= 4) || (bh * 2 > sms && steps >= 32))) var = 4;
    else var = (bh * 4 <= sms) ? 1 : 3;
  }
  if (vs == 0) {
    if (var == 1 || var == 5) vs = (bh * 16 <= sms) ? 16 : (bh * 8 <= sms) ? 8 : 4;
    else vs = (bh * 4 <= sms) ? 4 : 2;
  }
  if ((var == 1 || var == 5) && vs < 4) vs = 4;
  if (var != 1 && var != 5 && vs > 8) vs = 8;
  *vsplit = vs;
  *variant = var;
}

int* status_ptr(const KdaFwdArgs* a) { return static_cast<int*>(a->workspace); }
uint8_t* rec_ptr(const KdaFwdArgs* a) { return static_cast<uint8_t*>(a->workspace) + kda::WS_HEADER_BYTES; }

int device_sms() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Address range of a strided [B, T, heads, row] tensor (strides in elements, none negative).
struct Span { uintptr_t lo, hi; };
Span span_of(const void* ptr, const int64_t s[3], const KdaFwdArgs* a, int heads, int row, int elem_bytes) {
  const uintptr_t lo = reinterpret_cast<uintptr_t>(ptr);
  const int64_t last = (a->B - 1) * s[0] + (a->T - 1) * s[1] + (heads - 1) * s[2] + row;
  return {lo, lo + static_cast<uintptr_t>(last) * elem_bytes};
}

// A forward whose K2 runs beside its K1, on part of the chip.
//
// K1 walks the chunks of all chains in time order and counts the finished items of every window of chunks; K2's producer
// warps wait for the window of the record they load next.  K2 waits for K1 only, and starts when every K1 CTA
// is already running.  On k2_sms of the SMs only k2_sm_ctas of K1's CTAs stay (k1_stays), and K2's CTAs fit nowhere else.
// Which of it pays, measured on B200 as the whole forward in us, K2 after K1 against beside it unless said otherwise:
//   8-row form with one or two consumer warps per CTA (chains x 8 <= SMs), two K1 CTAs on every SM: B1 T131072 H16 3,705 / 3,438,
//     T32768 H16 935 / 872, T8192 H16 241 / 227, H12 225 / 214, H8 204.7 / 201.2, B2 T4096 H8 123.8 / 120.4; near the line of 16
//     items per SM it costs up to 1 %: T5000 H8 127.4 / 128.1, T2600 H16 80.9 / 81.5, T2400 H18 77.3 / 78.3.  With four on the SMs that K2 leaves free T131072 H16 3,727
//     against 3,704, B2 T4096 H8 129.6 / 129.0; with one on K2's SMs K1 is the longer part (T32768 H16 1,329).
//   Up to SMs / 6 chains: the 8-row form with four consumer warps on SMs of its own (4 per chain): T8192 H23 326 / 283, H24
//     330 / 309, T4096 H24 172 / 164, T2500 H23 107 / 102. Beyond, K1 has too few SMs left: T4096 H25 173 / 181.
//   From there to 42 of 148 chains: the 16-row form, whose bits are the same, on SMs of its own (2 per chain).  Where the 8-row
//     form is the choice, at chunk counts that make up for the longer step (0.61 us against 0.45 and K1's time): T8192 H25 335 /
//     322, H32 362 / 326, H37 380 / 346; T4096 H25 173 / 171, H28 178 / 172, H32 186 / 174; T2500 H25 110 / 113, H26 110 / 113, H28 115 /
//     113, H32 120 / 114; T1600 H28 77 / 79, H30 78 / 80, H32 80.6 / 80.1, H37 83 / 82.  Where the 16-row form is the choice anyway:
//     T8192 H38 461 / 362, H42 477 / 435, H44 483 / 477; T1200 H38 75 / 68, H42 78.6 / 78.3, H43 79.4 / 80.5, H44 79 / 84.  With a K1
//     CTA beside K2's: T8192 H32 403 against 363.
//   Tensor-memory form with one CTA per SM and two K1 CTAs there (a K1 of 112 registers: see there), four on the other SMs:
//     T1024 H75 108 / 101, H96 121 / 109, H123 136 / 127, H136 143 / 139, H148 149 / 152; T8192 H75 754 / 636, H96 834 / 686,
//     H123 942 / 867, H136 998 / 969, H148 1,046 / 1,082.
//   The same form, two CTAs per SM on SMs of their own, where its step for two (1.27 us) and K1 on the others take about the
//     same time, and long chains: against the line above T8192 H75 636 / 639, H88 672 / 655, H96 686 / 651, H104 716 / 705, H111
//     769 / 772; T1024 H88 106 / 108, H96 109 / 107, H111 115 / 120.  The line in chunks, 64 / 128 / 192 / 256: H81 100 and 108 / 173
//     and 174 / 249 and 248 / 339 and 329, H88 102 and 106 / 179 and 178 / 263 and 257 / 353 and 344, H96 106 and 109 / 187 and 185 / 278 and
//     274 / 362 and 358; with the most chains, where K1 on the SMs left is the longer part, it comes later: H100 equal at 256, H103
//     387 and 393 there.
struct Beside {
  int win;                       // chunks per window; 0 = K2 starts after K1
  int variant, vsplit;           // K2's form: pick_split's, or one with the same bits
  int sms, k2_sms, k2_sm_ctas;   // see K1Params
};

Beside beside_plan(const KdaFwdArgs* a) {
  Beside r = {};
  if (a->n_seqs > 0) return r;
  r.sms = device_sms();
  pick_split(a, false, &r.vsplit, &r.variant, r.sms);
  const long long chains = static_cast<long long>(a->B) * a->H, nt = (static_cast<long long>(a->T) + kda::BT - 1) / kda::BT;
  const bool automatic = a->k2_variant == 0 && a->k2_vsplit == 0;
  long long k2_sms = 0;
  if (r.variant == 1 && r.vsplit >= 8 && chains * r.vsplit <= r.sms) {
    k2_sms = r.sms; r.k2_sm_ctas = 2;
  } else if (automatic && r.variant == 1 && chains * 6 <= r.sms) {
    k2_sms = chains * 4;
  } else if (automatic && ((r.variant == 1 && (chains * 15 - 2LL * r.sms) * nt >= 18750) || (r.variant == 3 && chains * 7 <= 2LL * r.sms && nt >= 72))) {
    k2_sms = chains * 2; r.variant = 3; r.vsplit = 2;
  } else if (r.variant == 4 && chains * 11 > 6LL * r.sms && chains * 10 <= 7LL * r.sms && nt >= 256) {
    k2_sms = (chains + 1) / 2;
  } else if (r.variant == 4 && chains * 14 <= 13LL * r.sms) {
    k2_sms = chains; r.k2_sm_ctas = 2;
  } else {
    return r;
  }
  r.k2_sms = static_cast<int>(k2_sms);
  const long long round = 2LL * r.sms;   // items that K1 has in flight
  if (chains * nt < 8 * round) return r;   // K1 is over in a few rounds: nothing to run beside
  // o is written while K1 still reads its inputs: they may not overlap (h0 and ht are safe: a chain's final
  // state is written once every window, so every item of K1, is finished)
  const int64_t* os = a->o_stride;
  for (int i = 0; i < 3; ++i)
    if (os[i] < 0 || a->beta_stride[i] < 0) return r;
  const int hq = a->Hq > 0 ? a->Hq : a->H;
  const Span o = span_of(a->o, os, a, a->H, kda::D, 2);
  const Span in[7] = {span_of(a->q, a->q_stride, a, hq, kda::D, 2), span_of(a->k, a->k_stride, a, hq, kda::D, 2),
                      span_of(a->v, a->v_stride, a, a->H, kda::D, 2),
                      span_of(a->g, a->g_stride, a, a->H, kda::D, a->g_dtype == KDA_G_BF16 ? 2 : 4),
                      span_of(a->beta, a->beta_stride, a, a->H, 1, 4),
                      {reinterpret_cast<uintptr_t>(a->A_log), reinterpret_cast<uintptr_t>(a->A_log + (a->A_log ? a->H : 0))},
                      {reinterpret_cast<uintptr_t>(a->dt_bias),
                       reinterpret_cast<uintptr_t>(a->dt_bias + (a->dt_bias ? static_cast<int64_t>(a->H) * kda::D : 0))}};
  for (const Span& s : in)
    if (o.lo < s.hi && s.lo < o.hi) return r;
  // windows of two rounds of K1, where it has most SMs to itself of one: T8192 H32 359 -> 355, but B2 T4096 H8 138 -> 145
  const long long by_count = (nt + kda::MAX_WINDOWS - 1) / kda::MAX_WINDOWS;
  const long long by_round = ((r.k2_sm_ctas == 0 ? 1 : 2) * round + chains - 1) / chains;
  r.win = static_cast<int>(by_count > by_round ? by_count : by_round);
  return r;
}

// 2^g may be factored as 2^(g-g_mid) * 2^(g_mid) only while no factor can underflow:
// 16 tokens * |lower_bound| * RCP_LN2 must stay inside the fp32 exponent range.
bool fast_exp(const KdaFwdArgs* a) {
  return (a->flags & KDA_FLAG_GATE_IN_KERNEL) && (16.0f * -a->lower_bound * kda::RCP_LN2 <= 120.0f);
}

int do_k1(const KdaFwdArgs* a, cudaStream_t st, const Beside& side = Beside{}) {
  kda::K1Params p;
  memset(&p, 0, sizeof(p));
  p.q = static_cast<const __nv_bfloat16*>(a->q);
  p.k = static_cast<const __nv_bfloat16*>(a->k);
  p.v = static_cast<const __nv_bfloat16*>(a->v);
  p.g = a->g;
  p.beta = a->beta;
  p.A_log = a->A_log;
  p.dt_bias = a->dt_bias;
  p.rec = rec_ptr(a);
  p.status = status_ptr(a);
  p.g_out = a->g_out;
  p.ainv_out = a->ainv_out;
  p.B = a->B; p.T = a->T; p.H = a->H; p.NT = (a->T + kda::BT - 1) / kda::BT;
  p.div_h.set(static_cast<uint32_t>(p.H));
  p.div_nt.set(static_cast<uint32_t>(p.NT));
  for (int i = 0; i < 3; ++i) {
    p.q_s[i] = a->q_stride[i]; p.k_s[i] = a->k_stride[i]; p.v_s[i] = a->v_stride[i];
    p.g_s[i] = a->g_stride[i]; p.beta_s[i] = a->beta_stride[i];
  }
  p.scale = a->scale;
  p.lower_bound = a->lower_bound;
  p.flags = a->flags;
  if (a->n_seqs > 0) {
    p.chunk_table = reinterpret_cast<const int4*>(a->chunk_table);
    p.n_chunks = a->n_chunks;
  }
  p.Hq = a->Hq > 0 ? a->Hq : a->H;
  p.div_g.set(static_cast<uint32_t>(p.H / p.Hq));
  if (side.win > 0) {
    p.progress = status_ptr(a) + kda::HDR_PROGRESS;
    p.n_sms = side.sms; p.k2_sms = side.k2_sms; p.k2_sm_ctas = side.k2_sm_ctas;
    p.div_b.set(static_cast<uint32_t>(p.B));
    p.div_win.set(static_cast<uint32_t>(side.win) * p.B * p.H);
  }
  // The four tensor maps depend only on the input pointers, sizes and strides: a loop that calls with
  // the same buffers (a serving loop, a benchmark) re-uses the maps of its previous call.
  struct MapKey {
    const void *q, *k, *v, *g;
    int32_t B, T, H, Hq, g_dtype;
    int64_t s[12];
  };
  thread_local MapKey last_key;
  thread_local CUtensorMap last_maps[4];
  thread_local bool have_maps = false;
  MapKey key;
  memset(&key, 0, sizeof(key));
  key.q = a->q; key.k = a->k; key.v = a->v; key.g = a->g;
  key.B = a->B; key.T = a->T; key.H = a->H; key.Hq = p.Hq; key.g_dtype = a->g_dtype;
  for (int i = 0; i < 3; ++i) {
    key.s[i] = a->q_stride[i]; key.s[3 + i] = a->k_stride[i]; key.s[6 + i] = a->v_stride[i]; key.s[9 + i] = a->g_stride[i];
  }
  cudaError_t e = cudaSuccess;
  if (have_maps && memcmp(&key, &last_key, sizeof(key)) == 0) {
    p.tm_q = last_maps[0]; p.tm_k = last_maps[1]; p.tm_v = last_maps[2]; p.tm_g = last_maps[3];
  } else {
    const char* what = "";
    e = kda::k1_encode_tensor_maps(p, a->g_dtype == KDA_G_BF16, &what);
    if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: building the TMA descriptor failed for: %s", what);
    last_key = key;
    last_maps[0] = p.tm_q; last_maps[1] = p.tm_k; last_maps[2] = p.tm_v; last_maps[3] = p.tm_g;
    have_maps = true;
  }
  e = kda::launch_k1(p, a->g_dtype == KDA_G_BF16, fast_exp(a), st);
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: K1 launch failed: %s", cudaGetErrorString(e));
  ++g_launches;
  return KDA_OK;
}

struct H0Flags { const int32_t* flags; int n, epoch; };

int do_k2(const KdaFwdArgs* a, bool state_only, int zero_u, cudaStream_t st, const KdaPeerPushArgs* push = nullptr,
          const H0Flags* h0f = nullptr, bool after_k1 = false, const Beside& side = Beside{}) {
  kda::K2Params p;
  memset(&p, 0, sizeof(p));
  p.rec = rec_ptr(a);
  p.h0 = a->h0;
  p.o = static_cast<__nv_bfloat16*>(a->o);
  p.ht = a->ht;
  p.status = status_ptr(a);
  p.B = a->B; p.T = a->T; p.H = a->H; p.NT = (a->T + kda::BT - 1) / kda::BT;
  for (int i = 0; i < 3; ++i) p.o_s[i] = a->o_stride[i];
  p.scale = a->scale;
  p.zero_u = zero_u == 1;
  p.k_first = (a->flags & KDA_FLAG_STATE_K_FIRST) ? 1 : 0;
  if (side.win > 0) {
    p.progress = status_ptr(a) + kda::HDR_PROGRESS;
    p.win_chunks = side.win;
    // two CTAs of K1 leave K2 126 KB of an SM, 8 KB less with an fp32 gate, 17 with general centring
    p.long_ring = side.k2_sm_ctas == 0 ? 8 : 6 - (a->g_dtype == KDA_G_FP32) - !fast_exp(a);
  }
  p.pair_mode = (state_only && zero_u == 2) ? 1 : 0;
  if (a->n_seqs > 0) {
    p.seq_table = reinterpret_cast<const int4*>(a->seq_table);
    p.n_seqs = a->n_seqs;
  }
  int vsplit = 4, variant = 3;
  pick_split(a, state_only, &vsplit, &variant);
  if (side.win > 0) { vsplit = side.vsplit; variant = side.variant; }
  if (after_k1) {
    // Launched ahead of K1's end: K2's CTAs are set up (barriers, tensor memory, the initial state) on the SMs
    // that K1 leaves.  Whole forward on B200, ordinary launch against this one: B1 T100 H32 17.0 -> 14.9 us, T512
    // H32 35.6 -> 35.1, T1024 H8 41.3 -> 38.4, B8 T2048 H32 512 -> 507.  Not the 8-row form with four consumer
    // warps per CTA on more than 32 chunks: in the order in which K1 leaves the SMs its CTAs step slower than
    // in the order of an ordinary launch.  Of the calls that still run after K1 and reach this line that holds for the longest only
    // (T2500 H26 110.2 -> 112.5, T4096 H25 171.5 -> 171.7, T1600 H28 76.2 -> 76.3, T1540 H24 70.0 -> 70.2); shorter ones would be faster
    // started ahead: T1600 H30 76.2 -> 75.3, T1200 H32 61.6 -> 59.2, T1000 H24 47.6 -> 46.9, T800 H37 45.4 -> 43.0, T544 H20 28.8 -> 26.7.
    const long long steps = a->n_seqs > 0 ? a->n_chunks / a->n_seqs : p.NT;
    // Nor packed sequences of more than eight chunks in the mean in the 16-row form on more CTAs than SMs: the long
    // chains of unequal lengths then run on beside others of the launch.  3 to 64 sequences of log-normal lengths
    // (sigma 1), 75 to 148 chains, whole forward: up to three chunks in the mean 0.92 of the ordinary launch's time, four to
    // eight 0.97, nine to 16 1.03, more 1.04 and up to 1.31 (16 sequences, H8, the longest 264 chunks of 460: 285 -> 372 us).
    const long long chains = static_cast<long long>(a->n_seqs > 0 ? a->n_seqs : a->B) * a->H;
    const bool uneven = a->n_seqs > 0 && variant == 3 && chains * vsplit > device_sms() && steps > 8;
    p.pdl = side.win > 0 || (variant != 5 && !(variant == 1 && vsplit == 4 && steps > 32) && !uneven);
    // without the bound on the CTAs per SM: T1024 H8 48.2 us
    p.one_per_sm = p.pdl && (side.win > 0 ? side.k2_sm_ctas == 0 && chains * (variant == 4 ? 1 : vsplit) <= side.k2_sms
                                         : chains * (variant == 4 ? 1 : vsplit) <= device_sms());
  }
  if (p.pair_mode) {
    p.k_first = 0;   // the transforms are always written [chains][2][V][K]
    // Both transforms of a segment in one launch.  Few chains (two recurrences per chain still give
    // every warp an SM sub-partition to itself): the 8-row form over twice as many chains.  Up to
    // the 8-row form's own limit: the two recurrences share a warp and its operand loads.  Beyond:
    // the 16-row form over twice as many chains.
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long bh = static_cast<long long>(a->n_seqs > 0 ? a->n_seqs : a->B) * a->H;
    if (2 * bh > 0x3fffffffLL) return fail(KDA_ERR_INVALID_ARG, "kda: too many chains%s", "");
    cudaError_t pe;
    if (push != nullptr) {
      // the tiles go straight into the owners' receive buffers: only the 8-row pair form does that
      if (!(variant == 1 || variant == 5))
        return fail(KDA_ERR_UNSUPPORTED, "kda: the fused push needs the 8-row pair form%s (too many chains: %lld)", "", bh);
      const long long hp = push->slice_floats / (2LL * kda::D * kda::D);
      if (hp <= 0 || hp * push->world != bh || push->slice_floats % (2LL * kda::D * kda::D) != 0)
        return fail(KDA_ERR_INVALID_ARG, "kda: slice_floats must be chains / world whole (M, Q) pairs%s (chains %lld)", "", bh);
      p.push_on = 1;
      p.push_hp = static_cast<int>(hp);
      p.push_epoch = push->epoch;
      p.push_dst_offset = push->dst_offset_floats;
      p.push_counter = push->counter;
      for (int d = 0; d < push->world; ++d) { p.push_dst[d] = push->dst[d]; p.push_flag[d] = push->flag[d]; }
      p.pair_mode = 0;
      pe = kda::launch_k2n_pair(p, vsplit, st);
    } else if (a->k2_variant == 0 && a->k2_vsplit == 0 && 2 * bh * 4 <= sms) {
      p.n_chains = static_cast<int>(2 * bh);
      pe = kda::launch_k2n(p, 2 * bh * 16 <= sms ? 16 : 2 * bh * 8 <= sms ? 8 : 4, 1, true, st);
    } else if (variant == 1 || variant == 5) {
      p.pair_mode = 0;   // the pair is compiled into the kernel
      pe = kda::launch_k2n_pair(p, vsplit, st);
    } else {
      p.n_chains = static_cast<int>(2 * bh);
      pick_split(a, state_only, &vsplit, &variant, 0, 2);
      pe = (variant == 3) ? kda::launch_k2m(p, vsplit, true, st) : cudaErrorInvalidValue;
    }
    if (pe != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: K2 (transform pair) launch failed: %s", cudaGetErrorString(pe));
    ++g_launches;
    return KDA_OK;
  }
  if (h0f != nullptr) {
    // the entry state is stored by other GPUs: the kernels that can wait for it themselves are the 8-row and
    // the 16-row form
    if (!(variant == 1 || variant == 3))
      return fail(KDA_ERR_UNSUPPORTED, "kda: this K2 form cannot wait for the entry state%s (variant %lld)", "", variant);
    p.h0_flags = h0f->flags; p.h0_n_flags = h0f->n; p.h0_epoch = h0f->epoch;
  }
  cudaError_t e;
  if (variant == 4) {
    // Tail wave.  The tensor-memory form holds two chains per SM at once; when the chains left over
    // after the full waves are at most half as many as SMs, they run faster in an mma.sync form
    // (8-row for at most SMs/4 chains, 0.45 us per step; 16-row: two CTAs per chain, one per SM, 0.53 us
    // per step; against 0.84 for a lone tensor-memory CTA), launched behind the full waves, at every length that the
    // tensor-memory form is chosen for.  kda_fwd in us, no tail / 16-row / 8-row, 296 chains and so many more x chunks:
    // 9 x 4 45.5 / 43.4 / 41.3, 9 x 64 335 / 325 / 306; 37 x 4 47.3 / 45.0 / 45.2, 37 x 64 353 / 342 / 331; 38 x 4 47.9 /
    // 45.3 / 47.4, 38 x 64 353 / 343 / 363; 74 x 4 49.7 / 47.7 / 50.5, 74 x 64 374 / 365 / 389; 75 x 4 50.7 / 52.6,
    // 75 x 64 375 / 400.  Only for the automatic choice.
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long bh = static_cast<long long>(a->n_seqs > 0 ? a->n_seqs : a->B) * a->H;
    const long long tail = bh % (2LL * sms);
    // Packed sequences of unequal length: the CTAs come in waves, so the longest chains go first (a long one
    // that starts in the last wave runs on alone while the rest of the chip is idle): 24 sequences of 16,411
    // tokens, H32, whole forward 747 -> 616 us.  Every CTA works its chain out, which costs about 0.4 us per wave: up to
    // 2 % where the chains are of equal length and four chunks short.  Hence the bound on n_seqs (eight lengths per
    // lane), and none of it where many waves of short chains leave little at the end (256 sequences of about 4
    // chunks, H16: 420 us in their own order, 435 by length; of 8 to 13 chunks 701 and 709, of 29 1,240 and 1,040).
    const long long mean_steps = a->n_seqs > 0 ? a->n_chunks / a->n_seqs : 0;
    p.by_length = a->n_seqs > 1 && a->n_seqs <= kda::MAX_SORTED_SEQS && bh > sms && bh <= 4LL * sms * mean_steps;
    // A sequence much longer than the others: its chains go on alone when the rest is done, at 1.3 us per step while their SM
    // has a second CTA and 0.85 without, against 0.53 in the 16-row form.  So the longest sequences, on at most half of the
    // SMs, run there, in front of and beside the tensor-memory launch (which starts when K1 has ended, about 2 us later
    // than without), if they are long: more steps than 0.9 x the chunks of all chains per SM, which take 0.67 us each in pairs,
    // and than 1.5 x the mean.  The lengths are on the device: either kernel leaves out what the other does.  Whole forward on one
    // set of buffers, us, without / with, log-normal lengths (sigma 1): 24 sequences of 16,411 tokens H32 525 / 519 (as one call among
    // others on changing buffers 536 / 534), 16 of 20,000 H32 636 / 630, 8 of 24,000 H32 780 / 763, 6 of 20,000 H32 774 / 657, 30 of
    // 24,000 H16 388 / 379, 40 of 28,000 H8 306 / 228, 64 of 32,000 H8 470 / 366.  Where no sequence is long, or hardly, the launch costs
    // up to 1.6 %: 16 x 1,024 H32 494 / 501, 32 x 500 H16 258 / 262, 5 x 2,000 H32 329 / 331, 64 x 500 H32 1,001 / 1,007, 48 of 32,000 H16
    // 495 / 503; shorter ones do not pay for it (8 x 520 H32 126 / 128).  The factor at 0.8 / 0.9 / 1.0: 24 of 16,411 H32 517 / 519 / 542 and
    // with other lengths 516 / 514 / 510, 16 of 20,000 H32 621 / 630 / 659, 6 of 20,000 639 / 657 / 663, 30 of 24,000 H16 373 / 379 / 402, 40
    // of 28,000 H8 228 / 228 / 233.  On all SMs instead of half of them 6 of 20,000 H32 took 692 in place of 653; with 1.25 x the mean
    // 4 x 2,500 H32 356 in place of 304.
    const long long items = static_cast<long long>(a->n_chunks) * a->H;
    const int long_max = static_cast<int>(std::min<long long>(a->n_seqs - 1, sms / (4LL * a->H)));
    if (a->k2_variant == 0 && (p.by_length || bh <= sms) && a->n_seqs <= kda::MAX_SORTED_SEQS && long_max > 0 && items >= 64LL * sms) {
      p.by_length = 1;
      p.long_max = long_max;
      p.long_len = static_cast<int>(std::max(9 * items / (10LL * sms), 3LL * a->n_chunks / (2LL * a->n_seqs))) + 1;
      p.n_chains = long_max * a->H;
      p.one_per_sm = 1;
      e = kda::launch_k2m(p, 2, false, st);
      if (e == cudaSuccess) {
        ++g_launches;
        p.n_chains = p.one_per_sm = 0;
        p.pdl = 1;
        e = kda::launch_k2t(p, st);
      }
    } else if (a->k2_variant == 0 && bh > 2LL * sms && tail > 0 && tail * 2 <= sms) {
      p.chain0 = 0;
      p.n_chains = static_cast<int>(bh - tail);
      e = kda::launch_k2t(p, st);
      if (e == cudaSuccess) {
        ++g_launches;
        p.pdl = p.one_per_sm = 0;   // behind the full waves, an ordinary launch
        p.chain0 = static_cast<int>(bh - tail);
        p.n_chains = static_cast<int>(tail);
        // the few-chain rule of pick_split applied to the tail alone
        if (tail * 4 <= sms) e = kda::launch_k2n(p, tail * 16 <= sms ? 16 : tail * 8 <= sms ? 8 : 4, 1, false, st);
        else e = kda::launch_k2m(p, 2, false, st);
      }
    } else {
      e = kda::launch_k2t(p, st);
    }
  } else {
    e = (variant == 3) ? kda::launch_k2m(p, vsplit, state_only, st)
        : (variant == 5) ? kda::launch_k2la(p, vsplit, state_only, st)
                         : kda::launch_k2n(p, vsplit, 1, state_only, st);
  }
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: K2 launch failed: %s", cudaGetErrorString(e));
  ++g_launches;
  return KDA_OK;
}

}  // namespace

namespace kda {
// lets the other translation units of the library report through kda_last_error()
void set_last_error(const char* msg) { snprintf(g_err, sizeof(g_err), "%s", msg); }
}  // namespace kda

extern "C" {

size_t kda_fwd_workspace_bytes(int32_t B, int32_t T, int32_t H) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  const size_t nt = (static_cast<size_t>(T) + kda::BT - 1) / kda::BT;
  return kda::WS_HEADER_BYTES + static_cast<size_t>(B) * H * nt * kda::REC_BYTES;
}

int kda_fwd(const KdaFwdArgs* a, void* stream) {
  g_launches = 0;
  if (int rc = check_k1(a)) return rc;
  if (int rc = check_k2(a, false)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const Beside side = beside_plan(a);
  if (side.win > 0) {   // the window counters must be zero before either kernel starts
    cudaError_t e = kda::launch_clear_header(status_ptr(a), st);
    if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: header clear failed: %s", cudaGetErrorString(e));
    ++g_launches;
  }
  if (int rc = do_k1(a, st, side)) return rc;
  return do_k2(a, false, 0, st, nullptr, nullptr, true, side);
}

int kda_selftest_window_wait(const KdaFwdArgs* a, void* stream) {
  g_launches = 0;
  if (int rc = check_k1(a)) return rc;
  if (int rc = check_k2(a, false)) return rc;
  const Beside side = beside_plan(a);
  if (side.win == 0) return fail(KDA_ERR_INVALID_ARG, "kda: K2 does not run beside K1 for this problem%s", "");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(status_ptr(a) + kda::HDR_PROGRESS, 0, kda::MAX_WINDOWS * sizeof(int), st);
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: header clear failed: %s", cudaGetErrorString(e));
  return do_k2(a, false, 0, st, nullptr, nullptr, false, side);
}

int kda_fwd_k1(const KdaFwdArgs* a, void* stream) {
  g_launches = 0;
  if (int rc = check_k1(a)) return rc;
  return do_k1(a, static_cast<cudaStream_t>(stream));
}

int kda_fwd_k2(const KdaFwdArgs* a, void* stream) {
  g_launches = 0;
  if (int rc = check_k2(a, false)) return rc;
  return do_k2(a, false, 0, static_cast<cudaStream_t>(stream));
}

int kda_fwd_k2_state(const KdaFwdArgs* a, int zero_u, void* stream) {
  g_launches = 0;
  if (int rc = check_k2(a, true)) return rc;
  if (a->ht == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: the state-only pass needs ht%s", "");
  if (zero_u < 0 || zero_u > 2) return fail(KDA_ERR_INVALID_ARG, "kda: zero_u must be 0, 1 or 2%s (got %lld)", "", zero_u);
  return do_k2(a, true, zero_u, static_cast<cudaStream_t>(stream));
}

int kda_recurrent_fwd(const KdaFwdArgs* a, void* stream) {
  g_launches = 0;
  if (a == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: args is NULL%s", "");
  if (a->B <= 0 || a->T <= 0 || a->H <= 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: B, T, H must be positive%s (T=%lld, H=%lld)", "", a->T, a->H);
  if (a->n_seqs != 0) return fail(KDA_ERR_INVALID_ARG, "kda: the recurrent step takes a fixed-length batch%s (n_seqs must be 0)", "");
  if (a->Hq < 0 || (a->Hq > 0 && a->H % a->Hq != 0))
    return fail(KDA_ERR_INVALID_ARG, "kda: H%s (%lld) must be a multiple of Hq (%lld)", "", a->H, a->Hq);
  if (!a->q || !a->k || !a->v || !a->g || !a->beta || !a->o || !a->A_log)
    return fail(KDA_ERR_INVALID_ARG, "kda: the recurrent step needs q, k, v, g, beta, A_log and o%s", "");
  const uint32_t all = KDA_FLAG_GATE_IN_KERNEL | KDA_FLAG_QK_L2NORM | KDA_FLAG_BETA_SIGMOID;
  if ((a->flags & all) != all)
    return fail(KDA_ERR_INVALID_ARG, "kda: the recurrent step computes gate, l2-norm and beta sigmoid in the kernel%s; set all three flags", "");
  if (a->g_dtype != KDA_G_FP32 && a->g_dtype != KDA_G_BF16)
    return fail(KDA_ERR_INVALID_ARG, "kda: g_dtype must be KDA_G_FP32 or KDA_G_BF16%s (got %lld)", "", a->g_dtype);
  if (!(a->lower_bound > -11.0f && a->lower_bound < 0.0f))
    return fail(KDA_ERR_INVALID_ARG, "kda: lower_bound must be in (-11, 0)%s", "");
  if (!row_aligned(a->q, a->q_stride, 2) || !row_aligned(a->k, a->k_stride, 2) || !row_aligned(a->v, a->v_stride, 2) ||
      !row_aligned(a->g, a->g_stride, a->g_dtype == KDA_G_BF16 ? 2 : 4) || !row_aligned(a->o, a->o_stride, 2))
    return fail(KDA_ERR_INVALID_ARG, "kda: q/k/v/g/o rows must start on 16-byte boundaries%s", "");
  if (!params_aligned(a, true))
    return fail(KDA_ERR_INVALID_ARG, "kda: beta, A_log and dt_bias must be 4-byte aligned%s", "");
  for (const void* ptr : {static_cast<const void*>(a->h0), static_cast<const void*>(a->ht), static_cast<const void*>(a->dt_bias)})
    if (ptr != nullptr && reinterpret_cast<uintptr_t>(ptr) % 16 != 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: h0, ht and dt_bias must be 16-byte aligned%s", "");
  kda::RecurrentParams p;
  memset(&p, 0, sizeof(p));
  p.q = static_cast<const __nv_bfloat16*>(a->q);
  p.k = static_cast<const __nv_bfloat16*>(a->k);
  p.v = static_cast<const __nv_bfloat16*>(a->v);
  p.g = a->g; p.beta = a->beta; p.A_log = a->A_log; p.dt_bias = a->dt_bias;
  p.h0 = a->h0; p.ht = a->ht; p.o = static_cast<__nv_bfloat16*>(a->o);
  p.B = a->B; p.T = a->T; p.H = a->H;
  p.group = a->Hq > 0 ? a->H / a->Hq : 1;
  p.k_first = (a->flags & KDA_FLAG_STATE_K_FIRST) ? 1 : 0;
  for (int i = 0; i < 3; ++i) {
    p.q_s[i] = a->q_stride[i]; p.k_s[i] = a->k_stride[i]; p.v_s[i] = a->v_stride[i];
    p.g_s[i] = a->g_stride[i]; p.beta_s[i] = a->beta_stride[i]; p.o_s[i] = a->o_stride[i];
  }
  p.scale = a->scale;
  p.lower_bound = a->lower_bound;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = kda::launch_recurrent(p, a->g_dtype == KDA_G_BF16, sms, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: recurrent launch failed: %s", cudaGetErrorString(e));
  ++g_launches;
  return KDA_OK;
}

static_assert(KDA_MAX_PEERS == kda::MAX_PEERS, "header and kernel limits differ");
static_assert(sizeof(KdaPeerPushArgs) == 296 && offsetof(KdaPeerPushArgs, epoch) == 292 && sizeof(KdaFoldPeerArgs) == 296 &&
                  offsetof(KdaFoldPeerArgs, counter) == 288,
              "the ctypes mirrors of these structures pin their layout");

static int fold_impl(const KdaFoldArgs* f, const KdaFoldPeerArgs* peer, void* stream) {
  g_launches = 0;
  if (f == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: fold args is NULL%s", "");
  if (f->mq == nullptr || (peer == nullptr && f->s_in == nullptr && f->final_out == nullptr))
    return fail(KDA_ERR_INVALID_ARG, "kda: the fold needs mq and at least one of s_in / final_out%s", "");
  if (peer != nullptr) {
    if (peer->n_wait < 0 || peer->n_wait > KDA_MAX_PEERS || peer->n_signal < 0 || peer->n_signal > KDA_MAX_PEERS ||
        f->n_seg > KDA_MAX_PEERS)
      return fail(KDA_ERR_INVALID_ARG, "kda: the peer fold takes at most %s16 segments, flags and signals", "");
    if ((peer->n_wait > 0 && peer->wait_flags == nullptr) || (peer->n_signal > 0 && peer->counter == nullptr) || peer->epoch <= 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: the peer fold needs wait_flags, counter and a positive epoch%s", "");
    for (int i = 0; i <= f->n_seg && i <= KDA_MAX_PEERS; ++i)
      if (peer->s_in_seg[i] != nullptr && reinterpret_cast<uintptr_t>(peer->s_in_seg[i]) % 16 != 0)
        return fail(KDA_ERR_INVALID_ARG, "kda: s_in_seg entries must be 16-byte aligned%s", "");
    for (int i = 0; i < peer->n_signal; ++i)
      if (peer->signal[i] == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: signal[%s%lld] is NULL", "", i);
  }
  if (f->n_chains <= 0 || f->n_seg < 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the fold needs n_chains > 0 and n_seg >= 0%s (got %lld, %lld)", "", f->n_chains, f->n_seg);
  const int64_t state = static_cast<int64_t>(kda::D) * kda::D;
  const int64_t span = f->use_q ? 2 * state : state;   // without Q only the M block has to lie inside a stride
  if (f->n_seg > 0 && ((f->n_chains > 1 && f->chain_stride < span) || (f->n_seg > 1 && f->seg_stride < span)))
    return fail(KDA_ERR_INVALID_ARG, "kda: the fold's strides must span the 128 x 128 blocks they step over%s", "");
  if (f->seg_stride % 4 != 0 || f->chain_stride % 4 != 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the fold's strides must be multiples of 4 floats%s (every M_j is copied 16 bytes at a time)", "");
  const int64_t h0_stride = f->h0_stride != 0 ? f->h0_stride : state;
  const int64_t final_stride = f->final_stride != 0 ? f->final_stride : state;
  if (h0_stride < state || final_stride < state)
    return fail(KDA_ERR_INVALID_ARG, "kda: h0_stride and final_stride must be 0 (dense) or at least 128 x 128%s", "");
  if (f->status != nullptr && reinterpret_cast<uintptr_t>(f->status) % 4 != 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: status must be 4-byte aligned%s", "");
  for (const void* ptr : {static_cast<const void*>(f->mq), static_cast<const void*>(f->h0), static_cast<const void*>(f->s_in),
                          static_cast<const void*>(f->final_out)})
    if (ptr != nullptr && reinterpret_cast<uintptr_t>(ptr) % 16 != 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: mq, h0, s_in and final_out must be 16-byte aligned%s", "");
  if (static_cast<long long>(f->n_chains) * (kda::D / 4) > 0x7fffffffLL)
    return fail(KDA_ERR_INVALID_ARG, "kda: too many chains for one fold launch%s", "");
  kda::FoldParams p;
  memset(&p, 0, sizeof(p));
  p.mq = f->mq; p.seg_stride = f->seg_stride; p.chain_stride = f->chain_stride;
  p.h0 = f->h0; p.h0_stride = h0_stride;
  p.s_in = f->s_in; p.final_out = f->final_out; p.final_stride = final_stride;
  p.n_chains = f->n_chains; p.n_seg = f->n_seg; p.use_q = f->use_q ? 1 : 0;
  p.status = f->status;
  if (peer != nullptr) {
    p.s_in = nullptr;
    p.wait_flags = peer->wait_flags; p.n_wait = peer->n_wait; p.epoch = peer->epoch;
    p.s_in_seg_on = 1;
    for (int i = 0; i <= f->n_seg; ++i) p.s_in_seg[i] = peer->s_in_seg[i];
    p.n_signal = peer->n_signal;
    for (int i = 0; i < peer->n_signal; ++i) p.signal[i] = peer->signal[i];
    p.counter = peer->counter;
  }
  cudaError_t e = kda::launch_state_fold(p, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: fold launch failed: %s", cudaGetErrorString(e));
  ++g_launches;
  return KDA_OK;
}

int kda_state_fold_ex(const KdaFoldArgs* f, void* stream) { return fold_impl(f, nullptr, stream); }

int kda_state_fold_peer(const KdaFoldArgs* f, const KdaFoldPeerArgs* peer, void* stream) {
  if (peer == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: peer args is NULL%s", "");
  return fold_impl(f, peer, stream);
}

static int check_push_targets(const KdaPeerPushArgs* a) {
  if (a == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: push args is NULL%s", "");
  if (a->world < 1 || a->world > KDA_MAX_PEERS || a->epoch <= 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the push needs 1..16 ranks and a positive epoch%s (world %lld)", "", a->world);
  if (a->counter == nullptr || a->slice_floats <= 0 || a->slice_floats % 4 != 0 || a->dst_offset_floats < 0 ||
      a->dst_offset_floats % 4 != 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the push needs a counter and 16-byte multiples for slice and offset%s", "");
  for (int d = 0; d < a->world; ++d)
    if (a->dst[d] == nullptr || a->flag[d] == nullptr || reinterpret_cast<uintptr_t>(a->dst[d]) % 16 != 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: dst[%s%lld] and its flag must be set, dst 16-byte aligned", "", d);
  return KDA_OK;
}

int kda_fwd_k2_state_push(const KdaFwdArgs* a, const KdaPeerPushArgs* push, void* stream) {
  g_launches = 0;
  if (int rc = check_common(a)) return rc;
  if (int rc = check_k2(a, true)) return rc;
  if (int rc = check_push_targets(push)) return rc;
  return do_k2(a, true, 2, static_cast<cudaStream_t>(stream), push);
}

int kda_fwd_k2_after_flags(const KdaFwdArgs* a, const int32_t* flags, int32_t n, int32_t epoch, void* stream) {
  g_launches = 0;
  if (int rc = check_common(a)) return rc;
  if (int rc = check_k2(a, false)) return rc;
  if (flags == nullptr || n < 1 || n > KDA_MAX_PEERS || epoch <= 0 || a->h0 == nullptr)
    return fail(KDA_ERR_INVALID_ARG, "kda: the call needs h0, 1..16 flags and a positive epoch%s (n %lld)", "", n);
  const H0Flags h0f{flags, n, epoch};
  return do_k2(a, false, 0, static_cast<cudaStream_t>(stream), nullptr, &h0f);
}

int kda_peer_push(const KdaPeerPushArgs* a, void* stream) {
  g_launches = 0;
  if (a == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: push args is NULL%s", "");
  if (a->world < 1 || a->world > KDA_MAX_PEERS || a->epoch <= 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the push needs 1..16 ranks and a positive epoch%s (world %lld)", "", a->world);
  if (a->src == nullptr || a->counter == nullptr || a->slice_floats <= 0 || a->slice_floats % 4 != 0 ||
      a->dst_offset_floats < 0 || a->dst_offset_floats % 4 != 0 || reinterpret_cast<uintptr_t>(a->src) % 16 != 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the push needs src, counter and 16-byte multiples for slice and offset%s", "");
  kda::PeerPushParams p;
  memset(&p, 0, sizeof(p));
  for (int d = 0; d < a->world; ++d) {
    if (a->dst[d] == nullptr || a->flag[d] == nullptr || reinterpret_cast<uintptr_t>(a->dst[d]) % 16 != 0)
      return fail(KDA_ERR_INVALID_ARG, "kda: dst[%s%lld] and its flag must be set, dst 16-byte aligned", "", d);
    p.dst[d] = reinterpret_cast<float4*>(a->dst[d]);
    p.flag[d] = a->flag[d];
  }
  p.src = reinterpret_cast<const float4*>(a->src);
  p.dst_offset = a->dst_offset_floats / 4;
  p.slice = a->slice_floats / 4;
  p.counter = a->counter;
  p.world = a->world; p.epoch = a->epoch;
  cudaError_t e = kda::launch_peer_push(p, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: push launch failed: %s", cudaGetErrorString(e));
  ++g_launches;
  return KDA_OK;
}

int kda_peer_enable(int32_t peer_device) {
  int dev = 0, can = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: cudaGetDevice failed: %s", cudaGetErrorString(e));
  if (peer_device == dev) return KDA_OK;
  e = cudaDeviceCanAccessPeer(&can, dev, peer_device);
  if (e != cudaSuccess || !can) {
    cudaGetLastError();
    return fail(KDA_ERR_CUDA, "kda: this GPU cannot map the memory of GPU %s%lld", "", peer_device);
  }
  e = cudaDeviceEnablePeerAccess(peer_device, 0);
  if (e == cudaErrorPeerAccessAlreadyEnabled) {
    cudaGetLastError();
    e = cudaSuccess;
  }
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: enabling peer access failed: %s", cudaGetErrorString(e));
  return KDA_OK;
}

// ---- CUDA IPC for the peer exchange -------------------------------------------------------------
// The importing side opens a handle with ITS OWN device current, which is what maps the exporting
// GPU's memory for kernels of the importing GPU (a mapping made with another device current is
// not reachable from this one).  A handle is opened once per process and stays mapped.
namespace {
struct IpcOpened { cudaIpcMemHandle_t h; int dev; void* base; int refs; };
std::mutex g_ipc_mu;
std::vector<IpcOpened> g_ipc_opened;
}  // namespace

int kda_ipc_export(const void* ptr, void* handle_out, int64_t* offset_out) {
  if (ptr == nullptr || handle_out == nullptr || offset_out == nullptr)
    return fail(KDA_ERR_INVALID_ARG, "kda: ptr, handle_out and offset_out are required%s", "");
  typedef CUresult (*RangeFn)(CUdeviceptr*, size_t*, CUdeviceptr);
  static RangeFn range_fn = nullptr;
  if (range_fn == nullptr) {
    void* fp = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fp, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      return fail(KDA_ERR_CUDA, "kda: cuMemGetAddressRange is not available from this driver%s", "");
    range_fn = reinterpret_cast<RangeFn>(fp);
  }
  CUdeviceptr base = 0;
  size_t size = 0;
  if (range_fn(&base, &size, reinterpret_cast<CUdeviceptr>(ptr)) != CUDA_SUCCESS)
    return fail(KDA_ERR_CUDA, "kda: the pointer does not belong to a device allocation%s", "");
  cudaIpcMemHandle_t h;
  cudaError_t e = cudaIpcGetMemHandle(&h, reinterpret_cast<void*>(base));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(KDA_ERR_CUDA, "kda: cudaIpcGetMemHandle failed: %s", cudaGetErrorString(e));
  }
  memcpy(handle_out, &h, sizeof(h));
  *offset_out = static_cast<int64_t>(reinterpret_cast<CUdeviceptr>(ptr) - base);
  return KDA_OK;
}

int kda_ipc_open(const void* handle, int64_t offset, void** ptr_out) {
  if (handle == nullptr || ptr_out == nullptr || offset < 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: handle and ptr_out are required%s", "");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: cudaGetDevice failed: %s", cudaGetErrorString(e));
  cudaIpcMemHandle_t h;
  memcpy(&h, handle, sizeof(h));
  std::lock_guard<std::mutex> lock(g_ipc_mu);
  for (IpcOpened& o : g_ipc_opened)
    if (o.dev == dev && memcmp(&o.h, &h, sizeof(h)) == 0) {
      ++o.refs;
      *ptr_out = static_cast<char*>(o.base) + offset;
      return KDA_OK;
    }
  void* base = nullptr;
  e = cudaIpcOpenMemHandle(&base, h, cudaIpcMemLazyEnablePeerAccess);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(KDA_ERR_CUDA, "kda: cudaIpcOpenMemHandle failed: %s", cudaGetErrorString(e));
  }
  g_ipc_opened.push_back(IpcOpened{h, dev, base, 1});
  *ptr_out = static_cast<char*>(base) + offset;
  return KDA_OK;
}

int kda_ipc_close(const void* handle) {
  if (handle == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: handle is required%s", "");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: cudaGetDevice failed: %s", cudaGetErrorString(e));
  std::lock_guard<std::mutex> lock(g_ipc_mu);
  for (size_t i = 0; i < g_ipc_opened.size(); ++i) {
    IpcOpened& o = g_ipc_opened[i];
    if (o.dev != dev || memcmp(&o.h, handle, sizeof(o.h)) != 0) continue;
    if (--o.refs > 0) return KDA_OK;
    e = cudaIpcCloseMemHandle(o.base);
    g_ipc_opened.erase(g_ipc_opened.begin() + static_cast<long>(i));
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(KDA_ERR_CUDA, "kda: cudaIpcCloseMemHandle failed: %s", cudaGetErrorString(e));
    }
    return KDA_OK;
  }
  return fail(KDA_ERR_INVALID_ARG, "kda: this handle is not open on the current device%s", "");
}

int kda_flag_wait(const int32_t* flags, int32_t n, int32_t epoch, int32_t* status, void* stream) {
  g_launches = 0;
  if (flags == nullptr || n < 1 || n > 32 || epoch <= 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: the flag wait needs 1..32 flags and a positive epoch%s (n %lld)", "", n);
  cudaError_t e = kda::launch_flag_wait(flags, n, epoch, status, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: flag wait launch failed: %s", cudaGetErrorString(e));
  ++g_launches;
  return KDA_OK;
}

int kda_state_fold(const float* mq, int64_t seg_stride, int64_t chain_stride, const float* h0, float* s_in,
                   int32_t n_chains, int32_t n_seg, int32_t* status, void* stream) {
  if (s_in == nullptr) return fail(KDA_ERR_INVALID_ARG, "kda: the fold needs mq and s_in%s", "");
  KdaFoldArgs f;
  memset(&f, 0, sizeof(f));
  f.mq = mq; f.seg_stride = seg_stride; f.chain_stride = chain_stride; f.h0 = h0; f.s_in = s_in;
  f.n_chains = n_chains; f.n_seg = n_seg; f.use_q = 1; f.status = status;
  return kda_state_fold_ex(&f, stream);
}

int kda_varlen_fill_tables(const int32_t* cu, int32_t n_seqs, int32_t H, int32_t* chunk_table, int32_t* seq_table) {
  if (cu == nullptr || n_seqs <= 0 || H <= 0)
    return fail(KDA_ERR_INVALID_ARG, "kda: cu_seqlens, n_seqs and H are required%s", "");
  if (cu[0] != 0) return fail(KDA_ERR_INVALID_ARG, "kda: cu_seqlens must start at 0%s (got %lld)", "", cu[0]);
  long long chunks = 0;
  for (int i = 0; i < n_seqs; ++i) {
    const long long len = static_cast<long long>(cu[i + 1]) - cu[i];
    if (len <= 0) return fail(KDA_ERR_INVALID_ARG, "kda: sequence %s%lld is empty or cu_seqlens decreases", "", i);
    const long long nt = (len + kda::BT - 1) / kda::BT;
    if ((chunks + nt) * H > 0x7fffffffLL) return fail(KDA_ERR_INVALID_ARG, "kda: too many chunk records%s", "");
    if (chunk_table != nullptr && seq_table != nullptr) {
      seq_table[4 * i + 0] = cu[i];
      seq_table[4 * i + 1] = static_cast<int32_t>(nt);
      seq_table[4 * i + 2] = static_cast<int32_t>(chunks * H);
      seq_table[4 * i + 3] = static_cast<int32_t>(len);
      for (long long n = 0; n < nt; ++n) {
        int32_t* e = chunk_table + 4 * (chunks + n);
        e[0] = cu[i] + static_cast<int32_t>(n * kda::BT);
        e[1] = static_cast<int32_t>(len - n * kda::BT < kda::BT ? len - n * kda::BT : kda::BT);
        e[2] = static_cast<int32_t>(chunks * H + n);
        e[3] = static_cast<int32_t>(nt);
      }
    }
    chunks += nt;
  }
  return static_cast<int>(chunks);
}

int kda_fwd_status(const void* workspace, void* stream, int32_t* status_out) {
  if (workspace == nullptr || status_out == nullptr)
    return fail(KDA_ERR_INVALID_ARG, "kda: workspace and status_out are required%s", "");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int32_t v = 0;
  cudaError_t e = cudaMemcpyAsync(&v, workspace, sizeof(v), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: status read failed: %s", cudaGetErrorString(e));
  if (v != 0) {   // a K1 that gave up is the cause of what its K2 reported after it
    int32_t k1 = 0;
    e = cudaMemcpyAsync(&k1, static_cast<const int32_t*>(workspace) + kda::HDR_K1_STATUS, sizeof(k1), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(KDA_ERR_CUDA, "kda: status read failed: %s", cudaGetErrorString(e));
    if (k1 == kda::ST_K1_LOAD_TIMEOUT) v = k1;
  }
  *status_out = v;
  if (v != 0) return fail(KDA_ERR_DEVICE_STATUS, "kda: a bounded device-side wait gave up%s (status %lld)", "", v);
  return KDA_OK;
}

int kda_fwd_k2_choice(const KdaFwdArgs* args, int state_only, int sm_count, int32_t* variant_out, int32_t* vsplit_out) {
  if (args == nullptr || variant_out == nullptr || vsplit_out == nullptr)
    return fail(KDA_ERR_INVALID_ARG, "kda: null pointer%s", "");
  if (args->k2_variant < 0 || args->k2_variant > 5 || args->k2_variant == 2)
    return fail(KDA_ERR_INVALID_ARG, "kda: k2_variant%s %lld is not one of 0, 1, 3, 4, 5", "", static_cast<long long>(args->k2_variant));
  int vs = 0, var = 0;
  pick_split(args, state_only != 0, &vs, &var, sm_count);
  *variant_out = var;
  *vsplit_out = (var == 4) ? 1 : vs;   // the tensor-memory form runs one CTA per chain
  return KDA_OK;
}

int kda_last_launch_count(void) { return g_launches; }

const char* kda_last_error(void) { return g_err; }

const char* kda_version(void) { return "0.1 sm_100a"; }

}  // extern "C"
