// Token-by-token KDA recurrence for decode and short sequences.  sm_100a.
//
// The reference has no decode kernel (its README lists prefill/decode separation as future work,
// README.md:503-505); the arithmetic is the token recurrence its tests use as the gold
// (fused_recurrent_kda at tests/test_kda_bt16.py:26-39), with the rounding points of the chunk
// path (normalised q, k rounded to bf16, everything else fp32), V-first state h[V][K]:
//   h   <- h * 2^gate[k]                       gate = lower_bound * sigmoid(e^A_log (g + bias)) / ln 2
//   v'  =  beta * (v - h khat)
//   h   <- h + v' (x) khat
//   o   =  scale * h qhat
// The output is taken from the decayed state before the update, o = scale * (h qhat + v' (khat . qhat)), so that both
// products of a token with the state go through one reduction.
// Every state row v is independent, so a warp owns ROWS rows of one (batch, head) state and keeps
// them in registers over all T tokens: lane l holds columns 4l..4l+3 of each row (one 16-byte
// load per row), and the 2 x ROWS dot products of a token are reduced over the warp together.  The kernel moves
// 64 KiB of state in and out per (batch, head) and a few hundred bytes per token: HBM bound; the
// grid is (batch x head) x (128 / rows per CTA) CTAs.  A K-first state h[K][V] (the layout
// flash-linear-attention keeps) is read and written in place: for one column k the warp's ROWS
// rows are ROWS consecutive floats, so the lane moves them as 16- or 8-byte pieces (full 32-byte
// sectors at 8 rows per warp) into the same registers; with enough heads two kernels with the lanes along v take
// over (below).
#include "kda_common.cuh"
#include "kda_kernels.h"

namespace kda {

namespace {
constexpr int REC_WARPS = 4;   // warps per CTA

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
  return x;
}

// Sums N per-lane values over the warp at once: each exchange halves the number of values a lane
// still carries (the upper half of the lanes keeps the upper half of the rows), so N values cost
// N - 1 + (5 - log2 N) shuffles instead of 5 N.  Afterwards the lanes l with l >> (5 - log2 N) == r
// hold the total of value r.
template <int N> struct Log2 { static constexpr int v = 1 + Log2<N / 2>::v; };
template <> struct Log2<1> { static constexpr int v = 0; };
template <int N>
__device__ __forceinline__ float warp_sum_rows(float (&p)[N], int lane) {
  constexpr int LG = Log2<N>::v;
#pragma unroll
  for (int lv = 0; lv < LG; ++lv) {
    const int half = N >> (lv + 1), mask = 16 >> lv;
    const bool up = (lane & mask) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = up ? p[i] : p[i + half];
      const float keep = up ? p[i + half] : p[i];
      p[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
    }
  }
  float x = p[0];
#pragma unroll
  for (int lv = LG; lv < 5; ++lv) x += __shfl_xor_sync(0xffffffffu, x, 16 >> lv);
  return x;
}

// Everything of a token that does not depend on the state, worked out once per CTA: for calls of several
// tokens, warp w prepares token w of a group of TOK_GROUP while the state's loads are under way.
constexpr int TOK_GROUP = REC_WARPS;
struct TokenTile {
  float q[TOK_GROUP][D], k[TOK_GROUP][D];   // normalised, rounded to bf16
  float dec[TOK_GROUP][D];                  // 2^gate
  float v[TOK_GROUP][32];                   // of the CTA's state rows
  float beta[TOK_GROUP], qk[TOK_GROUP];     // activated beta; khat . qhat
};
// Lane l of the calling warp: columns 4l .. 4l + 3.  n_v (a multiple of 8, at most 32) rows of v from v_first.
template <bool G_BF16>
__device__ __forceinline__ void prepare_token(const RecurrentParams& p, TokenTile& tile, int slot, int b, int h, int t,
                                              int v_first, int n_v, int lane) {
  auto load4 = [](const __nv_bfloat16* src) {
    const uint2 raw = *reinterpret_cast<const uint2*>(src);
    return make_float4(bf16_lo_to_f32(raw.x), bf16_hi_to_f32(raw.x), bf16_lo_to_f32(raw.y), bf16_hi_to_f32(raw.y));
  };
  const int c0 = lane * 4, hq = h / p.group;   // grouped value heads share a q/k head
  const float4 qr = load4(p.q + b * p.q_s[0] + hq * p.q_s[2] + t * p.q_s[1] + c0);
  const float4 kr = load4(p.k + b * p.k_s[0] + hq * p.k_s[2] + t * p.k_s[1] + c0);
  const uint8_t* gp = static_cast<const uint8_t*>(p.g) + (b * p.g_s[0] + h * p.g_s[2] + t * p.g_s[1] + c0) * (G_BF16 ? 2 : 4);
  const float4 gr = G_BF16 ? load4(reinterpret_cast<const __nv_bfloat16*>(gp)) : *reinterpret_cast<const float4*>(gp);
  float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c0 < n_v) v4 = load4(p.v + b * p.v_s[0] + h * p.v_s[2] + t * p.v_s[1] + v_first + c0);
  const float beta = p.beta[b * p.beta_s[0] + h * p.beta_s[2] + t * p.beta_s[1]];
  const float expA = expf(p.A_log[h]);
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.dt_bias != nullptr) bias = *reinterpret_cast<const float4*>(p.dt_bias + h * D + c0);
  const float lbr = p.lower_bound * RCP_LN2;

  // l2 normalisation, rounded to bf16 like the chunk path
  const float rq = rsqrtf(warp_sum(qr.x * qr.x + qr.y * qr.y + qr.z * qr.z + qr.w * qr.w) + L2NORM_EPS);
  const float rk = rsqrtf(warp_sum(kr.x * kr.x + kr.y * kr.y + kr.z * kr.z + kr.w * kr.w) + L2NORM_EPS);
  const float4 qn = make_float4(bf16_round(qr.x * rq), bf16_round(qr.y * rq), bf16_round(qr.z * rq), bf16_round(qr.w * rq));
  const float4 kn = make_float4(bf16_round(kr.x * rk), bf16_round(kr.y * rk), bf16_round(kr.z * rk), bf16_round(kr.w * rk));
  const float qk = warp_sum(qn.x * kn.x + qn.y * kn.y + qn.z * kn.z + qn.w * kn.w);
  // decay 2^(lb * sigmoid(e^A (g + bias)) / ln 2)
  auto dec1 = [&](float g, float bi) {
    const float z = expA * (g + bi);
    return ex2f(lbr / (1.0f + __expf(-z)));
  };
  *reinterpret_cast<float4*>(&tile.q[slot][c0]) = qn;
  *reinterpret_cast<float4*>(&tile.k[slot][c0]) = kn;
  *reinterpret_cast<float4*>(&tile.dec[slot][c0]) = make_float4(dec1(gr.x, bias.x), dec1(gr.y, bias.y), dec1(gr.z, bias.z), dec1(gr.w, bias.w));
  if (c0 < n_v) *reinterpret_cast<float4*>(&tile.v[slot][c0]) = v4;
  if (lane == 0) {
    tile.beta[slot] = 1.0f / (1.0f + __expf(-beta));
    tile.qk[slot] = qk;
  }
}

// ONE: a call of one token, every warp on its own.  Otherwise any number of tokens, in groups prepared
// once per CTA.  The state passes through once per call and is larger than what the caches should keep for
// it: its loads and stores carry the evict-first hint.  Measured on B200 (H32, V-first), before -> now:
//   T1 B64 48.2 -> 41.8 us (6.4 TB/s; 46.2 without the hint), B8 10.7 -> 7.8, B4 6.3 -> 5.2, B1 3.1 -> 2.8: bound by
//   the state's traffic from B8 on, below by latency;
//   T4 B16 30.0 -> 19.8, B8 19.5 -> 11.4, B1 6.2 -> 4.4, T2 B64 64.5 -> 50.5 (each warp prepared every token and
//   reduced twice before): bound by the tokens' serial chain.  Six CTAs per SM; without that bound the
//   registers allow four and T4 B16 takes 24.3.
template <int ROWS, bool G_BF16, bool ONE>
__global__ void __launch_bounds__(REC_WARPS * 32, 6) kda_recurrent_kernel(const RecurrentParams p) {
  constexpr int ROWS_PER_CTA = ROWS * REC_WARPS;
  constexpr int SLICES = D / ROWS_PER_CTA;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bh = blockIdx.x / SLICES, slice = blockIdx.x % SLICES;
  const int b = bh / p.H, h = bh % p.H;
  const int v0 = slice * ROWS_PER_CTA + warp * ROWS;   // first state row of this warp
  const int k0 = lane * 4;                             // first state column of this lane
  constexpr int SH = 4 - Log2<ROWS>::v;                // lanes that end up with one sum of a token: 1 << SH

  // Launched ahead of the end of whatever runs before it in the stream; nothing of global memory is touched before this.  It
  // does not let the next kernel start in turn: one that starts with this one's last wave, or behind its loads, and not at its end
  // takes places that this one's loads could use (in place of 42.3 us 43.9 and 44.5, B64 H32).
  grid_dep_wait();
  float4 s[ROWS];
  constexpr int PIECE = (ROWS % 4 == 0) ? 4 : 2;   // floats per access along v in the K-first layout
  if (p.h0 != nullptr && p.k_first) {
    const float* h0 = p.h0 + (static_cast<size_t>(bh) * D + k0) * D + v0;   // element (k0 + c, v0 + r) at c * D + r
    float t[4][ROWS];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < ROWS; r += PIECE) {
        if (PIECE == 4) {
          const float4 x = *reinterpret_cast<const float4*>(h0 + c * D + r);
          t[c][r] = x.x; t[c][r + 1] = x.y; t[c][r + 2] = x.z; t[c][r + 3] = x.w;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(h0 + c * D + r);
          t[c][r] = x.x; t[c][r + 1] = x.y;
        }
      }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) s[r] = make_float4(t[0][r], t[1][r], t[2][r], t[3][r]);
  } else if (p.h0 != nullptr) {
    const float* h0 = p.h0 + (static_cast<size_t>(bh) * D + v0) * D + k0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) s[r] = __ldcs(reinterpret_cast<const float4*>(h0 + r * D));
  } else {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) s[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  __nv_bfloat16* op = p.o + b * p.o_s[0] + h * p.o_s[2] + v0;
  // One token on the state.  With the decayed h, both h khat and h qhat are taken before the update: the
  // output of the updated state is h qhat + v' (khat . qhat).  All 2 x ROWS sums go through one reduction;
  // afterwards the lower half of the warp holds the predictions (lane >> SH == row), the upper half h qhat.
  // vmine: v of row (lane & 15) >> SH.
  auto advance = [&](const float4& qn, const float4& kn, const float4& dc, float qk, float beta, float vmine, int t) {
    float part[2 * ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      s[r].x *= dc.x; s[r].y *= dc.y; s[r].z *= dc.z; s[r].w *= dc.w;
      part[r] = s[r].x * kn.x + s[r].y * kn.y + s[r].z * kn.z + s[r].w * kn.w;
      part[ROWS + r] = s[r].x * qn.x + s[r].y * qn.y + s[r].z * qn.z + s[r].w * qn.w;
    }
    const float sum = warp_sum_rows<2 * ROWS>(part, lane);
    const float vn_mine = beta * (vmine - sum);           // lower half: v' of row lane >> SH
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const float vn = __shfl_sync(0xffffffffu, vn_mine, r << SH);
      s[r].x = fmaf(vn, kn.x, s[r].x); s[r].y = fmaf(vn, kn.y, s[r].y);
      s[r].z = fmaf(vn, kn.z, s[r].z); s[r].w = fmaf(vn, kn.w, s[r].w);
    }
    const float od = fmaf(__shfl_xor_sync(0xffffffffu, vn_mine, 16), qk, sum);   // upper half: o of row (lane - 16) >> SH
    if (lane >= 16 && (lane & ((1 << SH) - 1)) == 0) op[t * p.o_s[1] + ((lane - 16) >> SH)] = __float2bfloat16(p.scale * od);
  };
  const int my_row = (lane & 15) >> SH;

  if constexpr (ONE) {
    const float expA = expf(p.A_log[h]);
    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.dt_bias != nullptr) bias = *reinterpret_cast<const float4*>(p.dt_bias + h * D + k0);
    const float lbr = p.lower_bound * RCP_LN2;
    auto load4 = [](const __nv_bfloat16* src) {
      const uint2 raw = *reinterpret_cast<const uint2*>(src);
      return make_float4(bf16_lo_to_f32(raw.x), bf16_hi_to_f32(raw.x), bf16_lo_to_f32(raw.y), bf16_hi_to_f32(raw.y));
    };
    const int hq = h / p.group;   // grouped value heads share a q/k head
    const float4 qr = load4(p.q + b * p.q_s[0] + hq * p.q_s[2] + k0);
    const float4 kr = load4(p.k + b * p.k_s[0] + hq * p.k_s[2] + k0);
    const uint8_t* gp = static_cast<const uint8_t*>(p.g) + (b * p.g_s[0] + h * p.g_s[2] + k0) * (G_BF16 ? 2 : 4);
    const float4 gr = G_BF16 ? load4(reinterpret_cast<const __nv_bfloat16*>(gp)) : *reinterpret_cast<const float4*>(gp);
    const float vmine = __bfloat162float(p.v[b * p.v_s[0] + h * p.v_s[2] + v0 + my_row]);
    const float beta = 1.0f / (1.0f + __expf(-p.beta[b * p.beta_s[0] + h * p.beta_s[2]]));
    // l2 normalisation, rounded to bf16 like the chunk path
    const float rq = rsqrtf(warp_sum(qr.x * qr.x + qr.y * qr.y + qr.z * qr.z + qr.w * qr.w) + L2NORM_EPS);
    const float rk = rsqrtf(warp_sum(kr.x * kr.x + kr.y * kr.y + kr.z * kr.z + kr.w * kr.w) + L2NORM_EPS);
    const float4 qn = make_float4(bf16_round(qr.x * rq), bf16_round(qr.y * rq), bf16_round(qr.z * rq), bf16_round(qr.w * rq));
    const float4 kn = make_float4(bf16_round(kr.x * rk), bf16_round(kr.y * rk), bf16_round(kr.z * rk), bf16_round(kr.w * rk));
    // decay 2^(lb * sigmoid(e^A (g + bias)) / ln 2) of this lane's four columns
    auto dec1 = [&](float g, float bi) {
      const float z = expA * (g + bi);
      return ex2f(lbr / (1.0f + __expf(-z)));
    };
    const float4 dc = make_float4(dec1(gr.x, bias.x), dec1(gr.y, bias.y), dec1(gr.z, bias.z), dec1(gr.w, bias.w));
    advance(qn, kn, dc, warp_sum(qn.x * kn.x + qn.y * kn.y + qn.z * kn.z + qn.w * kn.w), beta, vmine, 0);
  } else {
    __shared__ TokenTile tile;
    for (int t0 = 0; t0 < p.T; t0 += TOK_GROUP) {
      if (t0 > 0) __syncthreads();   // the previous group's slots have been read
      if (t0 + warp < p.T) prepare_token<G_BF16>(p, tile, warp, b, h, t0 + warp, slice * ROWS_PER_CTA, ROWS_PER_CTA, lane);
      __syncthreads();
      const int nt = min(TOK_GROUP, p.T - t0);
      for (int i = 0; i < nt; ++i)
        advance(*reinterpret_cast<const float4*>(&tile.q[i][k0]), *reinterpret_cast<const float4*>(&tile.k[i][k0]),
                *reinterpret_cast<const float4*>(&tile.dec[i][k0]), tile.qk[i], tile.beta[i], tile.v[i][warp * ROWS + my_row], t0 + i);
    }
  }

  if (p.ht != nullptr && p.k_first) {
    float* ht = p.ht + (static_cast<size_t>(bh) * D + k0) * D + v0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < ROWS; r += PIECE) {
        auto comp = [&](int rr) { return c == 0 ? s[rr].x : (c == 1 ? s[rr].y : (c == 2 ? s[rr].z : s[rr].w)); };
        if (PIECE == 4) *reinterpret_cast<float4*>(ht + c * D + r) = make_float4(comp(r), comp(r + 1), comp(r + 2), comp(r + 3));
        else *reinterpret_cast<float2*>(ht + c * D + r) = make_float2(comp(r), comp(r + 1));
      }
  } else if (p.ht != nullptr) {
    float* ht = p.ht + (static_cast<size_t>(bh) * D + v0) * D + k0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) __stcs(reinterpret_cast<float4*>(ht + r * D), s[r]);
  }
}

// K-first state h[K][V] with enough heads to fill the GPU: lanes along v.
// A CTA owns all 128 k of a 32-wide slice of v (one full 128-byte line per k); thread (vq = tid % 8,
// kg = tid / 8) keeps rows k = 8 kg .. 8 kg + 7 of columns v = 4 vq .. 4 vq + 3 of that slice in
// registers (eight 16-byte accesses, four whole lines per warp instruction -- the access pattern of
// the V-first kernel above on the transposed state).
// A call of several tokens takes them in groups prepared once per CTA.  What remains serial per token is the
// two products with the state, which go through ONE reduction (as in the kernel above): six shuffles over the
// four k-groups of a warp and an exchange through shared memory over the warps, double-buffered, so one CTA
// barrier per token.  Same arithmetic and rounding points as the kernel above; the fp32 sums run in another
// order.  Measured on B200 (H32, T4) against every warp preparing every token and two reductions per token:
// B16 32.9 -> 20.9 us, B64 110.8 -> 65.4; B64 T2 68.9 -> 49.4.  Bound by the tokens' serial chain; seven CTAs
// per SM (72 registers) cover most of it: five take 25.4 us at B16, eight spill (22.7).
template <bool G_BF16>
__global__ void __launch_bounds__(128, 7) kda_recurrent_kfirst_kernel(const RecurrentParams p) {
  __shared__ TokenTile tile;
  __shared__ float red[2][4][2][32];   // [token parity][warp][h khat | h qhat][v]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int vq = tid & 7, kg = tid >> 3;
  const int bh = blockIdx.x >> 2, slice = blockIdx.x & 3;
  const int b = bh / p.H, h = bh % p.H;
  const int v0 = slice * 32 + vq * 4;   // first state column of this thread
  const int k0 = kg * 8;                // first state row of this thread

  grid_dep_wait();
  float4 s[8];
  if (p.h0 != nullptr) {
    const float* h0 = p.h0 + (static_cast<size_t>(bh) * D + k0) * D + v0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = __ldcs(reinterpret_cast<const float4*>(h0 + i * D));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  __nv_bfloat16* op = p.o + b * p.o_s[0] + h * p.o_s[2] + v0;
  for (int t0 = 0; t0 < p.T; t0 += TOK_GROUP) {
    // the previous group's slots are free: every thread read them before its last token's barrier
    if (t0 + warp < p.T) prepare_token<G_BF16>(p, tile, warp, b, h, t0 + warp, slice * 32, 32, lane);
    __syncthreads();
    const int nt = min(TOK_GROUP, p.T - t0);
    for (int i = 0; i < nt; ++i) {
      float kn[8], pk[4] = {0.f, 0.f, 0.f, 0.f}, pq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(&tile.k[i][k0 + j]);
        const float4 q4 = *reinterpret_cast<const float4*>(&tile.q[i][k0 + j]);
        const float4 d4 = *reinterpret_cast<const float4*>(&tile.dec[i][k0 + j]);
        const float qv[4] = {q4.x, q4.y, q4.z, q4.w}, dv[4] = {d4.x, d4.y, d4.z, d4.w};
        kn[j] = k4.x; kn[j + 1] = k4.y; kn[j + 2] = k4.z; kn[j + 3] = k4.w;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float4& r = s[j + jj];
          r.x *= dv[jj]; r.y *= dv[jj]; r.z *= dv[jj]; r.w *= dv[jj];
          pk[0] = fmaf(r.x, kn[j + jj], pk[0]); pk[1] = fmaf(r.y, kn[j + jj], pk[1]);
          pk[2] = fmaf(r.z, kn[j + jj], pk[2]); pk[3] = fmaf(r.w, kn[j + jj], pk[3]);
          pq[0] = fmaf(r.x, qv[jj], pq[0]); pq[1] = fmaf(r.y, qv[jj], pq[1]);
          pq[2] = fmaf(r.z, qv[jj], pq[2]); pq[3] = fmaf(r.w, qv[jj], pq[3]);
        }
      }
      // over the four k-groups of the warp: the upper half keeps h qhat, then odd groups the columns 2, 3
      const bool up = (lane & 16) != 0, odd = (lane & 8) != 0;
      float m[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) m[e] = (up ? pq[e] : pk[e]) + __shfl_xor_sync(0xffffffffu, up ? pk[e] : pq[e], 16);
      float2 y;
      y.x = (odd ? m[2] : m[0]) + __shfl_xor_sync(0xffffffffu, odd ? m[0] : m[2], 8);
      y.y = (odd ? m[3] : m[1]) + __shfl_xor_sync(0xffffffffu, odd ? m[1] : m[3], 8);
      float (*buf)[2][32] = red[i & 1];   // TOK_GROUP is even: the parity goes on across groups
      *reinterpret_cast<float2*>(&buf[warp][up ? 1 : 0][vq * 4 + (odd ? 2 : 0)]) = y;
      const float4 v4 = *reinterpret_cast<const float4*>(&tile.v[i][vq * 4]);
      const float beta = tile.beta[i], qk = tile.qk[i];
      __syncthreads();
      auto total = [&](int which) {
        const float4 a = *reinterpret_cast<const float4*>(&buf[0][which][vq * 4]), c = *reinterpret_cast<const float4*>(&buf[1][which][vq * 4]);
        const float4 d = *reinterpret_cast<const float4*>(&buf[2][which][vq * 4]), e = *reinterpret_cast<const float4*>(&buf[3][which][vq * 4]);
        return make_float4((a.x + c.x) + (d.x + e.x), (a.y + c.y) + (d.y + e.y), (a.z + c.z) + (d.z + e.z), (a.w + c.w) + (d.w + e.w));
      };
      const float4 pred = total(0);
      const float4 vn = make_float4(beta * (v4.x - pred.x), beta * (v4.y - pred.y), beta * (v4.z - pred.z), beta * (v4.w - pred.w));
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s[j].x = fmaf(vn.x, kn[j], s[j].x); s[j].y = fmaf(vn.y, kn[j], s[j].y);
        s[j].z = fmaf(vn.z, kn[j], s[j].z); s[j].w = fmaf(vn.w, kn[j], s[j].w);
      }
      if (tid < 8) {
        const float4 hq4 = total(1);
        uint2 out;
        out.x = pack_bf16(p.scale * fmaf(vn.x, qk, hq4.x), p.scale * fmaf(vn.y, qk, hq4.y));
        out.y = pack_bf16(p.scale * fmaf(vn.z, qk, hq4.z), p.scale * fmaf(vn.w, qk, hq4.w));
        *reinterpret_cast<uint2*>(op + (t0 + i) * p.o_s[1]) = out;
      }
    }
  }

  if (p.ht != nullptr) {
    float* ht = p.ht + (static_cast<size_t>(bh) * D + k0) * D + v0;
#pragma unroll
    for (int i = 0; i < 8; ++i) __stcs(reinterpret_cast<float4*>(ht + i * D), s[i]);
  }
}

// One token: every warp prepares it for itself, so that nothing stands between the state's loads and the first
// product; two reductions through shared memory (one for both takes more registers: B64 H32 51.0 us against
// 46.6).  The state's traffic bounds it, and the CTAs per SM that cover its latency.  Every bound on the registers below 96
// (five CTAs) spills a few of a thread's own inputs: seven CTAs (72 registers) 68 bytes with a bf16 gate, 84 with an fp32
// gate, six (80 registers) 56 and 64.  Steps in a graph, H32, states beyond L2, B8 / B64 / B256, no hint and no bound first:
//   bf16 gate 10.9 / 49.8 / 179 us; now 8.4 / 45.8 / 169 with seven, 9.3 / 48.3 / 193 with six, 9.1 / 46.0 / 173 with five;
//   fp32 gate 10.9 / 50.5 / 181 us; now 8.9 / 49.2 / 191 with seven, 8.8 / 45.9 / 172-178 with six, 9.1 / 46.0 / 174 with five.
template <bool G_BF16>
__global__ void __launch_bounds__(128, G_BF16 ? 7 : 6) kda_recurrent_kfirst_one_kernel(const RecurrentParams p) {
  __shared__ float4 red[2][4][8];   // [prediction | output][warp][v quad]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int vq = tid & 7, kg = tid >> 3;
  const int bh = blockIdx.x >> 2, slice = blockIdx.x & 3;
  const int b = bh / p.H, h = bh % p.H;
  const int v0 = slice * 32 + vq * 4;   // first state column of this thread
  const int k0 = kg * 8;                // first state row of this thread

  grid_dep_wait();
  float4 s[8];
  if (p.h0 != nullptr) {
    const float* h0 = p.h0 + (static_cast<size_t>(bh) * D + k0) * D + v0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = __ldcs(reinterpret_cast<const float4*>(h0 + i * D));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  const float expA = expf(p.A_log[h]);
  float bias[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) bias[i] = (p.dt_bias != nullptr) ? p.dt_bias[h * D + k0 + i] : 0.f;
  const float lbr = p.lower_bound * RCP_LN2;

  const int hq = h / p.group;   // grouped value heads share a q/k head
  const __nv_bfloat16* qp = p.q + b * p.q_s[0] + hq * p.q_s[2];
  const __nv_bfloat16* kp = p.k + b * p.k_s[0] + hq * p.k_s[2];
  const __nv_bfloat16* vp = p.v + b * p.v_s[0] + h * p.v_s[2] + v0;
  const uint8_t* gp = static_cast<const uint8_t*>(p.g) + (b * p.g_s[0] + h * p.g_s[2] + k0) * (G_BF16 ? 2 : 4);
  const float* bp = p.beta + b * p.beta_s[0] + h * p.beta_s[2];
  __nv_bfloat16* op = p.o + b * p.o_s[0] + h * p.o_s[2] + v0;

  auto load4 = [](const __nv_bfloat16* src) {
    const uint2 raw = *reinterpret_cast<const uint2*>(src);
    return make_float4(bf16_lo_to_f32(raw.x), bf16_hi_to_f32(raw.x), bf16_lo_to_f32(raw.y), bf16_hi_to_f32(raw.y));
  };
  auto load8 = [](const __nv_bfloat16* src, float (&x)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(src);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { x[2 * i] = bf16_lo_to_f32(w[i]); x[2 * i + 1] = bf16_hi_to_f32(w[i]); }
  };
  // sum over the k-groups of this warp (lanes with the same vq), then over the warps
  auto reduce_k = [&](float4 x, int which) {
#pragma unroll
    for (int m = 8; m <= 16; m <<= 1) {
      x.x += __shfl_xor_sync(0xffffffffu, x.x, m); x.y += __shfl_xor_sync(0xffffffffu, x.y, m);
      x.z += __shfl_xor_sync(0xffffffffu, x.z, m); x.w += __shfl_xor_sync(0xffffffffu, x.w, m);
    }
    if (lane < 8) red[which][warp][vq] = x;
    __syncthreads();
    const float4 a = red[which][0][vq], c = red[which][1][vq], d = red[which][2][vq], e = red[which][3][vq];
    return make_float4((a.x + c.x) + (d.x + e.x), (a.y + c.y) + (d.y + e.y), (a.z + c.z) + (d.z + e.z), (a.w + c.w) + (d.w + e.w));
  };

  {
    constexpr int t = 0;
    // l2 norms over all 128 k: every warp computes them (lane l: k = 4 l .. 4 l + 3), rounded to bf16 like the chunk path
    const float4 qa = load4(qp + t * p.q_s[1] + lane * 4);
    const float4 ka = load4(kp + t * p.k_s[1] + lane * 4);
    const float rq = rsqrtf(warp_sum(qa.x * qa.x + qa.y * qa.y + qa.z * qa.z + qa.w * qa.w) + L2NORM_EPS);
    const float rk = rsqrtf(warp_sum(ka.x * ka.x + ka.y * ka.y + ka.z * ka.z + ka.w * ka.w) + L2NORM_EPS);
    float qn[8], kn[8], gr[8];
    load8(qp + t * p.q_s[1] + k0, qn);
    load8(kp + t * p.k_s[1] + k0, kn);
    if (G_BF16) load8(reinterpret_cast<const __nv_bfloat16*>(gp + t * p.g_s[1] * 2), gr);
    else {
      const float4 g0 = *reinterpret_cast<const float4*>(gp + t * p.g_s[1] * 4);
      const float4 g1 = *reinterpret_cast<const float4*>(gp + t * p.g_s[1] * 4 + 16);
      gr[0] = g0.x; gr[1] = g0.y; gr[2] = g0.z; gr[3] = g0.w; gr[4] = g1.x; gr[5] = g1.y; gr[6] = g1.z; gr[7] = g1.w;
    }
    const float4 v4 = load4(vp + t * p.v_s[1]);
    float beta = bp[t * p.beta_s[1]];
    beta = 1.0f / (1.0f + __expf(-beta));

    float4 part = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      qn[i] = bf16_round(qn[i] * rq);
      kn[i] = bf16_round(kn[i] * rk);
      // decay 2^(lb * sigmoid(e^A (g + bias)) / ln 2) of row k0 + i
      const float z = expA * (gr[i] + bias[i]);
      const float dc = ex2f(lbr / (1.0f + __expf(-z)));
      s[i].x *= dc; s[i].y *= dc; s[i].z *= dc; s[i].w *= dc;
      part.x = fmaf(s[i].x, kn[i], part.x); part.y = fmaf(s[i].y, kn[i], part.y);
      part.z = fmaf(s[i].z, kn[i], part.z); part.w = fmaf(s[i].w, kn[i], part.w);
    }
    const float4 pred = reduce_k(part, 0);
    const float4 vn = make_float4(beta * (v4.x - pred.x), beta * (v4.y - pred.y), beta * (v4.z - pred.z), beta * (v4.w - pred.w));
    part = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      s[i].x = fmaf(vn.x, kn[i], s[i].x); s[i].y = fmaf(vn.y, kn[i], s[i].y);
      s[i].z = fmaf(vn.z, kn[i], s[i].z); s[i].w = fmaf(vn.w, kn[i], s[i].w);
      part.x = fmaf(s[i].x, qn[i], part.x); part.y = fmaf(s[i].y, qn[i], part.y);
      part.z = fmaf(s[i].z, qn[i], part.z); part.w = fmaf(s[i].w, qn[i], part.w);
    }
    const float4 od = reduce_k(part, 1);
    if (tid < 8) {
      uint2 out;
      out.x = pack_bf16(p.scale * od.x, p.scale * od.y);
      out.y = pack_bf16(p.scale * od.z, p.scale * od.w);
      *reinterpret_cast<uint2*>(op + t * p.o_s[1]) = out;
    }
  }

  if (p.ht != nullptr) {
    float* ht = p.ht + (static_cast<size_t>(bh) * D + k0) * D + v0;
#pragma unroll
    for (int i = 0; i < 8; ++i) __stcs(reinterpret_cast<float4*>(ht + i * D), s[i]);
  }
}

template <int ROWS>
cudaError_t launch_rows(const RecurrentParams& p, bool g_bf16, cudaStream_t stream) {
  const int grid = p.B * p.H * (D / (ROWS * REC_WARPS));
  if (p.T == 1)
    return g_bf16 ? launch_dep(kda_recurrent_kernel<ROWS, true, true>, grid, REC_WARPS * 32, 0, stream, 1, p)
                  : launch_dep(kda_recurrent_kernel<ROWS, false, true>, grid, REC_WARPS * 32, 0, stream, 1, p);
  return g_bf16 ? launch_dep(kda_recurrent_kernel<ROWS, true, false>, grid, REC_WARPS * 32, 0, stream, 1, p)
                : launch_dep(kda_recurrent_kernel<ROWS, false, false>, grid, REC_WARPS * 32, 0, stream, 1, p);
}
}  // namespace

// rows per warp: 8 (four CTAs per head) once there are enough heads to fill the GPU, else 2
// (sixteen CTAs per head) so that a handful of heads still spreads over many SMs
cudaError_t launch_recurrent(const RecurrentParams& p, bool g_bf16, int sms, cudaStream_t stream) {
  const long long bh = static_cast<long long>(p.B) * p.H;
  if (p.k_first && bh * 4 >= 2LL * sms) {
    // four CTAs per head with the lanes along v; with fewer heads the calls are latency-bound and the
    // row-per-warp kernel's strided state accesses cost nothing measurable
    const int grid = static_cast<int>(bh) * 4;
    if (p.T == 1)
      return g_bf16 ? launch_dep(kda_recurrent_kfirst_one_kernel<true>, grid, 128, 0, stream, 1, p)
                    : launch_dep(kda_recurrent_kfirst_one_kernel<false>, grid, 128, 0, stream, 1, p);
    return g_bf16 ? launch_dep(kda_recurrent_kfirst_kernel<true>, grid, 128, 0, stream, 1, p)
                  : launch_dep(kda_recurrent_kfirst_kernel<false>, grid, 128, 0, stream, 1, p);
  }
  if (bh * 4 >= 2LL * sms) return launch_rows<8>(p, g_bf16, stream);
  if (bh * 8 >= 2LL * sms) return launch_rows<4>(p, g_bf16, stream);
  return launch_rows<2>(p, g_bf16, stream);
}

}  // namespace kda
