// K1: intra-chunk stage of the KDA forward.  Persistent CTAs of 128 threads, each walking
// (batch, head, chunk-of-16-tokens) work items with the next chunk's inputs in flight while
// the current one computes.  sm_100a.
//
// Replaces kda_bt16_kernel_k1 of the reference (src/kda_bt16/kernels.py:53-184) and
// follows the arithmetic and rounding points of the reference's torch chunk
// implementation (tests/test_torch_reference.py:77-173):
//   1. gate pre-pass: beta sigmoid, q/k l2-norm (eps 1e-6, result rounded to bf16),
//      gate = lower_bound*sigmoid(exp(A_log)*(g+dt_bias))*RCP_LN2, chunk-local cumsum
//   2. Aqk = scale*tril((qhat 2^gm)(khat 2^-gm)^T), Akk = tril_-1((khat 2^gm)(khat 2^-gm)^T)*beta_i
//      with gm = g - g[centre]; tensor-core MMAs on hi/lo bf16 splits of the fp32 operands
//      (three partial products, fp32 accumulate => ~2^-16 relative, "fp32-like")
//   3. X = (I + Akk)^-1 by forward substitution, fp32, one lane per column of X
//   4. w = X (khat beta 2^g)   (bf16 out);   u = X diag(beta) v is left to K2 as its two factors: X diag(beta) as a
//      hi/lo bf16 pair, and v as it came
// and additionally pre-computes what the reference's Triton K2 re-derives every step
// (src/kda_bt16/kernels.py:255-259,271,286-287): qg = bf16(qhat 2^g),
// kg = khat 2^(g_last-g) as a hi/lo bf16 pair, dec = 2^g_last -- the arrangement of
// the reference's Ascend pipeline (python/kda_ascendc_v1/api.py:890-897).
//
// Data movement: the 16x128 input tiles arrive by tiled TMA copies (4-D tensor maps over
// (d, head, token, batch) built from the caller's strides, so head-shard and segment views
// need no copy; rows past T are zero-filled by the copy).  Those of q, k and g complete on one mbarrier; as soon as
// a chunk's have been consumed the copies of the CTA's next chunk are issued into the
// same tiles, so the ~2.5 us load latency hides behind the rest of the chunk.  v is only passed on (of packed sequences, with the
// rows behind a sequence's end cleared): its two 64-column boxes, with a barrier of their own, arrive, swizzled by the copy, where
// the record's part with kg, Aqk, dec, Xb and v is put together.  They are asked for within their own item, once the stores of the
// item before have left that place (the first item's at once with the rest: T100 H32 11.3 -> 11.5 us), and waited for two phases
// later.  That part, qg and w leave by five bulk stores.  With u worked out here and stored as fp32 from the accumulator fragments K1 alone took 147.5 us, now
// 132.7 (T8192 H32; H96 426 -> 383, in a row of calls at the power limit 468 -> 410; the prepared batch 276 -> 257).
// khat beta 2^g is rounded to bf16 with beta in it, as ever: without, where gates are near zero khat 2^g rounds back to
// khat more often than not, and the state's error against 64 bits grows by 1 % (gates of -8: 1.283e-3 -> 1.298e-3).
#include "kda_common.cuh"
#include "kda_kernels.h"

namespace kda {

// shared-memory map (bytes): four CTAs of the production variant (bf16 gate, FAST_EXP) per SM
constexpr int S_QG = 0;                               // two halves of 2048 bytes -> the record's qg parts
// as in the record from REC_KGH on (kg, Aqk, dec, Xb, dec again, v): one bulk store
constexpr int S_KGH = 4096, S_KGL = S_KGH + (REC_KGL - REC_KGH);
constexpr int S_AQK = S_KGH + (REC_AQK - REC_KGH), S_AQL = S_KGH + (REC_AQL - REC_KGH), S_DEC = S_KGH + (REC_DEC - REC_KGH);
constexpr int S_XBH = S_KGH + (REC_XBH - REC_KGH), S_XBL = S_KGH + (REC_XBL - REC_KGH), S_DEC2 = S_KGH + (REC_DEC2 - REC_KGH);
constexpr int S_V = S_KGH + (REC_V - REC_KGH);
static_assert(S_V % 1024 == 0, "the copies of v swizzle within 1024 bytes");
constexpr int S_L = S_KGH + (REC_USED_BYTES - REC_KGH);   // fp32 [16][16], -Akk
constexpr int S_XH = S_L, S_XL = S_L + (REC_XBL - REC_XBH);   // bf16 hi / lo of (I+Akk)^-1 in the layout of Xb, over -Akk
constexpr int S_GRAM = S_L + 1024;
constexpr int S_QGH = S_GRAM, S_QGL = S_GRAM + 4096, S_KQH = S_GRAM + 8192, S_KQL = S_GRAM + 12288,
              S_KNH = S_GRAM + 16384, S_KNL = S_GRAM + 20480;   // KN tiles only without FAST_EXP
// once the Grams are done their A tiles hold the B operand of w
constexpr int S_KBH = S_GRAM;
constexpr int S_WST = S_GRAM + 12288;   // staging tile of w (the fourth Gram tile slot), -> the record's w parts

// element (r, c) of a staged w or qg tile: the record's layout with the two halves back to back
__device__ __forceinline__ uint32_t stage_off(int r, int c) {
  return wq_off(r, c) - static_cast<uint32_t>((c >> 6) * (REC_HALF - TILE_BYTES / 2));
}

template <bool G_BF16, bool FAST_EXP>
struct K1Smem {
  static constexpr int IN = S_GRAM + (FAST_EXP ? 16384 : 24576);
  static constexpr int Q = IN, K = IN + 4096, G = IN + 8192;
  static constexpr int G_BYTES = G_BF16 ? 4096 : 8192;
  static constexpr int SMALL = G + G_BYTES;
  static constexpr int BETA = SMALL;          // fp32 [2][16] activated beta + [2] exp(A_log): this item / next item
  static constexpr int TOT = BETA + 144;      // fp32 [2][128]: column sums of the gate over rows 0..7 and rows 8..15
  static constexpr int GMID = TOT + 1024;     // fp32 [128] g[mid] (not needed with FAST_EXP)
  static constexpr int MBAR = GMID + (FAST_EXP ? 0 : 512);
  static constexpr int MBAR_V = MBAR + 8;
  static constexpr int FLAG = MBAR_V + 8;   // a wait gave up; the item after the next one (beside K2)
  static constexpr int TOTAL = FLAG + 8;
};

struct K1Item {   // one (batch, head, chunk) work item
  int b, h, hq, t0, nvalid;   // hq: the q/k head this (value) head reads
  int win;                    // window the item counts towards (0 unless K2 runs beside K1)
  size_t rec_idx;
};

template <bool BESIDE>
__device__ __forceinline__ K1Item k1_item(const K1Params& p, int id) {
  // id -> (b, n, h) with h fastest: CTAs that run together read one contiguous span of tokens.
  // With K2 beside K1 the order is (n, b, h): every chain's next chunk is finished before any chain's
  // later one.
  K1Item w;
  w.win = BESIDE ? static_cast<int>(p.div_win.div(id)) : 0;
  const int bn = static_cast<int>(p.div_h.div(id));
  w.h = id - bn * p.H;
  w.hq = static_cast<int>(p.div_g.div(w.h));
  if (p.chunk_table != nullptr) {   // packed sequences: the chunk's place comes from the table
    const int4 e = __ldg(p.chunk_table + bn);
    w.b = 0;
    w.t0 = e.x;
    w.nvalid = e.y;
    w.rec_idx = static_cast<size_t>(e.z) + static_cast<size_t>(w.h) * e.w;
    return w;
  }
  int n;
  if (BESIDE) {
    n = static_cast<int>(p.div_b.div(bn));
    w.b = bn - n * p.B;
  } else {
    w.b = static_cast<int>(p.div_nt.div(bn));
    n = bn - w.b * p.NT;
  }
  w.t0 = n * BT;
  w.nvalid = min(BT, p.T - w.t0);
  w.rec_idx = (static_cast<size_t>(w.b) * p.H + w.h) * p.NT + n;
  return w;
}

// BESIDE: K2 runs beside this kernel (time-major items, finished items counted per window).  Registers: four CTAs per
// SM need 128 a thread or fewer.  Beside K2, two CTAs share every SM sub-partition's 16,384 registers with up to three
// warps of the tensor-memory K2 (96 a thread): 2 x 32 x 112 + 3 x 32 x 96 is all of them, and with more K2 does not
// start before K1 ends.  kda_fwd, with 128 registers and with 112: T2048 H80 262 and 172 us, T1024 H120 173 and 120.
// Beside the other forms, and a tensor-memory K2 on SMs of its own, either fits: T32768 H16 871 and 872, B2 T4096 H8 119.9 and
// 120.2, T8192 H32 326 and 325, H96 623 and 628, H24 302 and 308.
// FORM: what is known when the kernel is compiled.  FORM_ALL: gate, l2-norm and beta sigmoid in the kernel, dt_bias at an 8-byte
// boundary; FORM_NONE: all three done by the caller (then FAST_EXP is false); neither with debug outputs.  FORM_ANY: the flags
// decide.  Against FORM_ANY for the same call, with u still worked out here: K1 alone T8192 H32 156.4 -> 147.8 us, H96 445 -> 427, inputs
// prepared by the caller (B8 T2037 H32 with 8 q/k heads) 294 -> 274.
enum K1Form { FORM_ANY, FORM_ALL, FORM_NONE };

// Beside K2 the work is handed out item by item, and not every SM does the same share of it: on k2_sms of the SMs (spread
// evenly) only the first k2_sm_ctas CTAs of this kernel stay, and K2's CTAs, which find no room on the others, are placed
// there.  The first ones, by the warp slots they run in, so that the registers and the shared memory that become free lie together:
// with two other CTAs staying (as they came) a tensor-memory K2 found no room on some SMs until K1 ended (T8192 H96
// 720 -> 1,200 us).  Those that leave wait until the whole grid has started, so that no later CTA takes their place,
// and stay too where that takes longer than 20 us, or where fewer than half of those that should stay do so (another stream's
// kernels hold the first warp slots): all this decides about speed only, whoever stays takes items until none is left.
__device__ __forceinline__ bool k1_stays(const K1Params& p) {
  uint32_t sm, slot;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
  asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
  int* arrived = p.progress - HDR_PROGRESS + HDR_ARRIVED;
  const bool stays = sm >= static_cast<uint32_t>(p.n_sms) || (sm * p.k2_sms) % p.n_sms >= static_cast<uint32_t>(p.k2_sms) ||
                     slot < static_cast<uint32_t>(4 * p.k2_sm_ctas);
  constexpr int STAYS = 1 << 16;   // started CTAs in the lower half of the word (a grid is below 65,536), staying ones above
  atomicAdd(arrived, stays ? STAYS + 1 : 1);
  if (stays) return true;
  const unsigned long long t0 = globaltimer_ns();
  do {
    int n;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(n) : "l"(arrived) : "memory");
    if ((n & (STAYS - 1)) == static_cast<int>(gridDim.x)) {
      const int per_sm = static_cast<int>(gridDim.x) / p.n_sms;
      const int wanted = (p.n_sms - p.k2_sms) * per_sm + p.k2_sms * min(p.k2_sm_ctas, per_sm);
      return n / STAYS * 2 < wanted;
    }
  } while (globaltimer_ns() - t0 < 20000ull);
  return true;
}

template <bool G_BF16, bool FAST_EXP, bool BESIDE, K1Form FORM>
__global__ void __maxnreg__(BESIDE ? 112 : 128) kda_k1_kernel(const __grid_constant__ K1Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using SM = K1Smem<G_BF16, FAST_EXP>;
  constexpr int S_Q = SM::Q, S_K = SM::K, S_G = SM::G;
  constexpr uint32_t ROW_BYTES = D * 2;
  constexpr uint32_t G_ROW_BYTES = G_BF16 ? D * 2 : D * 4;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int n_items = (p.chunk_table != nullptr ? p.n_chunks : p.B * p.NT) * p.H;

  const uint32_t sbase = smem_u32(smem);
  const uint32_t mbar = sbase + SM::MBAR, mbar_v = sbase + SM::MBAR_V;
  float* sL = reinterpret_cast<float*>(smem + S_L);
  float* sBetaAll = reinterpret_cast<float*>(smem + SM::BETA);   // [2][16], then expA[2] at +32
  float* sTot = reinterpret_cast<float*>(smem + SM::TOT);
  float* sGmid = reinterpret_cast<float*>(smem + SM::GMID);
  float* sTot1 = sTot + D;
  volatile int* sFlag = reinterpret_cast<volatile int*>(smem + SM::FLAG);

  const bool use_gate = FORM == FORM_ANY ? (p.flags & 1u) != 0 : FORM == FORM_ALL;
  const bool use_l2 = FORM == FORM_ANY ? (p.flags & 2u) != 0 : FORM == FORM_ALL;
  const bool use_sigmoid = FORM == FORM_ANY ? (p.flags & 4u) != 0 : FORM == FORM_ALL;
  const int cp = tid & 63, rh = tid >> 6;   // phase-B mapping: column pair, row half
  const int c0 = cp * 2, r0 = rh * 8;

  if (tid == 0) {
    mbar_init(mbar, 1);
    mbar_init(mbar_v, 1);
    sFlag[0] = 0;   // a wait gave up
    fence_mbar_init();
    grid_dep_wait();   // the barrier holds the rest of the CTA
    // K2 may be set up, or run, beside this kernel.  Not before this kernel's own wait: K2 reads the initial state, and the table
    // of packed sequences, without waiting for more than this.  At once after it: behind the barrier below one chunk takes
    // 12.6 us in place of 12.4 on an idle stream, and 7.35 in place of 7.29 in a row of calls (T16 H32).
    if (!BESIDE) grid_dep_launch();
    if (!BESIDE && blockIdx.x == 0) *reinterpret_cast<int2*>(p.status) = make_int2(ST_OK, ST_OK);
    if (BESIDE) sFlag[1] = k1_stays(p) ? atomicAdd(p.progress - HDR_PROGRESS + HDR_TICKET, 2) : n_items;
  }
  __syncthreads();
  if (BESIDE) grid_dep_launch();   // those that leave have made way for K2

  // issue the input copies of one work item: one tiled TMA box (16 tokens x 128) per tensor.
  // The box may reach past T in the last chunk; those rows arrive as zeros and still count
  // towards the transaction bytes.
  auto issue_loads = [&](const K1Item& w) {
    if (tid == 0) {
      mbar_arrive_expect_tx(mbar, BT * (2 * ROW_BYTES + G_ROW_BYTES));
      tma_load_4d(sbase + S_Q, &p.tm_q, 0, w.hq, w.t0, w.b, mbar);
      tma_load_4d(sbase + S_K, &p.tm_k, 0, w.hq, w.t0, w.b, mbar);
      tma_load_4d(sbase + S_G, &p.tm_g, 0, w.h, w.t0, w.b, mbar);
    }
  };
  // thread 0: v goes straight into the record's part that leaves last, once that tile is free
  auto issue_v = [&](const K1Item& w) {
    mbar_arrive_expect_tx(mbar_v, BT * ROW_BYTES);
    tma_load_4d(sbase + S_V, &p.tm_v, 0, w.h, w.t0, w.b, mbar_v);
    tma_load_4d(sbase + S_V + REC_V_HALF, &p.tm_v, 64, w.h, w.t0, w.b, mbar_v);
  };
  // per-item parameters, fetched one item ahead so that their global-load latency is hidden
  struct Par { float a_log, bias0, bias1, beta; };
  auto load_params = [&](const K1Item& w) {
    Par q;
    q.a_log = use_gate ? ldg_pinned(p.A_log + w.h) : 0.f;
    q.bias0 = q.bias1 = 0.f;
    if (use_gate && p.dt_bias != nullptr) {
      if (FORM == FORM_ALL) {   // at an 8-byte boundary: see the choice of the instance
        const float2 bb = ldg_pinned2(p.dt_bias + w.h * D + c0);
        q.bias0 = bb.x; q.bias1 = bb.y;
      } else {
        q.bias0 = ldg_pinned(p.dt_bias + w.h * D + c0);
        q.bias1 = ldg_pinned(p.dt_bias + w.h * D + c0 + 1);
      }
    }
    q.beta = 0.f;   // held by threads 32..47 (warp 1), one token each
    if (tid >= 32 && tid < 48 && tid - 32 < w.nvalid)
      q.beta = ldg_pinned(p.beta + w.b * p.beta_s[0] + static_cast<int64_t>(w.t0 + tid - 32) * p.beta_s[1] + w.h * p.beta_s[2]);
    return q;
  };

  // Scalar per-item work -- exp(A_log) and the beta activation -- is done by warp 1 while warp 0
  // runs the triangular solve of the previous item, and handed over through shared memory.
  auto publish_params = [&](const Par& q, int nvalid_, int slot) {
    if (tid >= 32 && tid < 48) {
      float bv = q.beta;
      if (tid - 32 < nvalid_) { if (use_sigmoid) bv = 1.0f / (1.0f + __expf(-bv)); } else bv = 0.f;
      sBetaAll[slot * 16 + tid - 32] = bv;
    }
    if (tid == 48) sBetaAll[32 + slot] = use_gate ? expf(q.a_log) : 1.f;
  };

  // l2-normalisation of the q and k tiles in place: 8 threads per row, two 16-byte units each (units seg
  // and seg + 8, so that a quarter-warp's 16-byte accesses cover 128 contiguous bytes).
  auto l2_normalise = [&]() {
    const int r = tid >> 3, seg = tid & 7;
    uint4 qa[2], ka[2];
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int hseg = 0; hseg < 2; ++hseg) {
      qa[hseg] = *reinterpret_cast<const uint4*>(smem + S_Q + r * 256 + (seg + hseg * 8) * 16);
      ka[hseg] = *reinterpret_cast<const uint4*>(smem + S_K + r * 256 + (seg + hseg * 8) * 16);
      const uint32_t aw[4] = {qa[hseg].x, qa[hseg].y, qa[hseg].z, qa[hseg].w};
      const uint32_t cw[4] = {ka[hseg].x, ka[hseg].y, ka[hseg].z, ka[hseg].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float x0 = bf16_lo_to_f32(aw[i]), x1 = bf16_hi_to_f32(aw[i]);
        const float y0 = bf16_lo_to_f32(cw[i]), y1 = bf16_hi_to_f32(cw[i]);
        sq = fmaf(x0, x0, sq); sq = fmaf(x1, x1, sq);
        sk = fmaf(y0, y0, sk); sk = fmaf(y1, y1, sk);
      }
    }
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, m);
      sk += __shfl_xor_sync(0xffffffffu, sk, m);
    }
    const float rq = rsqrtf(sq + L2NORM_EPS), rk = rsqrtf(sk + L2NORM_EPS);
    auto scale4 = [](uint4 v, float f) {
      uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = pack_bf16(bf16_lo_to_f32(w[i]) * f, bf16_hi_to_f32(w[i]) * f);
      return make_uint4(w[0], w[1], w[2], w[3]);
    };
#pragma unroll
    for (int hseg = 0; hseg < 2; ++hseg) {
      *reinterpret_cast<uint4*>(smem + S_Q + r * 256 + (seg + hseg * 8) * 16) = scale4(qa[hseg], rq);
      *reinterpret_cast<uint4*>(smem + S_K + r * 256 + (seg + hseg * 8) * 16) = scale4(ka[hseg], rk);
    }
  };

  int id = BESIDE ? sFlag[1] : blockIdx.x;
  int id_next = BESIDE ? id + 1 : id + static_cast<int>(gridDim.x);
  if (BESIDE) __syncthreads();   // read by everyone before thread 0 puts the next one there
  K1Item cur{}, nxt{};
  Par par{}, par_next{};
  if (id < n_items) {
    cur = k1_item<BESIDE>(p, id);
    issue_loads(cur);
    par = load_params(cur);
    publish_params(par, cur.nvalid, 0);
  }

  // K2 beside K1: the items finished in the current window, and the window (and count) whose records
  // have been handed to the copy engine but not yet reported
  int done = 0, rep_win = 0, rep_done = 0;
  // thread 0, once per item and two phases after the stores were issued: the tiles may be rewritten
  // (their bulk stores have read them); with a window to report, the stores have also arrived
  auto drain_stores = [&]() {
    if (BESIDE && rep_done != 0) {
      bulk_wait_all();
      fence_proxy_async_all();
      red_release_gpu(p.progress + rep_win, rep_done);
    } else {
      bulk_wait_read_all();
    }
  };

  int it = 0;
  for (; id < n_items; ++it, id = id_next, id_next = BESIDE ? sFlag[1] : id_next + static_cast<int>(gridDim.x)) {
    const int b = cur.b, h = cur.h, t0 = cur.t0, nvalid = cur.nvalid;
    uint8_t* rec = p.rec + cur.rec_idx * REC_BYTES;
    const bool has_next = id_next < n_items;
    int ticket = n_items;   // thread 0: the item after the next one, on its way while this one is worked on
    if (has_next) {
      if (BESIDE && tid == 0) ticket = atomicAdd(p.progress - HDR_PROGRESS + HDR_TICKET, 1);
      nxt = k1_item<BESIDE>(p, id_next);
      par_next = load_params(nxt);
    }
    const float bias0 = par.bias0, bias1 = par.bias1;
    const float* sBeta = sBetaAll + (it & 1) * 16;

    // every thread waits for the input copies itself (no CTA barrier here); a thread whose wait runs
    // out raises the flag, and the whole CTA leaves together behind the barrier that ends phase A
    const bool ok = mbar_wait_bounded(mbar, it & 1, sFlag);
    if (!ok) *sFlag = 1;

    // packed sequences: behind the last token of a sequence the copies have brought the first tokens of the next one.  They
    // must not enter this chunk, not even times zero (they may not be finite): zeros, as behind the end of a batch row.
    // (Calls that do only some of gate, norms and sigmoid here, bf16 gate: T4096 H32 76.3 -> 77.4 us; the others the same.)
    if (!BESIDE && p.chunk_table != nullptr && nvalid < BT) {
#pragma unroll 1
      for (int i = nvalid * 16 + tid; ok && i < BT * 16; i += 128) {   // 16-byte units of a bf16 tile
        const uint4 z = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(smem + S_Q + i * 16) = z;
        *reinterpret_cast<uint4*>(smem + S_K + i * 16) = z;
        *reinterpret_cast<uint4*>(smem + S_G + i * (G_BF16 ? 16 : 32)) = z;
        if (!G_BF16) *reinterpret_cast<uint4*>(smem + S_G + i * 32 + 16) = z;
      }
      __syncthreads();
    }

    // ---- phase A: l2-normalise q and k in place.  (Not earlier, by the warps that do not solve under the previous
    //      item's solve: the inputs have rarely arrived by then; T8192 H32 149.5 us with a probe for them, 147.1 without.) ----
    if (use_l2 && ok) l2_normalise();
    __syncthreads();
    if (*sFlag != 0) {
      // a copy never completed: report, give in-flight copies one more bounded wait, leave
      if (tid == 0) {
        atomicExch(p.status, ST_K1_LOAD_TIMEOUT);
        p.status[HDR_K1_STATUS] = ST_K1_LOAD_TIMEOUT;
        mbar_wait_bounded(mbar, it & 1, nullptr);
        mbar_wait_bounded(mbar_v, (it + 1) & 1, nullptr);   // of the item before
        bulk_wait_read_all();
      }
      __syncthreads();
      return;
    }

    // ---- phase B: thread = (column pair, row half): gate, cumsum, gated operands ----
    // Two adjacent columns per thread: every bf16 conversion is the packed cvt.rn.bf16x2
    // (full-rate pipe), every tile store is 32 bits wide and the fp32 arithmetic runs as
    // packed f32x2 instructions.
    // Centring of the Gram exponents.  General path: the chunk's middle row, as in the reference
    // (src/kda_bt16/kernels.py:129-139), which keeps every factor finite for any lower_bound
    // in (-11, 0).  FAST_EXP (16*|lower_bound|*RCP_LN2 <= 120, e.g. the production -5): the
    // LAST row, where 2^(g_last-g) <= 1 is exactly K2's kg operand, so the Grams reuse the kg
    // tiles as their B operand and 2^g = 2^(g-g_last) * 2^g_last costs no third exponential.
    uint32_t kbh[8];
    float2 dec2;
    {
      float2 gv[8];
      float2 gmid, glast;
      auto ld_g = [&](int r) -> float2 {
        if (G_BF16) {
          const uint32_t gp = *reinterpret_cast<const uint32_t*>(smem + S_G + (r * D + c0) * 2);
          return make_float2(bf16_lo_to_f32(gp), bf16_hi_to_f32(gp));
        }
        return *reinterpret_cast<const float2*>(smem + S_G + (r * D + c0) * 4);
      };
      if (use_gate) {
        // exp(-z) = 2^(nA * x + nb) with nA = -exp(A_log) log2(e), nb = nA * bias
        const float nA = -sBetaAll[32 + (it & 1)] * 1.4426950408889634f;
        const float2 nA2 = make_float2(nA, nA), nb2 = make_float2(nA * bias0, nA * bias1);
        const float2 one2 = make_float2(1.f, 1.f);
        const float lbr = p.lower_bound * RCP_LN2;
        const int mid = min(BT / 2, nvalid - 1);
        float2 run = make_float2(0.f, 0.f), gm = run;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = r0 + i;
          const float2 z = __ffma2_rn(ld_g(r), nA2, nb2);
          const float2 den = __fadd2_rn(make_float2(ex2f(z.x), ex2f(z.y)), one2);
          const float lb_r = (r < nvalid) ? lbr : 0.f;           // rows past the end add nothing
          const float2 gate = __fmul2_rn(make_float2(rcpf(den.x), rcpf(den.y)), make_float2(lb_r, lb_r));
          run = __fadd2_rn(run, gate);
          gv[i] = run;
          if (r == mid) gm = run;
        }
        // rows 8..15 need the sum over rows 0..7, all rows need g[last] and g[centre]: both halves
        // publish their column sums (and the half that owns the centre row its running sum there),
        // one barrier, and every thread completes its own values
        *reinterpret_cast<float2*>((rh == 0 ? sTot : sTot1) + c0) = run;
        if (!FAST_EXP && rh == (mid >> 3)) *reinterpret_cast<float2*>(sGmid + c0) = gm;
        // the previous item's bulk stores must have read the qg / kg / Aqk / dec tiles before the
        // operand loop below rewrites them; by now they have had two phases to do so
        if (tid == 0) { drain_stores(); issue_v(cur); }
        __syncthreads();
        const float2 t0 = *reinterpret_cast<const float2*>(sTot + c0);
        const float2 t1 = *reinterpret_cast<const float2*>(sTot1 + c0);
        if (rh == 1) {
#pragma unroll
          for (int i = 0; i < 8; ++i) gv[i] = __fadd2_rn(gv[i], t0);
        }
        glast = __fadd2_rn(t1, t0);
        gmid = make_float2(0.f, 0.f);
        if (!FAST_EXP) {
          gmid = *reinterpret_cast<const float2*>(sGmid + c0);
          if ((mid >> 3) == 1) gmid = __fadd2_rn(gmid, t0);
        }
      } else {
        // g already holds the chunk-local log2 cumsum; rows past the end repeat the last valid row
#pragma unroll
        for (int i = 0; i < 8; ++i) gv[i] = ld_g(min(r0 + i, nvalid - 1));
        gmid = ld_g(min(BT / 2, nvalid - 1));
        glast = ld_g(nvalid - 1);
        if (tid == 0) { drain_stores(); issue_v(cur); }   // as above
        __syncthreads();
      }
      dec2 = make_float2(ex2f(glast.x), ex2f(glast.y));
      if (rh == 1) {
        *reinterpret_cast<float2*>(smem + S_DEC + c0 * 4) = dec2;
      } else {
        *reinterpret_cast<float*>(smem + S_DEC2 + dec_lane_off(c0)) = dec2.x;
        *reinterpret_cast<float*>(smem + S_DEC2 + dec_lane_off(c0 + 1)) = dec2.y;
      }

      if (FORM == FORM_ANY && p.g_out != nullptr) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (r0 + i < nvalid)
            *reinterpret_cast<float2*>(p.g_out + ((static_cast<size_t>(b) * p.T + t0 + r0 + i) * p.H + h) * D + c0) = gv[i];
      }

      const float2 centre = FAST_EXP ? glast : gmid;
      const float2 ncentre = make_float2(-centre.x, -centre.y);
      // kg goes out transposed, eight tokens of a column per 16-byte store: pairs of rows are packed
      uint32_t kgh[2][4], kgl[2][4];
#pragma unroll
      for (int i2 = 0; i2 < 4; ++i2) {
        float2 kg2[2];
#pragma unroll
        for (int ii = 0; ii < 2; ++ii) {
          const int i = i2 * 2 + ii, r = r0 + i;
          const uint32_t off = swz_off(r, c0);
          const uint32_t qp = *reinterpret_cast<const uint32_t*>(smem + S_Q + (r * D + c0) * 2);
          const uint32_t kp = *reinterpret_cast<const uint32_t*>(smem + S_K + (r * D + c0) * 2);
          const float2 qn = make_float2(bf16_lo_to_f32(qp), bf16_hi_to_f32(qp));   // already normalised
          const float2 kn = make_float2(bf16_lo_to_f32(kp), bf16_hi_to_f32(kp));
          const float2 d = __fadd2_rn(gv[i], ncentre);                  // g - centre
          const float2 e = make_float2(ex2f(d.x), ex2f(d.y));           // 2^(g - centre)
          const float2 en = make_float2(ex2f(-d.x), ex2f(-d.y));        // 2^(centre - g)
          float2 eg, ekg;                                               // 2^g, 2^(g_last - g)
          if (FAST_EXP) { eg = __fmul2_rn(e, dec2); ekg = en; }
          else {
            eg = make_float2(ex2f(gv[i].x), ex2f(gv[i].y));
            ekg = make_float2(ex2f(glast.x - gv[i].x), ex2f(glast.y - gv[i].y));
          }
          uint32_t hi, lo;
          split_pack2(__fmul2_rn(qn, e), hi, lo);
          *reinterpret_cast<uint32_t*>(smem + S_QGH + off) = hi;
          *reinterpret_cast<uint32_t*>(smem + S_QGL + off) = lo;
          split_pack2(__fmul2_rn(kn, e), hi, lo);
          *reinterpret_cast<uint32_t*>(smem + S_KQH + off) = hi;
          *reinterpret_cast<uint32_t*>(smem + S_KQL + off) = lo;
          if (!FAST_EXP) {
            split_pack2(__fmul2_rn(kn, en), hi, lo);
            *reinterpret_cast<uint32_t*>(smem + S_KNH + off) = hi;
            *reinterpret_cast<uint32_t*>(smem + S_KNL + off) = lo;
          }
          kg2[ii] = __fmul2_rn(kn, ekg);
          const float2 qgo = __fmul2_rn(qn, eg);
          *reinterpret_cast<uint32_t*>(smem + S_QG + stage_off(r, c0)) = pack_bf16(qgo.x, qgo.y);
          const float br = sBeta[r];
          const float2 kbv = __fmul2_rn(__fmul2_rn(kn, make_float2(br, br)), eg);
          kbh[i] = pack_bf16(kbv.x, kbv.y);
        }
        split_pack(kg2[0].x, kg2[1].x, kgh[0][i2], kgl[0][i2]);
        split_pack(kg2[0].y, kg2[1].y, kgh[1][i2], kgl[1][i2]);
      }
      // a lane's two columns are neighbours: half of the lanes store the odd one first, so that the eight lanes of a
      // shared-memory pass cover 128 different bytes
      const bool odd_first = (lane & 4) != 0;
      auto put = [&](int base, const uint32_t (&t)[2][4]) {
        uint32_t x[4], y[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) { x[w] = odd_first ? t[1][w] : t[0][w]; y[w] = odd_first ? t[0][w] : t[1][w]; }
        const uint32_t off = base + kg_off(r0, c0);
        *reinterpret_cast<uint4*>(smem + off + (odd_first ? 16 : 0)) = make_uint4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<uint4*>(smem + off + (odd_first ? 0 : 16)) = make_uint4(y[0], y[1], y[2], y[3]);
      };
      put(S_KGH, kgh);
      put(S_KGL, kgl);
    }
    __syncthreads();  // every thread has read its q/k/g elements: the input tiles are free

    // ---- prefetch: the next item's inputs go into the same tiles while this one finishes ----
    if (has_next) {
      if (tid == 0) fence_proxy_async();   // order the earlier generic accesses (made visible by the barrier) before the async writes
      issue_loads(nxt);
    }

    // ---- phase C: Grams on the tensor cores (one 16x8 output tile per warp) ----
    {
      const int mt = warp >> 1;  // 0: Aqk, 1: Akk
      const int nt = warp & 1;   // column block j in [8nt, 8nt+8)
      const int arow = (lane & 7) + ((lane >> 3) & 1) * 8, acol = (lane >> 4) * 8;
      // swizzled address of k-step ks = (256-byte aligned tile base + lane part) ^ (ks << 5)
      const uint32_t a_hi = sbase + (mt == 0 ? S_QGH : S_KQH) + swz_off(arow, acol);
      // B operand: out of the transposed kg tile (rows k, columns tok; a k-step is 256 bytes), or with the general
      // centring out of the swizzled kn tile (rows tok, columns k)
      const uint32_t b_hi = sbase + (FAST_EXP ? S_KGH + kg_off(nt * 8, lane) : S_KNH + swz_off(nt * 8 + (lane & 7), (lane >> 3) * 8));
      constexpr uint32_t A_LO = S_QGL - S_QGH, B_LO = FAST_EXP ? S_KGL - S_KGH : S_KNL - S_KNH;
      static_assert(S_KQL - S_KQH == S_QGL - S_QGH && S_GRAM % 256 == 0, "tile layout");
      float acc0[4] = {0, 0, 0, 0}, acc1[4] = {0, 0, 0, 0}, acc2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int kp = 0; kp < 4; ++kp) {
        uint32_t bh[4], bl[4];   // two k-steps
        if (FAST_EXP) {
          ldsm_x4_t(b_hi + kp * 512, bh[0], bh[1], bh[2], bh[3]);
          ldsm_x4_t(b_hi + kp * 512 + B_LO, bl[0], bl[1], bl[2], bl[3]);
        } else {
          ldsm_x4(b_hi ^ (kp << 6), bh[0], bh[1], bh[2], bh[3]);
          ldsm_x4((b_hi ^ (kp << 6)) + B_LO, bl[0], bl[1], bl[2], bl[3]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int ks = kp * 2 + j;
          uint32_t ah[4], al[4];
          ldsm_x4(a_hi ^ (ks << 5), ah[0], ah[1], ah[2], ah[3]);
          ldsm_x4((a_hi ^ (ks << 5)) + A_LO, al[0], al[1], al[2], al[3]);
          mma_bf16(acc0, ah, bh[2 * j], bh[2 * j + 1]);
          mma_bf16(acc1, ah, bl[2 * j], bl[2 * j + 1]);
          mma_bf16(acc2, al, bh[2 * j], bh[2 * j + 1]);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) acc0[e] += acc1[e] + acc2[e];
      const int j0 = nt * 8 + tq * 2;
      if (mt == 0) {
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
          const int i = gq + hrow * 8;
          const float v0 = (i >= j0) ? acc0[hrow * 2] * p.scale : 0.f;
          const float v1 = (i >= j0 + 1) ? acc0[hrow * 2 + 1] * p.scale : 0.f;
          uint32_t hi2, lo2;
          split_pack(v0, v1, hi2, lo2);
          *reinterpret_cast<uint32_t*>(smem + S_AQK + aq_off(i, j0)) = hi2;
          *reinterpret_cast<uint32_t*>(smem + S_AQL + aq_off(i, j0)) = lo2;
        }
      } else {
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
          const int i = gq + hrow * 8;
          const float bi = sBeta[i];
          // the solve consumes -Akk
          *reinterpret_cast<float2*>(sL + i * 16 + j0) =
              make_float2((i > j0) ? -acc0[hrow * 2] * bi : 0.f, (i > j0 + 1) ? -acc0[hrow * 2 + 1] * bi : 0.f);
        }
      }
    }
    __syncthreads();   // Grams done: their A tiles are free, -Akk is visible

    // the B operand of w takes the place of a Gram A tile
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t off = swz_off(r0 + i, c0);
      *reinterpret_cast<uint32_t*>(smem + S_KBH + off) = kbh[i];
    }

    // next item's scalar parameters (warp 1, while warp 0 solves)
    if (has_next) publish_params(par_next, nxt.nvalid, (it + 1) & 1);

    // ---- phase D: X = (I + L)^-1, lanes j and 16 + j of warp 0 own column j (the latter go on with X diag(beta)) ----
    // Column sweep (right-looking): once x[m] is final, every later row takes its update, so the
    // dependent chain is 16 FMAs long; -L is read four columns at a time.
    if (warp == 0) {
      const int col = lane & 15;
      float x[BT];
#pragma unroll
      for (int i = 0; i < BT; ++i) x[i] = (i == col) ? 1.f : 0.f;
#pragma unroll
      for (int mb = 0; mb < 4; ++mb) {
#pragma unroll
        for (int i = mb * 4 + 1; i < BT; ++i) {
          const float4 l4 = *reinterpret_cast<const float4*>(sL + i * 16 + mb * 4);
          const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
          for (int mm = 0; mm < 4; ++mm)
            if (mb * 4 + mm < i) x[i] = fmaf(lv[mm], x[mb * 4 + mm], x[i]);
        }
      }
      __syncwarp();   // -Akk has been read by all lanes: X takes its place
      const float by = lane < 16 ? 1.f : sBeta[col];
      const uint32_t x_at = (lane < 16 ? S_XH : S_XBH) + xb_off(0, col);
      static_assert(S_XL - S_XH == S_XBL - S_XBH, "hi to lo");
#pragma unroll
      for (int i = 0; i < BT; ++i) {
        const float xb = x[i] * by, hi = bf16_round(xb);
        *reinterpret_cast<unsigned short*>(smem + x_at + i * 16) = bf16_bits(hi);
        *reinterpret_cast<unsigned short*>(smem + x_at + i * 16 + (S_XL - S_XH)) = bf16_bits(xb - hi);
      }
      if (FORM == FORM_ANY && p.ainv_out != nullptr) {
#pragma unroll
        for (int i = 0; i < BT; ++i)
          if (i < nvalid && lane < 16) p.ainv_out[((static_cast<size_t>(b) * p.T + t0 + i) * p.H + h) * BT + lane] = x[i];
      }
    }
    // packed sequences: v behind the last token of a sequence, as for the other inputs above
    if (!BESIDE && p.chunk_table != nullptr && nvalid < BT) {
      if (!mbar_wait_bounded(mbar_v, it & 1, sFlag)) {   // reported here: for thread 0 it may yet come
        *sFlag = 1;
        atomicExch(p.status, ST_K1_LOAD_TIMEOUT);
        p.status[HDR_K1_STATUS] = ST_K1_LOAD_TIMEOUT;
      }
#pragma unroll 1
      for (int i = nvalid * 16 + tid; *sFlag == 0 && i < BT * 16; i += 128)   // 16-byte units
        *reinterpret_cast<uint4*>(smem + S_V + (i & 1) * REC_V_HALF + (i >> 1) * 16) = make_uint4(0, 0, 0, 0);
    }
    fence_proxy_async();   // qg / kg / Aqk / dec / Xb tiles were written with plain stores
    __syncthreads();

    // the finished tiles leave while phase E runs
    if (tid == 0) {
      // v was asked for two phases ago; if it does not come, the CTA leaves at the start of the next item
      if (!mbar_wait_bounded(mbar_v, it & 1, nullptr)) {
        *sFlag = 1;
        atomicExch(p.status, ST_K1_LOAD_TIMEOUT);
        p.status[HDR_K1_STATUS] = ST_K1_LOAD_TIMEOUT;
      }
      bulk_s2g(rec + REC_QG, sbase + S_QG, TILE_BYTES / 2);
      bulk_s2g(rec + REC_QG + REC_HALF, sbase + S_QG + TILE_BYTES / 2, TILE_BYTES / 2);
      bulk_s2g(rec + REC_KGH, sbase + S_KGH, REC_USED_BYTES - REC_KGH);
      bulk_commit();
    }

    // ---- phase E: -w = -X (khat beta 2^g) (bf16), staged for a bulk store ----
    {
      // X as A operand (row-major [M=i][K=m]), hi and lo parts
      uint32_t xah[4], xal[4];
      {
        const uint32_t x_at = sbase + xb_off((lane & 7) + ((lane >> 3) & 1) * 8, (lane >> 4) * 8);
        ldsm_x4(x_at + S_XH, xah[0], xah[1], xah[2], xah[3]);
        ldsm_x4(x_at + S_XL, xal[0], xal[1], xal[2], xal[3]);
      }
      // B operands come from [tok][col] tiles through transposing ldmatrix; one x4 covers 16 columns
      const int btok = (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int ni = 0; ni < 2; ++ni) {
        const int n0 = warp * 32 + ni * 16;
        uint32_t bk[4];
        ldsm_x4_t(sbase + S_KBH + swz_off(btok, n0 + (lane >> 4) * 8), bk[0], bk[1], bk[2], bk[3]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float accw[4] = {0, 0, 0, 0};
          mma_bf16(accw, xah, bk[2 * j], bk[2 * j + 1]);
          mma_bf16(accw, xal, bk[2 * j], bk[2 * j + 1]);
          const int kc = n0 + j * 8 + tq * 2;
          *reinterpret_cast<uint32_t*>(smem + S_WST + stage_off(gq, kc)) = pack_bf16(-accw[0], -accw[1]);
          *reinterpret_cast<uint32_t*>(smem + S_WST + stage_off(gq + 8, kc)) = pack_bf16(-accw[2], -accw[3]);
        }
      }
    }
    // w leaves as one more bulk store (4-byte stores of a swizzled tile straight to global memory
    // would cost eight sectors per instruction)
    fence_proxy_async();
    ++done;
    rep_done = 0;
    if (BESIDE && (!has_next || nxt.win != cur.win)) {
      // the window's last item of this CTA: thread 0 reports it once its stores have arrived
      rep_win = cur.win;
      rep_done = done;
      done = 0;
    }
    if (BESIDE && tid == 0) sFlag[1] = ticket;
    __syncthreads();   // also orders phase E's reads of Xb / KB before the next item rewrites them
    if (tid == 0) {
      bulk_s2g(rec + REC_W, sbase + S_WST, TILE_BYTES / 2);
      bulk_s2g(rec + REC_W + REC_HALF, sbase + S_WST + TILE_BYTES / 2, TILE_BYTES / 2);
      bulk_commit();
    }
    cur = nxt;
    par = par_next;
  }
  if (tid == 0) {
    if (*sFlag == 0) {
      drain_stores();
    } else {   // v of the last item did not come: no window is reported
      mbar_wait_bounded(mbar_v, (it + 1) & 1, nullptr);
      bulk_wait_read_all();
    }
  }
}

// Clears the header for a K1 with K2 beside it: starts ahead of the end of the call before, and K1 ahead of this one's end.
__global__ void kda_clear_header_kernel(int* header) {
  grid_dep_wait();
  header[threadIdx.x] = 0;
  grid_dep_launch();
}

cudaError_t launch_clear_header(int* header, cudaStream_t stream) {
  return launch_dep(kda_clear_header_kernel, 1, WS_HEADER_BYTES / 4, 0, stream, 1, header);
}

template <bool G_BF16, bool FAST_EXP, bool BESIDE, K1Form FORM>
static cudaError_t launch_k1_t(const K1Params& p, cudaStream_t stream) {
  constexpr int smem_bytes = K1Smem<G_BF16, FAST_EXP>::TOTAL;
  // per device: SMs << 8 | resident CTAs per SM, 0 = not looked up yet.  One word, published after the attributes
  // are set: another thread's first call sees all of it or nothing.
  static std::atomic<int> residency[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64) return cudaErrorInvalidDevice;
  int res = residency[dev].load(std::memory_order_acquire);
  if (res == 0) {
    auto kern = kda_k1_kernel<G_BF16, FAST_EXP, BESIDE, FORM>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
    // ask for the full shared-memory carve-out so that four CTAs are resident per SM
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int n_sms = 0, per_sm = 0;
    e = cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, smem_bytes);
    if (e != cudaSuccess) return e;
    res = n_sms << 8 | (per_sm > 0 ? per_sm : 1);
    residency[dev].store(res, std::memory_order_release);
  }
  const long long n_items = (p.chunk_table != nullptr ? static_cast<long long>(p.n_chunks) : static_cast<long long>(p.B) * p.NT) * p.H;
  const int cap = (res >> 8) * (res & 255);   // persistent: one CTA per slot
  const int grid = static_cast<int>(n_items < cap ? n_items : cap);
  return launch_dep(kda_k1_kernel<G_BF16, FAST_EXP, BESIDE, FORM>, grid, 128, smem_bytes, stream, 1, p);
}

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}
}  // namespace

cudaError_t k1_encode_tensor_maps(K1Params& p, bool g_bf16, const char** what) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) { *what = "cuTensorMapEncodeTiled is not available from this driver"; return cudaErrorNotSupported; }
  struct T { CUtensorMap* m; const void* ptr; const int64_t* s; CUtensorMapDataType dt; int es; const char* name; };
  const T ts[4] = {
      {&p.tm_q, p.q, p.q_s, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, "q"},
      {&p.tm_k, p.k, p.k_s, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, "k"},
      {&p.tm_v, p.v, p.v_s, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, "v"},
      {&p.tm_g, p.g, p.g_s, g_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, g_bf16 ? 2 : 4, "g"}};
  for (const T& t : ts) {
    // dims innermost first: (d, head, token, batch); strides in bytes for dims 1..3.  A size-1
    // dimension may come with any stride: give it a legal one (it is never stepped).  A zero
    // stride on a larger dimension (an expanded view) is refused by the argument check.
    const bool qk = (t.m == &p.tm_q || t.m == &p.tm_k);
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(qk ? p.Hq : p.H),
                                static_cast<cuuint64_t>(p.T), static_cast<cuuint64_t>(p.B)};
    cuuint64_t strides[3] = {static_cast<cuuint64_t>(t.s[2]) * t.es, static_cast<cuuint64_t>(t.s[1]) * t.es,
                             static_cast<cuuint64_t>(t.s[0]) * t.es};
    for (int i = 0; i < 3; ++i)
      if (dims[i + 1] == 1) strides[i] = static_cast<cuuint64_t>(D) * t.es;
    // v arrives in two boxes of 64 columns, in the 128-byte swizzle of its place in the record
    const bool is_v = t.m == &p.tm_v;
    const cuuint32_t box[4] = {static_cast<cuuint32_t>(is_v ? D / 2 : D), 1, static_cast<cuuint32_t>(BT), 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(t.m, t.dt, 4, const_cast<void*>(t.ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     is_v ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { *what = t.name; return cudaErrorInvalidValue; }
  }
  return cudaSuccess;
}

template <bool G_BF16, bool BESIDE>
static cudaError_t launch_k1_b(const K1Params& p, bool fast_exp, cudaStream_t stream) {
  const uint32_t in_kernel = p.flags & 7u;
  const bool debug = p.g_out != nullptr || p.ainv_out != nullptr;
  // dt_bias may be a view that starts at any float of a larger buffer.  FORM_ALL reads it two floats at a time (one at a time
  // costs it 0.2 %: T8192 H96 719.7 -> 721.2 us, T100 H32 11.16 -> 11.22), the others by single floats.
  const bool all = in_kernel == 7u && !debug && reinterpret_cast<uintptr_t>(p.dt_bias) % sizeof(float2) == 0;
  if (fast_exp)
    return all ? launch_k1_t<G_BF16, true, BESIDE, FORM_ALL>(p, stream)
               : launch_k1_t<G_BF16, true, BESIDE, FORM_ANY>(p, stream);
  if (all) return launch_k1_t<G_BF16, false, BESIDE, FORM_ALL>(p, stream);
  if (in_kernel == 0u && !debug) return launch_k1_t<G_BF16, false, BESIDE, FORM_NONE>(p, stream);
  return launch_k1_t<G_BF16, false, BESIDE, FORM_ANY>(p, stream);
}

cudaError_t launch_k1(const K1Params& p, bool g_bf16, bool fast_exp, cudaStream_t stream) {
  if (g_bf16) return p.progress != nullptr ? launch_k1_b<true, true>(p, fast_exp, stream) : launch_k1_b<true, false>(p, fast_exp, stream);
  return p.progress != nullptr ? launch_k1_b<false, true>(p, fast_exp, stream) : launch_k1_b<false, false>(p, fast_exp, stream);
}

}  // namespace kda
