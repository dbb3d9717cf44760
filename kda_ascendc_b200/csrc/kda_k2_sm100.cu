// K2: delta-rule state recurrence and output of the KDA forward.  sm_100a.
//
// Replaces kda_bt16_kernel_k2 of the reference (src/kda_bt16/kernels.py:187-302); the
// arithmetic is the recurrence of the reference's torch chunk implementation
// (tests/test_torch_reference.py:175-194), V-first state h[V][K]:
//   v_new = u - w h^T ;  o = scale (qg h^T) + Aqk v_new ;  h = h diag(dec) + v_new^T kg
// The record holds -w, and u as its factors: u = Xb v.
//
// The recurrence is independent per state row v (v_new[:, v], o[:, v] and h[v, :] only use
// row v), so V is the dimension that is spread over warps.  It is mapped to the MMA *N*
// dimension, whose granularity is 8: a warp owns NVT tiles of 8 rows of h and keeps them,
// transposed, in registers for the whole sequence:  hT[k][v], fp32, m16n8 accumulator
// fragments (8 k-tiles of 16).  Per chunk, per warp:
//   P1: [-w hT | o] = [-w ; qg] hT      M = 16+16 tokens, N = 8 v, K = 128   (16 MMAs / tile)
//   u = Xb v                            M = 16 tokens,    N = 8 v, K = 16    (2 MMAs, hi and lo of Xb)
//   P2: hT += kg^T v_new                M = 128 k,        N = 8 v, K = 16    (3 x 8 MMAs)
//   P3: o += Aqk v_new                  M = 16 tokens,    N = 8 v, K = 16    (3 MMAs)
// A operands ([w;qg], kg^T, Aqk) are state independent and come from the chunk record in
// shared memory by ldmatrix; B operands are the warp's own data (bf16(hT), v_new): an
// accumulator fragment becomes a B fragment by an in-warp 8x8 transpose (movmatrix), so the
// serial chain  hT -> P1 -> v_new -> P2 -> hT  never leaves the warp: no shared-memory round
// trip and no inter-warp synchronisation sits on it.  That chain, NT dependent steps per
// head, is what bounds this kernel, together with the legacy tensor pipe (one m16n8k16 per
// 8 cycles per SM sub-partition).  P2 uses a hi/lo bf16 split of both v_new and kg (three
// MMAs) because the state must stay within 2e-3 of an fp32 implementation; P3 does the same
// with v_new and Aqk (the intra-chunk term dominates o); P1 uses plain bf16 operands.
// The result does not depend on how the rows are distributed over warps and CTAs.
//
// One warp executes its chain in program order: 45 MMAs of 8 cycles, 20 movmatrix of 5.5, 37 ldmatrix, and the waits
// between the dependent parts.  Loads are interleaved with the MMA sequences so that their latency is covered: P1
// carries this step's kg fragment loads and the decay of hT; P2 carries the next step's [w;qg] / decay loads and P3.
// A step takes 0.34 to 0.35 us with one or two consumer warps per CTA and 0.45 with four (T8192 H32 K2 230 us), where the operand
// fragments of four warps keep the SM's shared-memory pipe busy.  Measured without gain: the fragments copied into
// tensor memory once per SM (tcgen05.cp) and read by tcgen05.ld, 0.79 us: a copy stalls the SM's mma.sync while it runs.
//
// A CTA = CW consumer warps (CW*NVT*8 state rows of one (batch, head)) plus one producer warp
// that streams the chunk records through a ring of shared-memory stages with bulk (TMA)
// copies: full/empty mbarriers, every wait bounded.
#include <type_traits>

#include "kda_common.cuh"
#include "kda_kernels.h"

namespace kda {

// STAGES: 4, and beside K1, which holds up the records now and then, 6 (with four consumer warps, on SMs of their own, 8):
// whole forward T131072 H16 3,756 -> 3,704 us, B2 T4096 H8 131.4 -> 129.0, T8192 H19 296 -> 277, H22 293 -> 290
template <int STAGES>
struct K2Smem {
  static constexpr int STAGE = REC_SHARED_BYTES + REC_V_HALF;   // a CTA's columns of v lie in one half
  static constexpr int BARS = STAGES * STAGE;               // full[S], empty[S]
  static constexpr int FLAG = BARS + 2 * STAGES * 8;        // abort flag, issued count
  static constexpr int TOTAL = FLAG + 16;
};

// PAIR (state-only, NVT = 2): the transform-pair pass of the sequence split.  The two 8-row tiles
// of a warp are the SAME eight state rows of two recurrences over the same records -- tile 0 starts
// from the identity with the u term dropped (the segment's transition matrix M), tile 1 from zero
// with u (its offset Q) -- so every operand fragment fetched from shared memory feeds two MMAs.
// The states leave as [chains][2][128][128].
// ORD: packed sequences, longest first (an instantiation of its own: the plain one steps 10 % slower with the
// order compiled in, T8192 H32 418 -> 460 us).
template <int CW, int NVT, bool STATE_ONLY, bool PAIR = false, bool ORD = false, int K2_STAGES = 4>
__global__ void __launch_bounds__((CW + 1) * 32, 1) kda_k2_kernel(const K2Params p) {
  static_assert(!PAIR || (STATE_ONLY && NVT == 2), "the pair mode is a state-only pass over two tiles");
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int RT = PAIR ? 1 : NVT;    // distinct 8-row tiles per warp
  using SM = K2Smem<K2_STAGES>;
  constexpr int VCOLS = CW * RT * 8;    // state rows (v) per CTA
  constexpr int NV = D / VCOLS;         // CTAs per (batch, head)
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  // chain: index of the recurrence this CTA works on.  With K2Params::pair_mode (state-only, one
  // tile per warp) the launch runs two chains per (batch, head): 2c from the identity without u,
  // 2c + 1 from zero with u, and writes them as [chains][2][128][128].
  const int chain = ORD ? chain_by_length(p.seq_table, p.n_seqs, p.H, blockIdx.x / NV + p.chain0) : blockIdx.x / NV + p.chain0;
  const bool pair_rt = !PAIR && STATE_ONLY && p.pair_mode != 0;
  const int bh = pair_rt ? (chain >> 1) : chain;   // the (batch, head) whose records are walked
  const int plane = pair_rt ? (chain & 1) : 1;
  const int vs = blockIdx.x % NV;
  int b = bh / p.H;
  const int h = bh % p.H;
  int NT = p.NT, Tlen = p.T, tok0 = 0;
  size_t rec_first = static_cast<size_t>(bh) * NT;
  if (p.seq_table != nullptr) {   // packed sequences: bh = sequence * H + head
    const int4 e = __ldg(p.seq_table + b);
    tok0 = e.x; NT = e.y; Tlen = e.w;
    rec_first = static_cast<size_t>(e.z) + static_cast<size_t>(h) * NT;
    b = 0;
  }

  const uint32_t sbase = smem_u32(smem);
  const uint32_t full0 = sbase + SM::BARS;
  const uint32_t empty0 = full0 + K2_STAGES * 8;
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + SM::FLAG);
  volatile int* sIssued = sAbort + 1;

  if (tid == 0) {
    for (int s = 0; s < K2_STAGES; ++s) {
      mbar_init(full0 + s * 8, 1);
      mbar_init(empty0 + s * 8, CW);
    }
    *sAbort = 0;
    *sIssued = 0;
    fence_mbar_init();
  }
  __syncthreads();

  const uint8_t* rec_bh = p.rec + rec_first * REC_BYTES;

  if (warp == CW) {
    // ------------------------------ producer -------------------------------
    if (lane == 0) {
      if (p.progress == nullptr) grid_dep_wait();   // K1's records; everything above ran under K1's tail
      int gate = 0;                                 // beside K1: the first chunk of the next window
      for (int n = 0; n < NT; ++n) {
        const int s = n % K2_STAGES;
        if (p.progress != nullptr && n == gate) {
          if (!window_wait_bounded(p.progress + n / p.win_chunks, min(p.win_chunks, NT - n) * p.B * p.H, sAbort)) {
            if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K1_WINDOW_TIMEOUT); }
            break;
          }
          gate += p.win_chunks;
        }
        if (n >= K2_STAGES) {
          if (!mbar_wait_bounded(empty0 + s * 8, ((n / K2_STAGES) - 1) & 1, sAbort)) {
            if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2_EMPTY_TIMEOUT); }
            break;
          }
        }
        const uint8_t* rec = rec_bh + static_cast<size_t>(n) * REC_BYTES;
        const uint32_t dst = sbase + s * SM::STAGE;
        mbar_arrive_expect_tx(full0 + s * 8, SM::STAGE);
        bulk_g2s(dst, rec, REC_SHARED_BYTES, full0 + s * 8);
        bulk_g2s(dst + REC_SHARED_BYTES, rec + REC_V + (vs * VCOLS >> 6) * REC_V_HALF, REC_V_HALF, full0 + s * 8);
        *sIssued = n + 1;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------ consumers ------------------------------
    const int gq = lane >> 2, tq = lane & 3;
    const int v0 = vs * VCOLS + warp * (RT * 8);   // first state row of this warp
    // hT[m][nv][e]: k = 16m + gq (+8 for e >= 2), v = v0 + 8nv + 2tq + (e & 1)   (PAIR: v = v0 + 2tq + (e & 1))
    float hT[8][NVT][4];
    bool h0_ok = true;
    if (PAIR) {
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          hT[m][0][e] = ((v0 + tq * 2 + (e & 1)) == (m * 16 + gq + (e >> 1) * 8)) ? 1.f : 0.f;
          hT[m][NVT - 1][e] = (NVT > 1) ? 0.f : hT[m][0][e];
        }
    } else if (pair_rt) {
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            hT[m][nv][e] = (plane == 0 && (v0 + nv * 8 + tq * 2 + (e & 1)) == (m * 16 + gq + (e >> 1) * 8)) ? 1.f : 0.f;
    } else if (p.h0 != nullptr) {
      if (p.h0_n_flags > 0) {   // the entry state comes from other GPUs: wait for their flags (the producer warp is already loading records)
        int ok = 1;
        if (lane == 0)
          for (int i = 0; i < p.h0_n_flags; ++i) ok &= flag_wait_bounded(p.h0_flags + i, p.h0_epoch) ? 1 : 0;
        h0_ok = __shfl_sync(0xffffffffu, ok, 0) != 0;
      }
      const float* h0 = p.h0 + static_cast<size_t>(bh) * D * D;
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            hT[m][nv][e] = p.k_first ? h0[(m * 16 + gq + (e >> 1) * 8) * D + v0 + nv * 8 + tq * 2 + (e & 1)]
                                     : h0[(v0 + nv * 8 + tq * 2 + (e & 1)) * D + m * 16 + gq + (e >> 1) * 8];
    } else {
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) hT[m][nv][0] = hT[m][nv][1] = hT[m][nv][2] = hT[m][nv][3] = 0.f;
    }

    // per-lane ldmatrix address components (constant across steps): mi = the 8x8 matrix of an x4 load, r8 = its row.
    // Within a half of w / qg the k-step only moves bits 5 and 6 of the address, which the tile bases leave clear.
    static_assert(SM::STAGE % 128 == 0 && REC_W % 128 == 0 && REC_QG % 128 == 0 && REC_HALF % 128 == 0,
                  "tile bases must keep address bits 5 and 6 clear");
    const int mi = lane >> 3, r8 = lane & 7;
    const uint32_t a1_lane = wq_off(r8 + (mi & 1) * 8, (mi >> 1) * 8);                 // [w;qg]: rows tok, cols k
    const uint32_t a2_lane = kg_off((mi >> 1) * 8, (mi & 1) * 8 + r8);                 // kg^T: rows k, cols tok
    const uint32_t a3_off = REC_AQK + aq_off(r8 + (mi & 1) * 8, (mi >> 1) * 8);        // Aqk: rows i, cols j
    auto wq_at = [](uint32_t base, int ks) { return (base ^ ((ks & 3) << 5)) + (ks >> 2) * REC_HALF; };
    const uint32_t x_off = REC_XBH + xb_off(r8 + (mi & 1) * 8, (mi >> 1) * 8);         // Xb: rows i, cols j
    auto v_at = [&](int nv) { return REC_SHARED_BYTES + v_off(lane & 15, (v0 + nv * 8) & 63); };   // v: rows tok, 8 columns
    __nv_bfloat16* const ob = STATE_ONLY ? nullptr : p.o + b * p.o_s[0] + tok0 * p.o_s[1] + h * p.o_s[2] + v0 + tq * 2;
    const bool use_u = PAIR || (pair_rt ? plane == 1 : !(STATE_ONLY && p.zero_u));

    uint32_t aw[8][4], aq[8][4];     // A fragments of w and qg (one per 16-wide k-step)
    float dk[8][2];                  // decay of the rows k = 16m+gq and 16m+gq+8
    float u[NVT][4];                 // Xb v
    float oa[NVT][4];                // output tile

    uint32_t xh[4], xl[4], bu[RT][2];
    auto load_xv = [&](uint32_t sp) {
      ldsm_x4(sp + x_off, xh[0], xh[1], xh[2], xh[3]);
      ldsm_x4(sp + x_off + (REC_XBL - REC_XBH), xl[0], xl[1], xl[2], xl[3]);
#pragma unroll
      for (int nv = 0; nv < RT; ++nv) ldsm_x2_t(sp + v_at(nv), bu[nv][0], bu[nv][1]);
    };
    auto make_u = [&]() {
#pragma unroll
      for (int nv = 0; nv < NVT; ++nv) {
        float (&acc)[4] = u[nv];
        if (PAIR && nv == 0) {
          acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
          continue;
        }
        mma_bf16_z(acc, xh, bu[PAIR ? 0 : nv][0], bu[PAIR ? 0 : nv][1]);
        mma_bf16_v(acc, xl, bu[PAIR ? 0 : nv][0], bu[PAIR ? 0 : nv][1]);
        if (STATE_ONLY && !PAIR) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] = use_u ? acc[e] : 0.f;
        }
      }
    };
    auto load_dec = [&](uint32_t sp, int j) {
      const float4 d = lds_f32x4(sp + REC_DEC2 + j * 128 + gq * 16);
      dk[2 * j][0] = d.x; dk[2 * j][1] = d.y; dk[2 * j + 1][0] = d.z; dk[2 * j + 1][1] = d.w;
    };

    bool failed = false;
    if (!h0_ok) {
      if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_PEER_TIMEOUT); }
      failed = true;
    } else if (!__all_sync(0xffffffffu, mbar_wait_bounded(full0, 0, sAbort))) {
      if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2_FULL_TIMEOUT); }
      failed = true;
    } else {
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        ldsm_x4(wq_at(sbase + a1_lane, ks) + REC_W, aw[ks][0], aw[ks][1], aw[ks][2], aw[ks][3]);
        if (!STATE_ONLY)
          ldsm_x4(wq_at(sbase + a1_lane, ks) + REC_QG, aq[ks][0], aq[ks][1], aq[ks][2], aq[ks][3]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) load_dec(sbase, j);
      load_xv(sbase);
      if (STATE_ONLY) make_u();
    }

    // A step is two straight runs of instructions around one branch (the slow path of the wait for the next record),
    // which is what the compiler schedules well: the last step, which has no next record to wait for and to load from, is an
    // instantiation of its own, the output stores are predicated and the shared-memory loads are pinned.  The stage goes
    // round as an address and a parity carried from step to step; worked out from n instead, a step takes 6 % longer, except in
    // the transform pairs, where the compiler does better with n.  K2 alone (us), before the address was carried and v_new and
    // o were summed in pairs, after that, and now that u is worked out here and the decay comes in four loads instead of 16:
    // T8192 H32 249 / 242 / 230, H8 185 / 172 / 173, T4096 H8 96.8 / 90.7 / 91.0; state-only T8192 H32 183 / 181 / 185, H8 148 /
    // 146 / 150; transform pairs T8192 H16 181 / 177 / 183, H32 258 / 260 / 263.
    __nv_bfloat16* o_at = STATE_ONLY ? nullptr : ob + static_cast<int64_t>(gq) * p.o_s[1];
    const int64_t o_step = BT * p.o_s[1], o_8 = 8 * p.o_s[1];
    int left = Tlen;
    uint32_t at = sbase, at_bar = full0, at_ph = 0;   // the chunk's stage, its full barrier and that barrier's parity
    auto step = [&](auto more_c, int n) {
      constexpr bool MORE = decltype(more_c)::value;   // chunk n + 1 exists
      const int s = n % K2_STAGES, s1 = (n + 1) % K2_STAGES;
      const bool wrap = at == sbase + (K2_STAGES - 1) * SM::STAGE;
      const uint32_t sp = PAIR ? sbase + s * SM::STAGE : at, bar = PAIR ? full0 + s * 8 : at_bar;
      const uint32_t sp1 = PAIR ? sbase + s1 * SM::STAGE : wrap ? sbase : at + SM::STAGE;
      const uint32_t bar1 = PAIR ? full0 + s1 * 8 : wrap ? full0 : at_bar + 8;
      const uint32_t ph1 = PAIR ? ((n + 1) / K2_STAGES) & 1 : wrap ? at_ph ^ 1 : at_ph;
      const uint32_t t2 = sp + a2_lane, t1n = sp1 + a1_lane;

      // B fragments of bf16(hT) (pre-chunk state): accumulator fragment -> pack -> 8x8 transpose
      uint32_t bh[8][NVT][2];
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) {
          bh[m][nv][0] = movmatrix_t(pack_bf16(hT[m][nv][0], hT[m][nv][1]));
          bh[m][nv][1] = movmatrix_t(pack_bf16(hT[m][nv][2], hT[m][nv][3]));
        }

      // P1 (two accumulator sets: even / odd k-steps), carrying the kg fragment loads of this
      // step and the decay of the fp32 state
      float pw[2][NVT][4], pq[2][NVT][4];
      uint32_t kgh[8][4], kgl[8][4];
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) {
          if (ks < 2) mma_bf16_z(pw[ks & 1][nv], aw[ks], bh[ks][nv][0], bh[ks][nv][1]);
          else mma_bf16_v(pw[ks & 1][nv], aw[ks], bh[ks][nv][0], bh[ks][nv][1]);
        }
        ldsm_x4(t2 + ks * 256 + REC_KGH, kgh[ks][0], kgh[ks][1], kgh[ks][2], kgh[ks][3]);
        if (!STATE_ONLY) {
#pragma unroll
          for (int nv = 0; nv < NVT; ++nv) {
            if (ks < 2) mma_bf16_z(pq[ks & 1][nv], aq[ks], bh[ks][nv][0], bh[ks][nv][1]);
            else mma_bf16_v(pq[ks & 1][nv], aq[ks], bh[ks][nv][0], bh[ks][nv][1]);
          }
        }
        ldsm_x4(t2 + ks * 256 + REC_KGL, kgl[ks][0], kgl[ks][1], kgl[ks][2], kgl[ks][3]);
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) {
          const float2 lo = __fmul2_rn(make_float2(hT[ks][nv][0], hT[ks][nv][1]), make_float2(dk[ks][0], dk[ks][0]));
          const float2 hi = __fmul2_rn(make_float2(hT[ks][nv][2], hT[ks][nv][3]), make_float2(dk[ks][1], dk[ks][1]));
          hT[ks][nv][0] = lo.x; hT[ks][nv][1] = lo.y; hT[ks][nv][2] = hi.x; hT[ks][nv][3] = hi.y;
        }
      }
      // u under the last products of P1 (T8192 H32 K2 230 us; at the end of the step before 237).  Without outputs there is
      // less to hide it under: at the end of the step before, its operands earlier still (state-only T8192 H8 150; here 152)
      if (!STATE_ONLY) make_u();
      // probed here and looked at when the answer is needed: a probe and the vote on it take 126 cycles
      const bool next_ready = MORE ? mbar_test_wait(bar1, ph1) : true;
      uint32_t ah3[4], al3[4];
      if (!STATE_ONLY) {
        ldsm_x4(sp + a3_off, ah3[0], ah3[1], ah3[2], ah3[3]);
        ldsm_x4(sp + a3_off + (REC_AQL - REC_AQK), al3[0], al3[1], al3[2], al3[3]);
      }

      // v_new (fp32, accumulator layout: rows tok, cols v) and its hi/lo B fragments
      uint32_t bvh[NVT][2], bvl[NVT][2];
#pragma unroll
      for (int nv = 0; nv < NVT; ++nv) {
        uint32_t h01, l01, h23, l23;
        split_pack_sum(&u[nv][0], &pw[0][nv][0], &pw[1][nv][0], h01, l01);
        split_pack_sum(&u[nv][2], &pw[0][nv][2], &pw[1][nv][2], h23, l23);
        bvh[nv][0] = movmatrix_t(h01); bvh[nv][1] = movmatrix_t(h23);
        bvl[nv][0] = movmatrix_t(l01); bvl[nv][1] = movmatrix_t(l23);
      }

      // release the stage only when its fragment loads have landed: shared-memory loads of a warp
      // return in issue order, so reading a register of the last-issued ones makes the warp wait
      // for all of them
      {
        uint32_t landed = kgh[7][0] ^ kgl[7][0];
        if (!STATE_ONLY) landed ^= ah3[0] ^ al3[0];
        asm volatile("" ::"r"(landed) : "memory");
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar + K2_STAGES * 8);
      if (MORE && !__all_sync(0xffffffffu, next_ready)) {
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar1, ph1, sAbort))) {
          if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2_FULL_TIMEOUT); }
          failed = true;
          return;
        }
      }

      // P2: hT += kg^T v_new  (hi*hi, then hi*lo(v), then lo(kg)*hi: three passes over independent
      // tiles), carrying the next step's operand loads, and P3: o = scale * (qg hT) +
      // Aqk v_new
#pragma unroll
      for (int m = 0; m < 8; ++m) {
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) mma_bf16_v(hT[m][nv], kgh[m], bvh[nv][0], bvh[nv][1]);
        if (MORE) ldsm_x4(wq_at(t1n, m) + REC_W, aw[m][0], aw[m][1], aw[m][2], aw[m][3]);
      }
#pragma unroll
      for (int m = 0; m < 8; ++m) {
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) mma_bf16_v(hT[m][nv], kgh[m], bvl[nv][0], bvl[nv][1]);
        if (MORE && (m & 1)) load_dec(sp1, m >> 1);
        if (MORE && STATE_ONLY && m == 4) load_xv(sp1);
      }
#pragma unroll
      for (int m = 0; m < 8; ++m) {
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) mma_bf16_v(hT[m][nv], kgl[m], bvh[nv][0], bvh[nv][1]);
        if (MORE && !STATE_ONLY) ldsm_x4(wq_at(t1n, m) + REC_QG, aq[m][0], aq[m][1], aq[m][2], aq[m][3]);
        if (!STATE_ONLY && (m == 0 || m == 3 || m == 6)) {
#pragma unroll
          for (int nv = 0; nv < NVT; ++nv) {
            if (m == 0) {
#pragma unroll
              for (int e = 0; e < 4; e += 2) {
                const float2 x = __fmul2_rn(make_float2(p.scale, p.scale), __fadd2_rn(make_float2(pq[0][nv][e], pq[0][nv][e + 1]),
                                                                                      make_float2(pq[1][nv][e], pq[1][nv][e + 1])));
                oa[nv][e] = x.x; oa[nv][e + 1] = x.y;
              }
              mma_bf16_v(oa[nv], ah3, bvh[nv][0], bvh[nv][1]);
            }
            if (m == 3) mma_bf16_v(oa[nv], ah3, bvl[nv][0], bvl[nv][1]);
            if (m == 6) mma_bf16_v(oa[nv], al3, bvh[nv][0], bvh[nv][1]);
          }
        }
      }

      if (!STATE_ONLY) {   // rows past the end of a partial last chunk stay as they are
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv) {
          stg_u32_if(o_at + nv * 8, pack_bf16(oa[nv][0], oa[nv][1]), gq < left);
          stg_u32_if(o_at + o_8 + nv * 8, pack_bf16(oa[nv][2], oa[nv][3]), gq + 8 < left);
        }
        o_at += o_step;
        left -= BT;
      }
      if (MORE) {
        if (!STATE_ONLY) load_xv(sp1);
        else make_u();
        if (!PAIR) { at = sp1; at_bar = bar1; at_ph = ph1; }
      }
    };
    // (With `&& !failed` as the loop's condition the compiler's schedule of a step is 10 to 15 % longer.)
    if (!failed) {
      if constexpr (PAIR) {   // (the compiler's schedule of a step: T8192 H32 264 us, 272 in the other spelling)
        int n = 0;
        for (; n + 1 < NT; ++n) {
          step(std::true_type{}, n);
          if (failed) break;
        }
        if (n + 1 >= NT) step(std::false_type{}, n);
      } else {
        for (int n = 0; n + 1 < NT; ++n) {
          step(std::true_type{}, n);
          if (failed) break;
        }
        if (!failed) step(std::false_type{}, NT - 1);
      }
    }

    if (!failed && (p.ht != nullptr || (PAIR && p.push_on))) {
      float* ht = (PAIR && p.push_on)
                      ? p.push_dst[bh / p.push_hp] + p.push_dst_offset + static_cast<size_t>(2 * (bh % p.push_hp)) * D * D
                      : p.ht + static_cast<size_t>(PAIR ? 2 * bh : chain) * D * D;
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int nv = 0; nv < NVT; ++nv)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (PAIR) ht[(static_cast<size_t>(nv) * D + v0 + tq * 2 + (e & 1)) * D + m * 16 + gq + (e >> 1) * 8] = hT[m][nv][e];
            else if (p.k_first) ht[(m * 16 + gq + (e >> 1) * 8) * D + v0 + nv * 8 + tq * 2 + (e & 1)] = hT[m][nv][e];
            else ht[(v0 + nv * 8 + tq * 2 + (e & 1)) * D + m * 16 + gq + (e >> 1) * 8] = hT[m][nv][e];
    }
  }

  __syncthreads();
  if (PAIR && p.push_on && tid == 0 && *sAbort == 0) {
    // the tiles went into another rank's receive buffer: the CTA barrier has put every warp's stores before
    // this count; the CTA that counts last for a destination raises its flag behind one system-scope fence
    const int owner = bh / p.push_hp;
    __threadfence();
    const int done = atomicAdd(p.push_counter + owner, 1);
    __threadfence();
    if (done == p.push_ctas_per_dst - 1) {
      p.push_counter[owner] = 0;
      __threadfence_system();
      st_release_sys(p.push_flag[owner], p.push_epoch);
    }
  }
  if (*sAbort != 0 && tid == 0) {
    // give copies that are still in flight a bounded chance to land before the CTA's
    // shared memory is released
    const int issued = *sIssued;
    for (int n = max(0, issued - K2_STAGES); n < issued; ++n)
      mbar_wait_bounded(full0 + (n % K2_STAGES) * 8, (n / K2_STAGES) & 1, nullptr);
  }
  if (p.progress != nullptr) grid_dep_wait();   // this grid ends after K1
}

template <int CW, int NVT, bool STATE_ONLY, bool PAIR = false, bool ORD = false, int K2_STAGES = 4>
static cudaError_t launch_k2_t(const K2Params& p, cudaStream_t stream) {
  constexpr int RT = PAIR ? 1 : NVT;
  constexpr int smem_bytes = K2Smem<K2_STAGES>::TOTAL;
  static std::atomic<bool> configured[64];   // set after the attributes, also for other threads
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kda_k2_kernel<CW, NVT, STATE_ONLY, PAIR, ORD, K2_STAGES>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes > ONE_CTA_SMEM ? smem_bytes : ONE_CTA_SMEM);
    if (e != cudaSuccess) return e;
    // the carve-out of K1, so that an SM can hold CTAs of both
    e = cudaFuncSetAttribute(kda_k2_kernel<CW, NVT, STATE_ONLY, PAIR, ORD, K2_STAGES>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int nblocks = (p.n_chains > 0 ? p.n_chains : (p.seq_table != nullptr ? p.n_seqs : p.B) * p.H) * (D / (CW * RT * 8));
  return launch_dep(kda_k2_kernel<CW, NVT, STATE_ONLY, PAIR, ORD, K2_STAGES>, nblocks, (CW + 1) * 32, k2_smem(p, smem_bytes), stream, p.pdl, p);
}

cudaError_t launch_k2n(const K2Params& p, int vsplit, int ntile, bool state_only, cudaStream_t stream) {
  // vsplit CTAs per head, ntile 8-row tiles per warp  =>  16 / (vsplit * ntile) consumer warps per CTA
  // (at most 4: a fifth warp is the producer, and CTAs of more than 8 warps lose registers per thread)
  if (p.long_ring > 4 && !state_only && ntile == 1) {
    if (vsplit == 4 && p.long_ring == 8) return launch_k2_t<4, 1, false, false, false, 8>(p, stream);
    if (vsplit == 8) return p.long_ring > 5 ? launch_k2_t<2, 1, false, false, false, 6>(p, stream) : launch_k2_t<2, 1, false, false, false, 5>(p, stream);
    if (vsplit == 16) return p.long_ring > 5 ? launch_k2_t<1, 1, false, false, false, 6>(p, stream) : launch_k2_t<1, 1, false, false, false, 5>(p, stream);
  }
#define KDA_K2_CASE(VS, NT_, CW_)                                                                  \
  if (vsplit == VS && ntile == NT_)                                                                \
    return state_only ? launch_k2_t<CW_, NT_, true>(p, stream)                                     \
           : p.by_length ? launch_k2_t<CW_, NT_, false, false, true>(p, stream)                    \
                         : launch_k2_t<CW_, NT_, false>(p, stream);
  KDA_K2_CASE(4, 1, 4)
  KDA_K2_CASE(8, 1, 2)
  KDA_K2_CASE(16, 1, 1)
#undef KDA_K2_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_k2n_pair(const K2Params& p0, int vsplit, cudaStream_t stream) {
  // the transform-pair pass: two recurrences over the same eight rows per warp, 16 / vsplit consumer warps per CTA
  K2Params p = p0;
  p.push_ctas_per_dst = p.push_hp * vsplit;   // vsplit CTAs share a chain
  switch (vsplit) {
    case 4: return launch_k2_t<4, 2, true, true>(p, stream);
    case 8: return launch_k2_t<2, 2, true, true>(p, stream);
    case 16: return launch_k2_t<1, 2, true, true>(p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kda
