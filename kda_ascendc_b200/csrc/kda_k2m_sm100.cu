// K2, "m16" organisation: the state rows on the MMA M dimension, 16 rows of h per warp.
//
// Same recurrence as kda_k2_sm100.cu (reference: src/kda_bt16/kernels.py:187-302,
// tests/test_torch_reference.py:175-194), evaluated in the transposed form
//   P1: [-h w^T | o^T] = h [-w^T | qg^T]    (M = 16 rows v, N = 16+16 tokens, K = 128)  32 MMAs
//   u^T = v^T Xb^T                          (M = 16 rows v, N = 16 tokens, K = 16)      4 MMAs
//   P2: h += v_new^T kg                     (M = 16 rows v, N = 128 k, K = 16 tokens)  3 x 16 MMAs
//   P3: o^T += v_new^T Aqk^T                (M = 16 rows v, N = 16 tokens, K = 16)     6 MMAs
// The state tile h[16 v][128 k] lives in registers as fp32 accumulator fragments; the
// accumulator layout of two adjacent 8-column tiles IS the A-operand layout of a 16x16 tile,
// so bf16(h) and v_new feed the next product by a register pack alone.  The shared operands
// (w, qg, kg, Aqk) are the B side here: a B fragment is half the size of an A fragment, so this
// organisation reads half as many shared-memory bytes per MMA as the "n8" one, at the price of
// a chain twice as long per warp (90 MMAs per step).  Per state row it needs fewer instructions
// (no transposes, operand loads shared by 16 rows), which makes it the better choice once
// there are more 8-row tiles than SM sub-partitions (more than about 37 (batch, head) chains).
//
// Loads are interleaved with the MMA sequences so that their latency is covered (an m16n8k16
// holds the sub-partition's issue port for 8 cycles; the step time is 8 x MMAs + 2 x the other
// instructions): P1 carries its own rolling B-fragment loads,
// the decay row and the kg(hi) fragments; P2's first two passes carry kg(lo), its last pass the
// next step's first fragments; the output tile is transposed through 512 bytes of a warp's own
// (stmatrix) and leaves one step late, 16 bytes a lane, as whole 32-byte sectors (four 4-byte stores behind movmatrix before:
// K2 alone T4096 H64 172 -> 167 us, the forward T8192 H32 with K2 on SMs of its own 381 -> 363), through a pointer that is carried
// along (worked out from the chunk number in front of every step: 162 instead of 155, 342 instead of 327).  The last step, which has no next record, is an instantiation of its own, and the next record's barrier is
// probed a pass ahead, so that one condition (the slow path of that wait) cuts a step behind the store of the previous
// output.  P1's sums run over even and odd k-steps apart, as in the 8-row form, so that both forms give the same bits (T8192
// H32 298 -> 303 us).  K2 alone with conditions around the loads and now: T4096 H64 201 -> 172 us, T2048 H32 CTA-split in four 90 -> 79,
// state-only T4096 H64 157 -> 130; one chunk, H32 in four 4.8 -> 4.4.  u from eight 4-byte loads of the record and from
// three ldmatrix and four MMAs, now: T4096 H64 167 -> 162, state-only 130 -> 122, T8192 H32 298 -> 288.  Producer warp, stage ring, bounded waits: as in kda_k2_sm100.cu.
#include <type_traits>

#include "kda_common.cuh"
#include "kda_kernels.h"

namespace kda {

// STAGES: 8 on an SM of its own beside K1, which holds up the records now and then (T8192 H32 363 -> 355 us); else 4
template <int CW, int STAGES>
struct K2mSmem {   // a CTA's columns of v lie in one half
  static constexpr int STAGE = REC_SHARED_BYTES + REC_V_HALF;
  static constexpr int BARS = STAGES * STAGE;
  static constexpr int FLAG = BARS + 2 * STAGES * 8;
  static constexpr int OST = FLAG + 16;              // a warp's output tile: [16 tok][16 v] bf16
  static constexpr int TOTAL = OST + CW * 512;
  static_assert(OST % 16 == 0, "the output tile is written and read 16 bytes at a time");
};

// MINB = CTAs that must fit on one SM.  With 2 (register cap 168) eight consumer warps share an
// SM; that pays as soon as there are more CTAs than SMs (measured: B1 T8192 H96 765 -> 677 us),
// while a grid that fits in one wave is faster with the uncapped registers.
// ORD: packed sequences, longest first
template <int CW, bool STATE_ONLY, int MINB, bool ORD = false, int K2M_STAGES = 4>
__global__ void __launch_bounds__((CW + 1) * 32, MINB) kda_k2m_kernel(const K2Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using SM = K2mSmem<CW, K2M_STAGES>;
  constexpr int NV = 8 / CW;            // CTAs per (batch, head)
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int chain = ORD ? chain_by_length(p.seq_table, p.n_seqs, p.H, blockIdx.x / NV + p.chain0) : blockIdx.x / NV + p.chain0;
  const bool pair = STATE_ONLY && p.pair_mode != 0;
  const int bh = pair ? (chain >> 1) : chain;      // the (batch, head) whose records are walked
  const int plane = pair ? (chain & 1) : 1;        // pair mode: 0 = transition matrix, 1 = offset
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
    if (ORD && NT < p.long_len) {   // left to the tensor-memory form, which takes the end of K1 from this kernel
      grid_dep_wait();
      return;
    }
  }

  const uint32_t sbase = smem_u32(smem);
  const uint32_t full0 = sbase + SM::BARS;
  const uint32_t empty0 = full0 + K2M_STAGES * 8;
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + SM::FLAG);
  volatile int* sIssued = sAbort + 1;

  if (tid == 0) {
    for (int s = 0; s < K2M_STAGES; ++s) {
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
      if (ORD && p.long_len > 0) grid_dep_launch();
      int gate = 0;                                 // beside K1: the first chunk of the next window
      for (int n = 0; n < NT; ++n) {
        const int s = n % K2M_STAGES;
        if (p.progress != nullptr && n == gate) {
          if (!window_wait_bounded(p.progress + n / p.win_chunks, min(p.win_chunks, NT - n) * p.B * p.H, sAbort)) {
            if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K1_WINDOW_TIMEOUT); }
            break;
          }
          gate += p.win_chunks;
        }
        if (n >= K2M_STAGES) {
          if (!mbar_wait_bounded(empty0 + s * 8, ((n / K2M_STAGES) - 1) & 1, sAbort)) {
            if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2_EMPTY_TIMEOUT); }
            break;
          }
        }
        const uint8_t* rec = rec_bh + static_cast<size_t>(n) * REC_BYTES;
        const uint32_t dst = sbase + s * SM::STAGE;
        mbar_arrive_expect_tx(full0 + s * 8, SM::STAGE);
        bulk_g2s(dst, rec, REC_SHARED_BYTES, full0 + s * 8);
        bulk_g2s(dst + REC_SHARED_BYTES, rec + REC_V + (vs * CW * 16 >> 6) * REC_V_HALF, REC_V_HALF, full0 + s * 8);
        *sIssued = n + 1;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------ consumers ------------------------------
    const int gq = lane >> 2, tq = lane & 3;
    const int vrow0 = (vs * CW + warp) * 16;
    // hs[nt][e]: v = vrow0 + gq (+8 for e >= 2), k = 8nt + 2tq + (e & 1)
    float hs[16][4];
    bool h0_ok = true;
    if (pair) {
#pragma unroll
      for (int nt = 0; nt < 16; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          hs[nt][e] = (plane == 0 && (vrow0 + gq + (e >> 1) * 8) == (nt * 8 + tq * 2 + (e & 1))) ? 1.f : 0.f;
    } else if (p.h0 != nullptr) {
      if (!STATE_ONLY && p.h0_n_flags > 0) {   // the entry state comes from other GPUs: wait for their flags (the producer warp is already loading records)
        int ok = 1;
        if (lane == 0)
          for (int i = 0; i < p.h0_n_flags; ++i) ok &= flag_wait_bounded(p.h0_flags + i, p.h0_epoch) ? 1 : 0;
        h0_ok = __shfl_sync(0xffffffffu, ok, 0) != 0;
      }
      const float* h0 = p.h0 + static_cast<size_t>(bh) * D * D;
#pragma unroll
      for (int nt = 0; nt < 16; ++nt) {
        if (p.k_first) {
          const float* c0 = h0 + (nt * 8 + tq * 2) * D + vrow0 + gq;
          hs[nt][0] = c0[0]; hs[nt][1] = c0[D]; hs[nt][2] = c0[8]; hs[nt][3] = c0[D + 8];
        } else {
          const float2 a = *reinterpret_cast<const float2*>(h0 + (vrow0 + gq) * D + nt * 8 + tq * 2);
          const float2 c = *reinterpret_cast<const float2*>(h0 + (vrow0 + gq + 8) * D + nt * 8 + tq * 2);
          hs[nt][0] = a.x; hs[nt][1] = a.y; hs[nt][2] = c.x; hs[nt][3] = c.y;
        }
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < 16; ++nt) hs[nt][0] = hs[nt][1] = hs[nt][2] = hs[nt][3] = 0.f;
    }

    // per-lane ldmatrix address components (constant across steps)
    const int mi = lane >> 3, r8 = lane & 7;   // the 8x8 matrix of an x4 load, and its row, that this lane addresses
    // w, qg: [N=tok][K=k]; within a half the k-step moves bits 5 and 6 of the address, which the tile bases leave clear
    const uint32_t b1_lane = wq_off(r8 + (mi >> 1) * 8, (mi & 1) * 8);
    const uint32_t b2_lane = kg_off((mi & 1) * 8, (mi >> 1) * 8 + r8);               // kg: [N=k][K=tok]
    const uint32_t b3_off = REC_AQK + aq_off((mi >> 1) * 8 + r8, (mi & 1) * 8);      // Aqk: [N=i][K=j]
    const uint32_t x_off = REC_XBH + xb_off((mi >> 1) * 8 + r8, (mi & 1) * 8);       // Xb: [N=i][K=j]
    const uint32_t v_lane = REC_SHARED_BYTES + v_off((mi >> 1) * 8 + r8, (vrow0 + (mi & 1) * 8) & 63);   // v: rows tok, through .trans
    // the output tile: the 16-byte units of tokens 4..7 and 12..15 swapped, so that eight rows of either unit lie in different banks
    auto ost_at = [&](int tok, int unit) { return sbase + SM::OST + warp * 512 + tok * 32 + ((unit ^ ((tok >> 2) & 1)) << 4); };
    const uint32_t ost_put = ost_at((mi >> 1) * 8 + r8, mi & 1), ost_get = ost_at(lane >> 1, lane & 1);
    __nv_bfloat16* const ob = STATE_ONLY ? nullptr : p.o + b * p.o_s[0] + tok0 * p.o_s[1] + h * p.o_s[2] + vrow0 +
                                                     (lane >> 1) * p.o_s[1] + (lane & 1) * 8;
    const bool use_u = pair ? (plane == 1) : !(STATE_ONLY && p.zero_u);

    // rolling B fragments of P1: two k-steps ahead
    uint32_t bw[2][4], bq[2][4];
    float ut[2][4];             // u^T = v^T Xb^T, [token tile]
    uint32_t av[4], xh[4], xl[4];
    float2 dec[16];             // decay of the columns k = 8nt + 2tq, +1 (loaded one step ahead)

    auto load_xv = [&](uint32_t sp) {
      ldsm_x4_t(sp + v_lane, av[0], av[1], av[2], av[3]);
      ldsm_x4(sp + x_off, xh[0], xh[1], xh[2], xh[3]);
      ldsm_x4(sp + x_off + (REC_XBL - REC_XBH), xl[0], xl[1], xl[2], xl[3]);
    };
    auto make_u = [&]() {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        mma_bf16_z(ut[c], av, xh[2 * c], xh[2 * c + 1]);
        mma_bf16_v(ut[c], av, xl[2 * c], xl[2 * c + 1]);
        if (STATE_ONLY) {
#pragma unroll
          for (int e = 0; e < 4; ++e) ut[c][e] = use_u ? ut[c][e] : 0.f;
        }
      }
    };
    auto load_dec = [&](uint32_t spg, int nt0, int nt1) {
#pragma unroll
      for (int nt = nt0; nt < nt1; ++nt) dec[nt] = lds_f32x2(spg + REC_DEC + (nt * 8 + tq * 2) * 4);
    };
    auto load_b1 = [&](uint32_t sp, int ks, int slot) {
      const uint32_t at = ((sp + b1_lane) ^ ((ks & 3) << 5)) + (ks >> 2) * REC_HALF;
      ldsm_x4(at + REC_W, bw[slot][0], bw[slot][1], bw[slot][2], bw[slot][3]);
      if (!STATE_ONLY) ldsm_x4(at + REC_QG, bq[slot][0], bq[slot][1], bq[slot][2], bq[slot][3]);
    };

    bool failed = false;
    if (!h0_ok) {
      if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_PEER_TIMEOUT); }
      failed = true;
    } else if (!__all_sync(0xffffffffu, mbar_wait_bounded(full0, 0, sAbort))) {
      if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2_FULL_TIMEOUT); }
      failed = true;
    } else {
      load_b1(sbase, 0, 0);
      load_b1(sbase, 1, 1);
      load_xv(sbase);
      make_u();
      load_dec(sbase, 0, 16);
    }

    __nv_bfloat16* o_at = ob;   // of the previous chunk
    const int64_t o_step = STATE_ONLY ? 0 : BT * p.o_s[1];
    auto step = [&](auto more_c, int n) {
      constexpr bool MORE = decltype(more_c)::value;   // chunk n + 1 exists
      const int s = n % K2M_STAGES;
      const uint32_t sp = sbase + s * SM::STAGE;
      const int s1 = (n + 1) % K2M_STAGES;
      const uint32_t sp1 = sbase + s1 * SM::STAGE;

      // the previous step's output tile (always a full chunk): 16 bytes of a token row per lane
      if (!STATE_ONLY && n > 0) {
        *reinterpret_cast<uint4*>(o_at) = lds_u32x4(ost_get);
        o_at += o_step;
      }

      // P1 with the A fragments of bf16(h) packed on the fly; carries the decay of the fp32 state,
      // its own rolling B loads and the kg(hi) fragments of this step
      float pw[2][2][4], pq[2][2][4];   // [k-step parity][token tile]: summed as in the 8-row form, so that the bits are the same
      uint32_t kgh[8][4], kgl[8][4];
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t ah[4];
        ah[0] = pack_bf16(hs[2 * ks][0], hs[2 * ks][1]);
        ah[1] = pack_bf16(hs[2 * ks][2], hs[2 * ks][3]);
        ah[2] = pack_bf16(hs[2 * ks + 1][0], hs[2 * ks + 1][1]);
        ah[3] = pack_bf16(hs[2 * ks + 1][2], hs[2 * ks + 1][3]);
        const int sl = ks & 1;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (ks < 2) mma_bf16_z(pw[sl][c], ah, bw[sl][2 * c], bw[sl][2 * c + 1]);
          else mma_bf16_v(pw[sl][c], ah, bw[sl][2 * c], bw[sl][2 * c + 1]);
        }
        if (!STATE_ONLY) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (ks < 2) mma_bf16_z(pq[sl][c], ah, bq[sl][2 * c], bq[sl][2 * c + 1]);
            else mma_bf16_v(pq[sl][c], ah, bq[sl][2 * c], bq[sl][2 * c + 1]);
          }
        }
        if (ks + 2 < 8) load_b1(sp, ks + 2, sl);
        ldsm_x4(sp + b2_lane + REC_KGH + ks * 256, kgh[ks][0], kgh[ks][1], kgh[ks][2], kgh[ks][3]);
        {
          const float2 d0 = dec[2 * ks], d1 = dec[2 * ks + 1];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const float2 dd = half ? d1 : d0;
            float* t = hs[2 * ks + half];
            const float2 lo = __fmul2_rn(make_float2(t[0], t[1]), dd), hi = __fmul2_rn(make_float2(t[2], t[3]), dd);
            t[0] = lo.x; t[1] = lo.y; t[2] = hi.x; t[3] = hi.y;
          }
        }
      }

      // v_new^T (fp32, accumulator layout: rows v, cols tok) and its hi/lo A fragments
      uint32_t avh[4], avl[4];
      auto vn = [&](int c, int e) { return ut[c][e] + (pw[0][c][e] + pw[1][c][e]); };
      split_pack(vn(0, 0), vn(0, 1), avh[0], avl[0]);
      split_pack(vn(0, 2), vn(0, 3), avh[1], avl[1]);
      split_pack(vn(1, 0), vn(1, 1), avh[2], avl[2]);
      split_pack(vn(1, 2), vn(1, 3), avh[3], avl[3]);

      // P2 pass 1 (hi * hi), carrying the kg(lo) fragments
#pragma unroll
      for (int np = 0; np < 8; ++np) {
        mma_bf16_v(hs[2 * np], avh, kgh[np][0], kgh[np][1]);
        mma_bf16_v(hs[2 * np + 1], avh, kgh[np][2], kgh[np][3]);
        ldsm_x4(sp + b2_lane + REC_KGL + np * 256, kgl[np][0], kgl[np][1], kgl[np][2], kgl[np][3]);
      }
      uint32_t ba[4], bl[4];
      if (!STATE_ONLY) {
        ldsm_x4(sp + b3_off, ba[0], ba[1], ba[2], ba[3]);
        ldsm_x4(sp + b3_off + (REC_AQL - REC_AQK), bl[0], bl[1], bl[2], bl[3]);
      }
      const bool next_ready = MORE ? mbar_test_wait(full0 + s1 * 8, ((n + 1) / K2M_STAGES) & 1) : true;
      // P2 pass 2 (lo(v) * hi)
#pragma unroll
      for (int np = 0; np < 8; ++np) {
        mma_bf16_v(hs[2 * np], avl, kgh[np][0], kgh[np][1]);
        mma_bf16_v(hs[2 * np + 1], avl, kgh[np][2], kgh[np][3]);
      }

      // every shared-memory operand of this stage has been requested; once the loads have landed
      // (they are consumed below) the stage is released and the next one checked

      // P2 pass 3 (hi * lo(kg)), with P3 and the next step's first operands in its gaps
      float oa[2][4];
      if (!STATE_ONLY) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) oa[j][e] = p.scale * (pq[0][j][e] + pq[1][j][e]);
      }
#pragma unroll
      for (int np = 0; np < 8; ++np) {
        mma_bf16_v(hs[2 * np], avh, kgl[np][0], kgl[np][1]);
        mma_bf16_v(hs[2 * np + 1], avh, kgl[np][2], kgl[np][3]);
        if (!STATE_ONLY) {
          if (np == 0) { mma_bf16_v(oa[0], avh, ba[0], ba[1]); mma_bf16_v(oa[1], avh, ba[2], ba[3]); }
          if (np == 2) { mma_bf16_v(oa[0], avl, ba[0], ba[1]); mma_bf16_v(oa[1], avl, ba[2], ba[3]); }
          if (np == 4) { mma_bf16_v(oa[0], avh, bl[0], bl[1]); mma_bf16_v(oa[1], avh, bl[2], bl[3]); }
        }
        if (np == 3) {
          // release the stage only when its fragment loads have landed: shared-memory loads of a
          // warp return in issue order, so reading a register of the last-issued ones makes the
          // warp wait for all of them
          uint32_t landed = kgl[7][0];
          if (!STATE_ONLY) landed ^= ba[0] ^ bl[0];
          asm volatile("" ::"r"(landed) : "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(empty0 + s * 8);
          if (MORE && !__all_sync(0xffffffffu, next_ready)) {
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(full0 + s1 * 8, ((n + 1) / K2M_STAGES) & 1, sAbort))) {
              // the loads below are made all the same, out of a stage that a copy may still be writing: nothing of them
              // is used, neither this step's output nor the state is stored
              if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2_FULL_TIMEOUT); }
              failed = true;
            }
          }
        }
        if (MORE) {
          if (np == 4) { load_b1(sp1, 0, 0); load_dec(sp1, 0, 6); }
          if (np == 5) { load_b1(sp1, 1, 1); load_dec(sp1, 6, 12); }
          if (np == 6) { load_xv(sp1); load_dec(sp1, 12, 16); }
          if (np == 7) make_u();
        }
      }

      // output tile: o^T fragments (rows v, cols tok) leave transposed: [tok][16 v]
      if (!STATE_ONLY) {
        __syncwarp();   // the previous tile has been read
        stsm_x4_t(ost_put, pack_bf16(oa[0][0], oa[0][1]), pack_bf16(oa[0][2], oa[0][3]), pack_bf16(oa[1][0], oa[1][1]),
                  pack_bf16(oa[1][2], oa[1][3]));
        __syncwarp();
      }
    };
    for (int n = 0; n + 1 < NT && !failed; ++n) step(std::true_type{}, n);
    if (!failed) step(std::false_type{}, NT - 1);

    // the last chunk's output tile (it may be a partial chunk)
    if (!STATE_ONLY && !failed) {
      const int tok = (NT - 1) * BT;   // (not by o_at: kept alive so far it costs the steps 2 %)
      if (tok + (lane >> 1) < Tlen) *reinterpret_cast<uint4*>(ob + static_cast<int64_t>(tok) * p.o_s[1]) = lds_u32x4(ost_get);
    }

    if (!failed && p.ht != nullptr) {
      float* ht = p.ht + static_cast<size_t>(chain) * D * D;
#pragma unroll
      for (int nt = 0; nt < 16; ++nt) {
        if (p.k_first && !pair) {
          float* c0 = ht + (nt * 8 + tq * 2) * D + vrow0 + gq;
          c0[0] = hs[nt][0]; c0[D] = hs[nt][1]; c0[8] = hs[nt][2]; c0[D + 8] = hs[nt][3];
        } else {
          *reinterpret_cast<float2*>(ht + (vrow0 + gq) * D + nt * 8 + tq * 2) = make_float2(hs[nt][0], hs[nt][1]);
          *reinterpret_cast<float2*>(ht + (vrow0 + gq + 8) * D + nt * 8 + tq * 2) = make_float2(hs[nt][2], hs[nt][3]);
        }
      }
    }
  }

  __syncthreads();
  if (*sAbort != 0 && tid == 0) {
    const int issued = *sIssued;
    for (int n = max(0, issued - K2M_STAGES); n < issued; ++n)
      mbar_wait_bounded(full0 + (n % K2M_STAGES) * 8, (n / K2M_STAGES) & 1, nullptr);
  }
  if (p.progress != nullptr) grid_dep_wait();   // this grid ends after K1
}

template <int CW, bool STATE_ONLY, int MINB, bool ORD = false, int K2M_STAGES = 4>
static cudaError_t launch_k2m_t(const K2Params& p, int nblocks, cudaStream_t stream) {
  constexpr int smem_bytes = K2mSmem<CW, K2M_STAGES>::TOTAL;
  static std::atomic<bool> configured[64];   // set after the attributes, also for other threads
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kda_k2m_kernel<CW, STATE_ONLY, MINB, ORD, K2M_STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes > ONE_CTA_SMEM ? smem_bytes : ONE_CTA_SMEM);
    if (e != cudaSuccess) return e;
    // K1's carve-out: CTAs of this kernel move onto an SM while K1 still leaves it (and two of them fit)
    e = cudaFuncSetAttribute(kda_k2m_kernel<CW, STATE_ONLY, MINB, ORD, K2M_STAGES>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return launch_dep(kda_k2m_kernel<CW, STATE_ONLY, MINB, ORD, K2M_STAGES>, nblocks, (CW + 1) * 32, k2_smem(p, smem_bytes), stream, p.pdl, p);
}

template <int CW, bool STATE_ONLY>
static cudaError_t launch_k2m_c(const K2Params& p, cudaStream_t stream) {
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64) return cudaErrorInvalidDevice;
  if (sms[dev] == 0) {
    cudaError_t e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
  }
  const int nblocks = (p.n_chains > 0 ? p.n_chains : (p.seq_table != nullptr ? p.n_seqs : p.B) * p.H) * (8 / CW);
  if constexpr (CW == 4 && !STATE_ONLY)
    if (p.long_ring == 8) return launch_k2m_t<4, false, 1, false, 8>(p, nblocks, stream);
  if (CW == 4 && nblocks > sms[dev]) return launch_k2m_t<CW, STATE_ONLY, 2>(p, nblocks, stream);
  if constexpr (CW == 4 && !STATE_ONLY)   // packed: the tail of a tensor-memory launch, or the long sequences in front of one
    if (p.by_length) return launch_k2m_t<4, false, 1, true>(p, nblocks, stream);
  return launch_k2m_t<CW, STATE_ONLY, 1>(p, nblocks, stream);
}

cudaError_t launch_k2m(const K2Params& p, int vsplit, bool state_only, cudaStream_t stream) {
  switch (vsplit) {
    case 2: return state_only ? launch_k2m_c<4, true>(p, stream) : launch_k2m_c<4, false>(p, stream);
    case 4: return state_only ? launch_k2m_c<2, true>(p, stream) : launch_k2m_c<2, false>(p, stream);
    case 8: return state_only ? launch_k2m_c<1, true>(p, stream) : launch_k2m_c<1, false>(p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kda
