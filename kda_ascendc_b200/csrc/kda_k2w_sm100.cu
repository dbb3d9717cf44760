// K2 for wide records: the state recurrence in steps of 64 tokens on the tensor cores (tcgen05 + TMEM).  sm_100a.
//
// Replaces kda_bt16_kernel_k2 of the reference (src/kda_bt16/kernels.py:187-302); the arithmetic per chunk is
//   r = beta v - kb S^T ;  o = qg S^T + ax r ;  S = S diag(dec) + r^T kx          (kda_wide.cuh)
// One CTA owns all 128 state rows of one chain (or of one segment of it).  The fp32 state stays in registers, 64 per
// thread; lanes of tensor memory are the state rows v.  Per chunk:
//   P1  D1[v][0..63]   = bf16(S) . kb^T     8 x M128 N64 K16, A from TMEM          -> r
//       D1[v][64..127] = bf16(S) . qg^T     the same, off the dependent path
//   E1  r = beta v - D1, hi/lo bf16 pair back into TMEM over D1                    (256 threads)
//   P2  D2[v][k]       = r^T . kx           12 x M128 N128 K16 (hi.hi, lo.hi, hi.lo)
//   P3  D1[v][64..127] += r^T . ax^T        12 x M128 N64..16 K16
//   E2  S = S dec + D2; bf16(S) is the next A operand; o leaves transposed, 16 bytes a thread
// Tensor memory, 256 columns: D1 128, D2 128; bf16(S) lies over D2 (read before it is written, read again by P1 before
// P2 writes), r over the first half of D1.  A dependent step is two commit -> wait hand-overs (~430 cycles each, whatever
// the product's size) and two passes over TMEM, for 64 tokens instead of 16.
//
// Warp roles: 0-7 element-wise work (warp w: TMEM lanes 32 (w%4).., tokens or state columns of half w/4); one CTA per SM
// (two stages of operands): 8-11 outputs, 12 MMA issue, copies and TMEM owner; two CTAs per SM (one stage): eight
// warps, of which the first issues besides its own part.  Every wait is bounded.
//
// Measured, K2 alone: B1 T8192 H96 606 us in the 16-token tensor-memory form, 280 here (2.2 us per 64 tokens and chain,
// 1.34 GB: 0.73 of the measured copy rate); B8 T2048 H32 205 -> 177.
#include <cuda.h>

#include "kda_common.cuh"
#include "kda_kernels.h"
#include "kda_tc.cuh"
#include "kda_wide.cuh"

namespace kda {

namespace {

constexpr int W2_EW = 8;
constexpr int ST_K2W_TIMEOUT = 9;
constexpr int WKX_BYTES = 2 * 16384;

template <int ST>
struct W2Smem {
  // Two CTAs of eight warps leave a thread 128 registers, two of nine only 96 (64 hold the state): there warp 0 issues
  // the products and copies besides its own part.
  static constexpr bool MERGED = ST == 1;
  // With one CTA per SM four more warps take the outputs (the element-wise warps' loop is what bounds a step).
  static constexpr int OUT_WARPS = MERGED ? 0 : 4;
  static constexpr int THREADS = (W2_EW + (MERGED ? 0 : OUT_WARPS + 1)) * 32;
  static constexpr int ISSUE_WARP = MERGED ? 0 : W2_EW + OUT_WARPS;
  // one stage: p1 | kx hi, kx lo, ax hi, ax lo | v
  static constexpr int P1 = 0, KX = WREC_P1_BYTES, AX = KX + WKX_BYTES, V = AX + 2 * WREC_AX_BYTES;
  static constexpr int STAGE = V + WT * D * 2;
  static constexpr int SMALL = ST * STAGE;                          // [ST + 1] dec, beta: dec is read until the step's end
  static constexpr int OST = SMALL + (ST + 1) * WREC_SMALL_BYTES;   // output staging: [warp][16 tok][32 v] bf16
  static constexpr int BARS = OST + W2_EW * 1024;
  static constexpr int NBARS = 2 * ST + 8;
  static constexpr int SLOT = BARS + NBARS * 8;
  static constexpr int TOTAL = SLOT + 16;
  static_assert(STAGE % 1024 == 0 && TOTAL <= 232448, "swizzled tiles; shared memory of an SM");
};

constexpr uint32_t C_R = 0, C_O = 64, C_D2 = 128, W2_COLS = 256;

__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

template <int ST>
__global__ void __launch_bounds__(W2Smem<ST>::THREADS, ST == 1 ? 2 : 1) kda_k2w_kernel(const __grid_constant__ K2wParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using SM = W2Smem<ST>;
  constexpr bool MERGED = SM::MERGED;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + SM::BARS;
  auto full_p = [&](int s) { return bar0 + s * 8; };
  auto full_k = [&](int s) { return bar0 + (ST + s) * 8; };
  const uint32_t bar_p1 = bar0 + (2 * ST + 0) * 8, bar_p1b = bar0 + (2 * ST + 1) * 8, bar_r = bar0 + (2 * ST + 2) * 8,
                 bar_p2 = bar0 + (2 * ST + 3) * 8, bar_p3 = bar0 + (2 * ST + 4) * 8, bar_o = bar0 + (2 * ST + 5) * 8;
  auto bar_s = [&](int q) { return bar0 + (2 * ST + 6 + q) * 8; };
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + SM::SLOT);
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + SM::SLOT + 4);

  if (tid == 0) {
    for (int s = 0; s < ST; ++s) { mbar_init(full_p(s), 1); mbar_init(full_k(s), 1); }
    mbar_init(bar_p1, 1);
    mbar_init(bar_p1b, 1);
    mbar_init(bar_r, W2_EW);
    mbar_init(bar_p2, 1);
    mbar_init(bar_p3, 1);
    mbar_init(bar_o, MERGED ? W2_EW : SM::OUT_WARPS);
    for (int q = 0; q < 2; ++q) mbar_init(bar_s(q), W2_EW);
    *sAbort = 0;
    fence_mbar_init();
  }
  if (warp == SM::ISSUE_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(W2_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // ---- which chain, which chunks of it, from which state, to where ----
  int bh = blockIdx.x;
  bool want_o = true, use_v = true, src_kf = p.k_first != 0, dst_kf = src_kf;
  const float* src = nullptr;   // null: zeros
  float* dst = nullptr;
  bool identity = false;
  int part = 0;   // which job of the chain
  if (p.job == W2_STATE_PAIR) { part = bh & 1; bh >>= 1; }
  else if (p.job == W2_SPLIT_FIRST || p.job == W2_SPLIT_LAST) { part = bh / p.n_chains; bh -= part * p.n_chains; }
  int b = bh / p.H, NT = p.NT, Tlen = p.T, tok0 = 0;
  size_t rec_first = 0;
  const int h = bh % p.H;
  if (p.seq_table != nullptr) {   // packed sequences: bh = sequence * H + head
    const int4 e = __ldg(p.seq_table + b);
    tok0 = e.x;
    Tlen = e.w;
    NT = (Tlen + WT - 1) / WT;
    int before = 0;               // wide chunks of the sequences before this one
    for (int j = lane; j < b; j += 32) before += (__ldg(&p.seq_table[j].w) + WT - 1) / WT;
    before = __reduce_add_sync(0xffffffffu, before);
    rec_first = static_cast<size_t>(before) * p.H + static_cast<size_t>(h) * NT;
    b = 0;
  } else {
    rec_first = static_cast<size_t>(bh) * NT;
  }
  const size_t state = static_cast<size_t>(D) * D;
  src = p.h0 != nullptr ? p.h0 + bh * state : nullptr;
  dst = p.ht != nullptr ? p.ht + bh * state : nullptr;
  int n0 = 0, n1 = NT;
  if (p.job == W2_SPLIT_FIRST && part == 0) {           // the first segment, to its end
    n1 = p.seg;
    dst = p.entry + bh * state;
    dst_kf = false;
  } else if (p.job == W2_SPLIT_LAST) {                  // segment part + 1 from its entry state
    n0 = (part + 1) * p.seg;
    n1 = min(NT, n0 + p.seg);
    src = p.entry + (static_cast<size_t>(part) * p.n_chains + bh) * state;
    src_kf = false;
    if (n1 < NT) dst = nullptr;
  } else if (p.job == W2_SPLIT_FIRST || p.job == W2_STATE_PAIR) {
    // a transform: M (identity entry state, no v) or Q (zero entry state) of one segment, or of the whole chain
    const int which = p.job == W2_STATE_PAIR ? part : (part - 1) & 1;
    if (p.job == W2_SPLIT_FIRST) {
      const int sgm = 1 + (part - 1) / 2;               // 1 .. n_seg - 2
      n0 = sgm * p.seg;
      n1 = n0 + p.seg;
      dst = p.mq + ((static_cast<size_t>(bh) * (p.n_seg - 2) + sgm - 1) * 2 + which) * state;
    } else {
      dst = p.push_on ? p.push_dst[bh / p.push_hp] + p.push_dst_offset + (static_cast<size_t>(bh % p.push_hp) * 2 + which) * state
                      : p.ht + (static_cast<size_t>(bh) * 2 + which) * state;
    }
    want_o = false;
    use_v = which == 1;
    identity = which == 0;
    src = nullptr;
    dst_kf = false;
  } else if (p.job == W2_STATE) {
    want_o = false;
    use_v = p.zero_u == 0;
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *slot;

  auto give_up = [&]() {
    if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2W_TIMEOUT); }
  };
  const int steps = n1 - n0;

  // ---- MMA issue and copies: whole-warp calls of one warp.  Chunk n's operands lie in stage n % ST.  ----
  const uint8_t* rec0 = p.rec + (rec_first + n0) * WREC_BYTES;
  int p_issued = 0, k_issued = 0;
  auto load_p = [&](int n) {   // kb, qg, dec, beta and v
    if (elect_one()) {
      const int s = n % ST;
      const uint32_t dstp = sbase + s * SM::STAGE, small = sbase + SM::SMALL + (n % (ST + 1)) * WREC_SMALL_BYTES;
      const uint8_t* rec = rec0 + static_cast<size_t>(n) * WREC_BYTES;
      mbar_arrive_expect_tx(full_p(s), (want_o ? WREC_P1_BYTES : WREC_P1_BYTES / 2) + WREC_SMALL_BYTES + (use_v ? WT * D * 2 : 0));
      if (want_o) {
        bulk_g2s(dstp + SM::P1, rec + WREC_P1, WREC_P1_BYTES, full_p(s));
      } else {
        bulk_g2s(dstp + SM::P1, rec + WREC_P1, 8192, full_p(s));
        bulk_g2s(dstp + SM::P1 + 16384, rec + WREC_P1 + 16384, 8192, full_p(s));
      }
      bulk_g2s(small, rec + WREC_DEC, WREC_SMALL_BYTES, full_p(s));
      if (use_v) tma_load_4d(dstp + SM::V, &p.tm_v, 0, h, tok0 + (n0 + n) * WT, b, full_p(s));
    }
    __syncwarp();
    p_issued = n + 1;
  };
  auto load_k = [&](int n) {   // kx and ax
    if (elect_one()) {
      const int s = n % ST;
      const uint32_t bytes = WKX_BYTES + (want_o ? 2 * WREC_AX_BYTES : 0);
      mbar_arrive_expect_tx(full_k(s), bytes);
      bulk_g2s(sbase + s * SM::STAGE + SM::KX, rec0 + static_cast<size_t>(n) * WREC_BYTES + WREC_KXH, bytes, full_k(s));
    }
    __syncwarp();
    k_issued = n + 1;
  };
  constexpr uint32_t ID_P1 = instr_desc(128, 64, 0), ID_P2 = instr_desc(128, 128, 0);
  // P1 of chunk n, the half that r needs: the snapshot comes in two groups of columns per half
  auto issue_p1 = [&](int n) -> bool {
    const int s = n % ST;
    if (!mbar_wait_parked(full_p(s), (n / ST) & 1, sAbort)) return false;
    const uint64_t dkb = smem_desc(sbase + s * SM::STAGE + SM::P1, 16, 1024, 2);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!mbar_wait_parked(bar_s(q), n & 1, sAbort)) return false;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int cc = 2 * q; cc < 2 * q + 2; ++cc)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf)
            umma_ts(tbase + C_R, tbase + C_D2 + hf * 64 + cc * 8, dkb + static_cast<uint64_t>((hf * 16384 + cc * 32) >> 4), ID_P1,
                    !(cc == 0 && hf == 0));
        if (q == 1) umma_commit(bar_p1);
      }
      __syncwarp();
    }
    return true;
  };
  // P3 of chunk n is done about when P1 of the next has been issued: its kx and ax make room
  auto refill_k = [&](int n) -> bool {
    if (n + ST >= steps) return true;
    if (!mbar_wait_parked(bar_p3, n & 1, sAbort)) return false;
    load_k(n + ST);
    return true;
  };
  // the other half of P1, once the outputs before it have left TMEM
  auto issue_p1_out = [&](int n) -> bool {
    if (want_o && n > 0 && !mbar_wait_parked(bar_o, (n - 1) & 1, sAbort)) return false;
    tc_fence_after();
    if (elect_one()) {
      if (want_o) {
        const uint64_t dqg = smem_desc(sbase + (n % ST) * SM::STAGE + SM::P1 + 8192, 16, 1024, 2);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_ts(tbase + C_O, tbase + C_D2 + (ks >> 2) * 64 + (ks & 3) * 8,
                  dqg + static_cast<uint64_t>(((ks >> 2) * 16384 + (ks & 3) * 32) >> 4), ID_P1, ks != 0);
      }
      umma_commit(bar_p1b);
    }
    __syncwarp();
    return true;
  };
  auto issue_p23 = [&](int n) -> bool {
    const int s = n % ST;
    const uint32_t st = sbase + s * SM::STAGE;
    if (!mbar_wait_parked(full_k(s), (n / ST) & 1, sAbort)) return false;
    if (!mbar_wait_parked(bar_r, n & 1, sAbort)) return false;   // r hi/lo are in TMEM
    tc_fence_after();
    if (elect_one()) {
      const uint64_t dkh = smem_desc(st + SM::KX, 2048, 128, 0), dkl = smem_desc(st + SM::KX + 16384, 2048, 128, 0);
#pragma unroll
      for (int c = 0; c < 4; ++c) {   // 16 tokens each
        const uint32_t rh = tbase + C_R + c * 16, rl = rh + 8;
        const uint64_t o = static_cast<uint64_t>((c * 4096) >> 4);
        umma_ts(tbase + C_D2, rh, dkh + o, ID_P2, c != 0);
        umma_ts(tbase + C_D2, rl, dkh + o, ID_P2, 1);
        umma_ts(tbase + C_D2, rh, dkl + o, ID_P2, 1);
      }
      umma_commit(bar_p2);
      if (want_o) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {   // column panel c of ax: token rows from 16 c on
          const uint32_t rh = tbase + C_R + c * 16, rl = rh + 8, id = instr_desc(128, WT - 16 * c, 0);
          const uint64_t dah = smem_desc(st + SM::AX + ax_panel(c), (WT - 16 * c) * 16, 128, 0);
          const uint64_t dal = smem_desc(st + SM::AX + WREC_AX_BYTES + ax_panel(c), (WT - 16 * c) * 16, 128, 0);
          umma_ts(tbase + C_O + 16 * c, rh, dah, id, 1);
          umma_ts(tbase + C_O + 16 * c, rl, dah, id, 1);
          umma_ts(tbase + C_O + 16 * c, rh, dal, id, 1);
        }
      }
      umma_commit(bar_p3);
    }
    __syncwarp();
    // p1 and v of this stage are free when P1 is done (r came from v)
    if (n + ST < steps) {
      if (!mbar_wait_parked(bar_p1b, n & 1, sAbort)) return false;
      load_p(n + ST);
      if (n + ST + 1 < steps && elect_one()) prefetch_l2(rec0 + static_cast<size_t>(n + ST + 1) * WREC_BYTES, WREC_BYTES);
      __syncwarp();
    }
    return true;
  };
  auto first_loads = [&]() {
    grid_dep_wait();   // K1's records; everything above ran under K1's tail
    for (int n = 0; n < ST && n < steps; ++n) { load_p(n); load_k(n); }
  };

  if (!MERGED && warp == SM::ISSUE_WARP) {
    first_loads();
    for (int n = 0; n < steps; ++n) {
      if (!issue_p1(n) || (n > 0 && !refill_k(n - 1)) || !issue_p1_out(n) || !issue_p23(n)) { give_up(); break; }
    }
  } else if (!MERGED && warp >= W2_EW) {
    // ------------------------------ outputs ---------------------------------
    const int quad = warp & 3, g4 = lane >> 2, t4 = lane & 3;
    const uint32_t tl = tbase + (static_cast<uint32_t>(quad * 32) << 16);
    uint8_t* const ost = smem + SM::OST + quad * 2048;
    __nv_bfloat16* const orow = want_o ? p.o + b * p.o_s[0] + tok0 * p.o_s[1] + h * p.o_s[2] + quad * 32 + t4 * 8 : nullptr;
    for (int n = 0; n < steps && want_o; ++n) {
      if (!mbar_wait_parked(bar_p3, n & 1, sAbort)) { give_up(); break; }
      tc_fence_after();
      uint32_t oo[32];   // bf16 pairs of tokens
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t d[32];
        tmem_ld32(tl + C_O + c * 32, d);
        tc_wait_ld();
        pin32(d);
#pragma unroll
        for (int j = 0; j < 16; ++j) oo[c * 16 + j] = pack_bf16(__uint_as_float(d[2 * j]), __uint_as_float(d[2 * j + 1]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_o);
#pragma unroll
      for (int c = 0; c < 2; ++c) {   // 32 tokens of the warp's 32 rows, transposed through 2 KB
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          *reinterpret_cast<unsigned short*>(ost + (2 * j) * 64 + lane * 2) = static_cast<unsigned short>(oo[c * 16 + j] & 0xffffu);
          *reinterpret_cast<unsigned short*>(ost + (2 * j + 1) * 64 + lane * 2) = static_cast<unsigned short>(oo[c * 16 + j] >> 16);
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int tok = (n0 + n) * WT + c * 32 + e * 8 + g4;
          if (tok < Tlen)
            *reinterpret_cast<uint4*>(orow + static_cast<int64_t>(tok) * p.o_s[1]) =
                *reinterpret_cast<const uint4*>(ost + (e * 8 + g4) * 64 + t4 * 16);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------ element-wise warps ----------------------
    const int quad = warp & 3, half = warp >> 2;
    const bool issuer = MERGED && warp == 0;
    if (issuer) first_loads();
    const int v = quad * 32 + lane;                        // state row = TMEM lane
    const uint32_t tl = tbase + (static_cast<uint32_t>(quad * 32) << 16);
    const int g4 = lane >> 2, t4 = lane & 3;
    bool ok = true;
    if (p.h0_n_flags > 0) {   // the entry state comes from other GPUs: wait for their flags (the first copies are under way)
      int got = 1;
      if (lane == 0)
        for (int i = 0; i < p.h0_n_flags; ++i) got &= flag_wait_bounded(p.h0_flags + i, p.h0_epoch) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, got, 0) != 0;
      if (!ok && *sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_PEER_TIMEOUT); }
    }
    float S[64];                                           // S[v][64 half + j]
    if (src != nullptr && src_kf) {
#pragma unroll
      for (int j = 0; j < 64; ++j) S[j] = src[static_cast<size_t>(half * 64 + j) * D + v];
    } else if (src != nullptr) {
      // rows of the state come in 32-byte pieces (the 16-lane access shapes) and are turned through TMEM
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t f[32];
        const float* at = src + static_cast<size_t>(quad * 32 + hh * 16 + g4) * D + half * 64 + t4 * 2;
#pragma unroll
        for (int n8 = 0; n8 < 8; ++n8) {
          const float2 x = *reinterpret_cast<const float2*>(at + n8 * 8), y = *reinterpret_cast<const float2*>(at + 8 * D + n8 * 8);
          f[n8 * 4] = __float_as_uint(x.x); f[n8 * 4 + 1] = __float_as_uint(x.y);
          f[n8 * 4 + 2] = __float_as_uint(y.x); f[n8 * 4 + 3] = __float_as_uint(y.y);
        }
        tmem_st_16x256b_x8(tbase + (static_cast<uint32_t>(quad * 32 + hh * 16) << 16) + C_D2 + half * 64, f);
      }
      tc_wait_st();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t f[32];
        tmem_ld32(tl + C_D2 + half * 64 + c * 32, f);
        tc_wait_ld();
        pin32(f);
#pragma unroll
        for (int j = 0; j < 32; ++j) S[c * 32 + j] = __uint_as_float(f[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 64; ++j) S[j] = identity && half * 64 + j == v ? 1.f : 0.f;
    }
    auto snapshot = [&](int c) {   // bf16 of columns 16 c .. 16 c + 15 of this half
      uint32_t a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = pack_bf16(S[c * 16 + 2 * j], S[c * 16 + 2 * j + 1]);
      tmem_st8(tl + C_D2 + half * 64 + c * 8, a);
    };
    auto hand_over = [&](uint32_t bar) {   // what this warp wrote to (or read from) TMEM is complete
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) snapshot(c);
    tc_wait_st();
    hand_over(bar_s(0));
    hand_over(bar_s(1));
    if (issuer && ok) ok = issue_p1(0) && issue_p1_out(0);

    __nv_bfloat16* const orow = want_o ? p.o + b * p.o_s[0] + tok0 * p.o_s[1] + h * p.o_s[2] : nullptr;
    uint8_t* const ost = smem + SM::OST + warp * 1024;
    for (int n = 0; n < steps && ok; ++n) {
      const int s = n % ST;
      const float* small = reinterpret_cast<const float*>(smem + SM::SMALL + (n % (ST + 1)) * WREC_SMALL_BYTES);
      const uint8_t* sv = smem + s * SM::STAGE + SM::V + half * 32 * 256 + v * 2;
      const int left = Tlen - (n0 + n) * WT - half * 32;   // valid tokens from this half's first on
      ok = mbar_wait_parked(full_p(s), (n / ST) & 1, sAbort);

      // ---- E1: r of this thread's row and 32 tokens ----
      // beta v of token j of the half.  With registers to spare it is worked out before P1 is done.
      auto bv_pair = [&](int j) {
        const float2 be = *reinterpret_cast<const float2*>(small + 128 + half * 32 + j);
        float2 x;
        x.x = be.x * __uint_as_float(static_cast<uint32_t>(*reinterpret_cast<const unsigned short*>(sv + j * 256)) << 16);
        x.y = be.y * __uint_as_float(static_cast<uint32_t>(*reinterpret_cast<const unsigned short*>(sv + (j + 1) * 256)) << 16);
        return x;
      };
      float2 bv[ST == 2 ? 16 : 1];
      if (ST == 2) {
#pragma unroll
        for (int j = 0; j < 16; ++j) bv[ST == 2 ? j : 0] = use_v && ok ? bv_pair(2 * j) : make_float2(0.f, 0.f);
      }
      ok = ok && mbar_wait_parked(bar_p1, n & 1, sAbort);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t d[16], hl[16];
        tmem_ld16(tl + C_R + half * 32 + c * 16, d);
        tc_wait_ld();
        pin16(d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float2 x = ST == 2 ? bv[ST == 2 ? c * 8 + j : 0] : use_v ? bv_pair(c * 16 + 2 * j) : make_float2(0.f, 0.f);
          x = __fadd2_rn(x, make_float2(-__uint_as_float(d[2 * j]), -__uint_as_float(d[2 * j + 1])));
          // rows past the end carry whatever follows the sequence in memory
          if (c * 16 + 2 * j >= left) x.x = 0.f;
          if (c * 16 + 2 * j + 1 >= left) x.y = 0.f;
          split_pack2(x, hl[j], hl[8 + j]);
        }
        tmem_st16(tl + C_R + half * 32 + c * 16, hl);   // hi in the first eight columns, lo in the others
      }
      tc_wait_st();
      hand_over(bar_r);
      if (issuer && !issue_p23(n)) { ok = false; break; }

      // ---- E2: the new state; its snapshot leaves in two groups of columns ----
      if (!mbar_wait_parked(bar_p2, n & 1, sAbort)) { ok = false; break; }
      tc_fence_after();
      const bool more = n + 1 < steps;
      const float* dec = small + half * 64;
      constexpr int AHEAD = ST == 2 ? 1 : 0;   // 16-column pieces fetched ahead of their use
      uint32_t dd2[AHEAD + 1][16];
      if (AHEAD) tmem_ld16(tl + C_D2 + half * 64, dd2[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t (&d)[16] = dd2[AHEAD ? c & 1 : 0];
        if (!AHEAD) tmem_ld16(tl + C_D2 + half * 64 + c * 16, d);
        tc_wait_ld();
        pin16(d);
        if (AHEAD && c < 3) tmem_ld16(tl + C_D2 + half * 64 + (c + 1) * 16, dd2[(c + 1) & AHEAD]);
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 dd = *reinterpret_cast<const float4*>(dec + c * 16 + j);
          const float2 a = __ffma2_rn(make_float2(S[c * 16 + j], S[c * 16 + j + 1]), make_float2(dd.x, dd.y),
                                      make_float2(__uint_as_float(d[j]), __uint_as_float(d[j + 1])));
          const float2 e = __ffma2_rn(make_float2(S[c * 16 + j + 2], S[c * 16 + j + 3]), make_float2(dd.z, dd.w),
                                      make_float2(__uint_as_float(d[j + 2]), __uint_as_float(d[j + 3])));
          S[c * 16 + j] = a.x; S[c * 16 + j + 1] = a.y; S[c * 16 + j + 2] = e.x; S[c * 16 + j + 3] = e.y;
        }
        if (more) {
          snapshot(c);
          if (c & 1) {
            tc_wait_st();
            hand_over(bar_s(c >> 1));
          }
        }
      }

      if (issuer && more && !(issue_p1(n + 1) && refill_k(n))) { ok = false; break; }

      // ---- outputs: o of this thread's row and 32 tokens, transposed through the warp's own 1 KB ----
      if (MERGED && want_o) {
        if (!mbar_wait_parked(bar_p3, n & 1, sAbort)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t d[16];
          tmem_ld16(tl + C_O + half * 32 + c * 16, d);
          tc_wait_ld();
          pin16(d);
          if (c == 1) {
            hand_over(bar_o);
            if (issuer && more && !issue_p1_out(n + 1)) ok = false;
          } else {
            __syncwarp();
          }
#pragma unroll
          for (int j = 0; j < 16; ++j)
            *reinterpret_cast<__nv_bfloat16*>(ost + j * 64 + lane * 2) = __float2bfloat16_rn(__uint_as_float(d[j]));
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int row = e * 8 + g4;
            if (c * 16 + row < left)
              *reinterpret_cast<uint4*>(orow + static_cast<int64_t>((n0 + n) * WT + half * 32 + c * 16 + row) * p.o_s[1] + quad * 32 + t4 * 8) =
                  *reinterpret_cast<const uint4*>(ost + row * 64 + t4 * 16);
          }
        }
      } else if (issuer && more && !issue_p1_out(n + 1)) {
        ok = false;
      }
    }
    if (ok && dst != nullptr) {
      if (dst_kf) {
#pragma unroll
        for (int j = 0; j < 64; ++j) dst[static_cast<size_t>(half * 64 + j) * D + v] = S[j];
      } else {
        // every thread of the warp has read D2; no product follows
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t f[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = __float_as_uint(S[c * 32 + j]);
          tmem_st32(tl + C_D2 + half * 64 + c * 32, f);
        }
        tc_wait_st();
#pragma unroll 1
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t f[32];
          tmem_ld_16x256b_x8(tbase + (static_cast<uint32_t>(quad * 32 + hh * 16) << 16) + C_D2 + half * 64, f);
          tc_wait_ld();
          pin32(f);
          float* at = dst + static_cast<size_t>(quad * 32 + hh * 16 + g4) * D + half * 64 + t4 * 2;
#pragma unroll
          for (int n8 = 0; n8 < 8; ++n8) {
            *reinterpret_cast<float2*>(at + n8 * 8) = make_float2(__uint_as_float(f[n8 * 4]), __uint_as_float(f[n8 * 4 + 1]));
            *reinterpret_cast<float2*>(at + 8 * D + n8 * 8) = make_float2(__uint_as_float(f[n8 * 4 + 2]), __uint_as_float(f[n8 * 4 + 3]));
          }
        }
      }
    }
    if (!ok) give_up();
  }
  if (warp == SM::ISSUE_WARP && *sAbort != 0) {   // copies still in flight get a bounded chance to land before the shared memory goes
    for (int n = max(0, p_issued - ST); n < p_issued; ++n) mbar_wait_parked(full_p(n % ST), (n / ST) & 1, nullptr);
    for (int n = max(0, k_issued - ST); n < k_issued; ++n) mbar_wait_parked(full_k(n % ST), (n / ST) & 1, nullptr);
  }
  __syncwarp();

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (p.push_on && tid == 0 && *sAbort == 0) {
    // the tiles went into another rank's receive buffer: the CTA barrier has put every warp's stores before this
    // count; the CTA that counts last for a destination raises its flag behind one system-scope fence
    const int owner = bh / p.push_hp;
    __threadfence();
    const int done = atomicAdd(p.push_counter + owner, 1);
    __threadfence();
    if (done == 2 * p.push_hp - 1) {
      p.push_counter[owner] = 0;
      __threadfence_system();
      st_release_sys(p.push_flag[owner], p.push_epoch);
    }
  }
  if (warp == SM::ISSUE_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(W2_COLS) : "memory");
}

template <int ST>
cudaError_t launch_k2w_t(const K2wParams& p, int jobs, cudaStream_t stream) {
  constexpr int smem_bytes = W2Smem<ST>::TOTAL;
  static std::atomic<bool> configured[64];   // set after the attributes, also for other threads
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kda_k2w_kernel<ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kda_k2w_kernel<ST>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return launch_dep(kda_k2w_kernel<ST>, jobs, W2Smem<ST>::THREADS, smem_bytes, stream, p.pdl, p);
}

}  // namespace

cudaError_t launch_k2w(const K2wParams& p, int jobs, bool one_per_sm, cudaStream_t stream) {
  return one_per_sm ? launch_k2w_t<2>(p, jobs, stream) : launch_k2w_t<1>(p, jobs, stream);
}

}  // namespace kda
