// K2 on the 5th-generation tensor cores (tcgen05 + TMEM): the throughput form of the state
// recurrence for problems with many (batch, head) chains.  sm_100a.
//
// Same arithmetic and record contract as kda_k2_sm100.cu (which replaces kda_bt16_kernel_k2 of the
// reference, src/kda_bt16/kernels.py:187-302):
//   v_new = u - w h^T ;  o = scale (qg h^T) + Aqk v_new ;  h = h diag(dec) + v_new^T kg
// One CTA owns ALL 128 state rows of one (batch, head): the fp32 state lives in tensor memory
// (128 lanes = rows v, 128 columns = k) for the whole sequence.  Per chunk:
//   P1  D1[v][32]  = bf16(h)[v][:] . [-w ; qg]^T         8 x tcgen05.mma M128 N32 K16   (A from TMEM)
//   P0  D1[v][0:16] += v^T[v][:] . Xb^T  (= u)            2 x M128 N16 K16   (A from shared memory, v as it lies)
//   E1  v_new = D1[:, 0:16]  ->  hi/lo bf16 pair back into TMEM              (256 threads)
//   P2  h[v][:]   += v_new^T[v][:] . kg                   3 x M128 N128 K16 (hi.hi, lo.hi, hi.lo)
//   P3  D3[v][16]  = v_new^T[v][:] . Aqk^T                3 x M128 N16 K16
//   E2  read h, write bf16(h) (next P1's A operand) and h * dec(next chunk); o = scale D1[:, 16:32] + D3
// The record's tiles are tensor-core operands as they stand (kda_common.cuh): one bulk copy per chunk, no second
// pass over them.
//
// P0 goes last, so that the sum over k is not rounded at the size of u again and again; first (under the state pass of the
// step before) it is no faster.  With u read by the element-wise warps: B8 T2048 H32 185 -> 176 us, T8192 H96 447 -> 446.
//
// A step is a chain of hand-overs: eight MMAs, commit and wait about 190 cycles, P2 300, a TMEM load 140, the state pass
// 600.  One CTA alone on its SM takes 0.84 us per step (the 8-row mma.sync form 0.34 to 0.45), two resident ones 1.34
// together (256 of the 512 TMEM columns, 100 KB of shared memory each): the form pays once there are enough chains.
// Every tcgen05 instruction is issued behind elect.sync (see elect_one) by a warp that walks the loop as a whole.  K2
// alone with the instructions behind lane == 0 and records loaded by tiled copies, and now: T8192 H96 606 -> 447 us,
// B8 T1024 H32 110.5 -> 98.6.
//
// Warp roles: 0-7 element-wise work (warp w: TMEM lanes 32 (w%4).., column / token half w/4),
// 8 = producer (TMA), 9 = MMA issuer and TMEM owner.  Every wait is bounded.
#include "kda_common.cuh"
#include "kda_kernels.h"
#include "kda_tc.cuh"

namespace kda {

namespace {

// Four stages, given back by a commit behind P3: K2 alone T8192 H96 447 -> 432 us (three and by an element-wise warp at the end of
// its state pass before; two: 689), the forward, K1 beside it, 654 -> 633.  Two CTAs of five do not fit an SM.
constexpr int KT_STAGES = 4;
constexpr int KT_EPI_WARPS = 8;
constexpr int KT_THREADS = (KT_EPI_WARPS + 2) * 32;
constexpr int T_STAGE = REC_USED_BYTES;   // a record as it is
static_assert(T_STAGE % 1024 == 0 && REC_V % 1024 == 0, "the swizzled atoms are 1024-byte aligned");
constexpr int T_BARS = KT_STAGES * T_STAGE;
// The state snapshot reaches the MMA thread in KT_PG column groups, so that the first k-steps of the
// next P1 are issued while the element-wise warps still convert the rest of the state.
constexpr int KT_PG = 2;
static_assert(KT_PG == 1 || KT_PG == 2 || KT_PG == 4, "column groups of the snapshot");
// barriers: full[S], empty[S], p1, v, p2, p3, s[KT_PG]
constexpr int T_NBARS = 2 * KT_STAGES + 4 + KT_PG;
constexpr int T_SLOT = T_BARS + T_NBARS * 8;      // TMEM base address, abort flag, issued count
constexpr int T_OST = (T_SLOT + 32 + 15) / 16 * 16;                // output staging, two chunks: [warp][8 tok][32 v] bf16
constexpr int T_TOTAL = T_OST + 2 * TILE_BYTES;
static_assert(T_OST % 16 == 0, "staging tiles are read 16 bytes at a time");
// TMEM columns
constexpr uint32_t C_S = 0, C_D1 = 128, C_D3 = 160, C_AS = 176, C_VH = 240, C_VL = 248, C_TOTAL = 256;

constexpr int ST_K2T_TIMEOUT = 4;

__global__ void __launch_bounds__(KT_THREADS, 2) kda_k2t_kernel(const __grid_constant__ K2Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // warp-uniform for the compiler
  int bh = blockIdx.x + p.chain0;
  if (p.by_length) bh = chain_by_length(p.seq_table, p.n_seqs, p.H, bh);
  int b = bh / p.H;
  const int h = bh % p.H;
  int NT = p.NT, Tlen = p.T, tok0 = 0;
  size_t rec_first = static_cast<size_t>(bh) * NT;
  if (p.seq_table != nullptr) {   // packed sequences: bh = sequence * H + head
    const int4 e = __ldg(p.seq_table + b);
    tok0 = e.x; NT = e.y; Tlen = e.w;
    rec_first = static_cast<size_t>(e.z) + static_cast<size_t>(h) * NT;
    b = 0;
    if (p.long_len > 0 && NT >= p.long_len && (blockIdx.x + p.chain0) / p.H < p.long_max) return;   // in the 16-row form
  }

  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + T_BARS;
  auto full = [&](int s) { return bar0 + s * 8; };
  auto empty = [&](int s) { return bar0 + (KT_STAGES + s) * 8; };
  const uint32_t bar_p1 = bar0 + (2 * KT_STAGES + 0) * 8, bar_v = bar0 + (2 * KT_STAGES + 1) * 8;
  const uint32_t bar_p2 = bar0 + (2 * KT_STAGES + 2) * 8, bar_p3 = bar0 + (2 * KT_STAGES + 3) * 8;
  auto bar_s = [&](int q) { return bar0 + (2 * KT_STAGES + 4 + q) * 8; };
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + T_SLOT);
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + T_SLOT + 4);
  volatile int* sIssued = sAbort + 1;

  if (tid == 0) {
    for (int s = 0; s < KT_STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    mbar_init(bar_p1, 1);
    mbar_init(bar_v, KT_EPI_WARPS);    // one arrival per element-wise warp (lane 0, after __syncwarp)
    mbar_init(bar_p2, 1);
    mbar_init(bar_p3, 1);
    for (int q = 0; q < KT_PG; ++q) mbar_init(bar_s(q), KT_EPI_WARPS);
    *sAbort = 0;
    *sIssued = 0;
    fence_mbar_init();
  }
  if (warp == KT_EPI_WARPS + 1) tmem_alloc(smem_u32(slot), C_TOTAL);   // the MMA warp owns the tensor memory of the CTA
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = __shfl_sync(0xffffffffu, *slot, 0);

  auto give_up = [&]() {
    if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K2T_TIMEOUT); }
  };

  if (warp == KT_EPI_WARPS) {
    // ------------------------------ producer -------------------------------
    if (elect_one()) {
      // K1's records; everything above ran under K1's tail.  Behind a 16-row launch for the long sequences K1 has ended.
      if (p.progress == nullptr && p.long_len == 0) grid_dep_wait();
      int gate = 0;                                 // beside K1: the first chunk of the next window
      for (int n = 0; n < NT; ++n) {
        const int s = n % KT_STAGES;
        if (p.progress != nullptr && n == gate) {
          if (!window_wait_bounded(p.progress + n / p.win_chunks, min(p.win_chunks, NT - n) * p.B * p.H, sAbort)) {
            if (*sAbort == 0) { *sAbort = 1; atomicExch(p.status, ST_K1_WINDOW_TIMEOUT); }
            break;
          }
          gate += p.win_chunks;
        }
        if (n >= KT_STAGES && !mbar_wait_bounded(empty(s), ((n / KT_STAGES) - 1) & 1, sAbort)) { give_up(); break; }
        mbar_arrive_expect_tx(full(s), REC_USED_BYTES);
        bulk_g2s(sbase + s * T_STAGE, p.rec + (rec_first + n) * REC_BYTES, REC_USED_BYTES, full(s));
        *sIssued = n + 1;
      }
    }
    __syncwarp();
  } else if (warp == KT_EPI_WARPS + 1) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp walks the loop, so that the descriptors stay in uniform registers; one lane issues.
    constexpr uint32_t ID_P0 = instr_desc(128, 16) | INSTR_A_MN_MAJOR, ID_P1 = instr_desc(128, 32), ID_P2 = instr_desc(128, 128), ID_P3 = instr_desc(128, 16);
    auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, sAbort)) != 0; };
    int s = 0;
    uint32_t ph = 0;
    for (int n = 0; n < NT; ++n) {
      const uint32_t st = sbase + s * T_STAGE;
      if (!wait(full(s), ph)) { give_up(); break; }
      const uint64_t dwq = smem_desc(st + REC_W, 16, 1024, 2);   // k-step ks: start address + (ks / 4) * 4096 + (ks % 4) * 32 bytes
      bool ready = true;
#pragma unroll
      for (int q = 0; q < KT_PG; ++q) {
        // column group q of both halves of bf16(h) is in TMEM (with the last group: the decayed h too)
        if (ready && !wait(bar_s(q), n & 1)) ready = false;
        if (ready) {
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int cc = q * (4 / KT_PG); cc < (q + 1) * (4 / KT_PG); ++cc)
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                const int ks = hf * 4 + cc;
                umma_ts(tbase + C_D1, tbase + C_AS + ks * 8, dwq + static_cast<uint64_t>((hf * REC_HALF + cc * 32) >> 4), ID_P1,
                        !(cc == 0 && hf == 0));
              }
            if (q == KT_PG - 1) {
              const uint64_t dv = smem_desc(st + REC_V, REC_V_HALF, 1024, 2);
              umma_ss(tbase + C_D1, dv, smem_desc(st + REC_XBL, 256, 128, 0), ID_P0, 1);
              umma_ss(tbase + C_D1, dv, smem_desc(st + REC_XBH, 256, 128, 0), ID_P0, 1);
              umma_commit(bar_p1);
            }
          }
          __syncwarp();
        }
      }
      if (!ready || !wait(bar_v, n & 1)) { give_up(); break; }     // v_new hi/lo are in TMEM
      tc_fence_after();
      if (elect_one()) {
        const uint64_t dkh = smem_desc(st + REC_KGH, 2048, 128, 0), dkl = smem_desc(st + REC_KGL, 2048, 128, 0);
        umma_ts(tbase + C_S, tbase + C_VH, dkh, ID_P2, 1);
        umma_ts(tbase + C_S, tbase + C_VL, dkh, ID_P2, 1);
        umma_ts(tbase + C_S, tbase + C_VH, dkl, ID_P2, 1);
        umma_commit(bar_p2);   // the state pass of the element-wise warps starts while P3 runs
        const uint64_t dah = smem_desc(st + REC_AQK, 512, 128, 0), dal = smem_desc(st + REC_AQL, 512, 128, 0);
        umma_ts(tbase + C_D3, tbase + C_VH, dah, ID_P3, 0);
        umma_ts(tbase + C_D3, tbase + C_VL, dah, ID_P3, 1);
        umma_ts(tbase + C_D3, tbase + C_VH, dal, ID_P3, 1);
        umma_commit(bar_p3);
        umma_commit(empty(s));   // the products are the last to read the stage: its decay was read in the step before
      }
      __syncwarp();
      if (++s == KT_STAGES) { s = 0; ph ^= 1; }
    }
  } else {
    // ------------------------------ element-wise warps ----------------------
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t tl = tbase + (static_cast<uint32_t>(quad * 32) << 16);
    bool ok = true;

    // initial state: TMEM <- h0 * dec(chunk 0); bf16(h0) as the first A operand
    ok = mbar_wait_bounded(full(0), 0, sAbort);
    if (ok) {
      // this warp's 32 rows x 64 columns in two 16-row halves, through the 16-lane access shapes
      const float* dec0 = reinterpret_cast<const float*>(smem + REC_DEC) + half * 64;
      const int g4 = lane >> 2, t4 = lane & 3;
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        const int r0 = quad * 32 + hh * 16 + g4;
        // element (v, k) sits at v*128 + k (V-first) or k*128 + v (K-first); this thread holds rows
        // v = r0, r0 + 8 and columns k = 64 half + 8 n8 + 2 t4, +1
        const float* src = p.h0 == nullptr ? nullptr
                           : p.k_first ? p.h0 + (static_cast<size_t>(bh) * D + half * 64 + t4 * 2) * D + r0
                                       : p.h0 + (static_cast<size_t>(bh) * D + r0) * D + half * 64 + t4 * 2;
        uint32_t sr[32], ar[16];
#pragma unroll
        for (int n8 = 0; n8 < 8; ++n8) {
          float2 x = make_float2(0.f, 0.f), y = x;
          if (src != nullptr) {
            if (p.k_first) {
              const float* c0 = src + n8 * 8 * D;
              x = make_float2(c0[0], c0[D]);
              y = make_float2(c0[8], c0[D + 8]);
            } else {
              x = *reinterpret_cast<const float2*>(src + n8 * 8);
              y = *reinterpret_cast<const float2*>(src + 8 * D + n8 * 8);
            }
          }
          const float2 dd = *reinterpret_cast<const float2*>(dec0 + n8 * 8 + t4 * 2);
          ar[n8 * 2] = pack_bf16(x.x, x.y);
          ar[n8 * 2 + 1] = pack_bf16(y.x, y.y);
          sr[n8 * 4 + 0] = __float_as_uint(x.x * dd.x); sr[n8 * 4 + 1] = __float_as_uint(x.y * dd.y);
          sr[n8 * 4 + 2] = __float_as_uint(y.x * dd.x); sr[n8 * 4 + 3] = __float_as_uint(y.y * dd.y);
        }
        const uint32_t th = tbase + (static_cast<uint32_t>(quad * 32 + hh * 16) << 16);
        tmem_st_16x256b_x8(th + C_S + half * 64, sr);
        tmem_st_16x128b_x8(th + C_AS + half * 32, ar);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        for (int q = 0; q < KT_PG; ++q) mbar_arrive(bar_s(q));
    } else {
      give_up();
    }

    float oq[8], o3[8];
    uint32_t aq[8];
    // this thread's 16 bytes of a chunk's outputs: token 8 half + lane / 4, rows 32 quad + 8 (lane % 4)
    __nv_bfloat16* o_at = p.o + b * p.o_s[0] + (tok0 + half * 8 + (lane >> 2)) * p.o_s[1] + h * p.o_s[2] + quad * 32 + (lane & 3) * 8;
    const int64_t o_step = BT * p.o_s[1];
    int left = Tlen - half * 8 - (lane >> 2);

    // o[tok][v] = scale * (qg h^T) + Aqk v_new of chunk nd, from the registers filled by its E2: a warp's 8 tokens
    // x 32 rows are transposed through its own 512 bytes, so that every thread stores 16 contiguous bytes of a
    // token row and no warp waits for another.  Against whole 256-byte rows, which take a barrier over the eight
    // warps, K2 alone: B8 T1024 H32 119.8 -> 115.7 us, H37 121.8 -> 118.8, B1 T4096 H96 311.8 -> 308.7.
    auto store_o = [&](int nd) {
      uint8_t* buf = smem + T_OST + (nd & 1) * TILE_BYTES + warp * 512;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<__nv_bfloat16*>(buf + j * 64 + lane * 2) = __float2bfloat16(fmaf(p.scale, oq[j], o3[j]));
      __syncwarp();
      if (left > 0) *reinterpret_cast<uint4*>(o_at) = *reinterpret_cast<const uint4*>(buf + lane * 16);
      o_at += o_step;
      left -= BT;
    };

    for (int n = 0; n < NT && ok; ++n) {
      const bool more = n + 1 < NT;

      // ---- E1: v_new for this thread's row and eight tokens ----
      if (!mbar_wait_bounded(bar_p1, n & 1, sAbort)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t d1[8];
        tmem_ld8(tl + C_D1 + half * 8, d1);
        tmem_ld8(tl + C_D1 + 16 + half * 8, aq);   // qg h^T of this chunk: it must leave TMEM before the next P1
        tc_wait_ld();
        pin8(d1);
        pin8(aq);
        uint32_t vh[4], vl[4];
#pragma unroll
        for (int c = 0; c < 4; ++c)
          split_pack(__uint_as_float(d1[2 * c]), __uint_as_float(d1[2 * c + 1]), vh[c], vl[c]);
        tmem_st4(tl + C_VH + half * 4, vh);
        tmem_st4(tl + C_VL + half * 4, vl);
        tc_wait_st();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_v);

      // while P2 runs: the next chunk's record (its decay)
#pragma unroll
      for (int j = 0; j < 8; ++j) oq[j] = __uint_as_float(aq[j]);
      if (more && !mbar_wait_bounded(full((n + 1) % KT_STAGES), ((n + 1) / KT_STAGES) & 1, sAbort)) { ok = false; break; }

      // ---- E2: after P2 / P3 ----
      if (!mbar_wait_bounded(bar_p2, n & 1, sAbort)) { ok = false; break; }
      tc_fence_after();
      // dec of the next chunk (its stage was waited for above)
      const float* decn = reinterpret_cast<const float*>(smem + ((n + 1) % KT_STAGES) * T_STAGE + REC_DEC) + half * 64;
      // the TMEM loads of the state are issued one 16-column step ahead of their use
      uint32_t sr[2][16];
      tmem_ld16(tl + C_S + half * 64, sr[0]);
      tc_wait_ld();
      pin16(sr[0]);
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        uint32_t (&cur)[16] = sr[cc & 1];
        if (cc < 3) tmem_ld16(tl + C_S + half * 64 + (cc + 1) * 16, sr[(cc + 1) & 1]);
        if (more) {
          uint32_t ar[8];
#pragma unroll
          for (int j4 = 0; j4 < 4; ++j4) {
            const float4 dd = *reinterpret_cast<const float4*>(decn + cc * 16 + j4 * 4);
            const float x0 = __uint_as_float(cur[j4 * 4]), x1 = __uint_as_float(cur[j4 * 4 + 1]);
            const float x2 = __uint_as_float(cur[j4 * 4 + 2]), x3 = __uint_as_float(cur[j4 * 4 + 3]);
            ar[j4 * 2] = pack_bf16(x0, x1);
            ar[j4 * 2 + 1] = pack_bf16(x2, x3);
            const float2 lo = __fmul2_rn(make_float2(x0, x1), make_float2(dd.x, dd.y));
            const float2 hi = __fmul2_rn(make_float2(x2, x3), make_float2(dd.z, dd.w));
            cur[j4 * 4 + 0] = __float_as_uint(lo.x); cur[j4 * 4 + 1] = __float_as_uint(lo.y);
            cur[j4 * 4 + 2] = __float_as_uint(hi.x); cur[j4 * 4 + 3] = __float_as_uint(hi.y);
          }
          tmem_st16(tl + C_S + half * 64 + cc * 16, cur);
          tmem_st8(tl + C_AS + half * 32 + cc * 8, ar);
        }
        if (more && (cc + 1) % (4 / KT_PG) == 0) {   // a column group of the snapshot is complete
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_s((cc + 1) / (4 / KT_PG) - 1));
        }
        if (cc < 3) {
          tc_wait_ld();
          pin16(sr[(cc + 1) & 1]);
        }
      }
      // Aqk v_new of this chunk (P3 was committed after P2; it must leave TMEM before the next P3)
      if (!mbar_wait_bounded(bar_p3, n & 1, sAbort)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t c3[8];
        tmem_ld8(tl + C_D3 + half * 8, c3);
        tc_wait_ld();
        pin8(c3);
#pragma unroll
        for (int j = 0; j < 8; ++j) o3[j] = __uint_as_float(c3[j]);
      }
      store_o(n);   // while the next P1 runs
    }
    if (ok && p.ht != nullptr) {
      // final state: TMEM -> global through the 16-lane shape (32-byte pieces of the state's rows);
      // every element-wise thread has seen the last P2 complete
      const int g4 = lane >> 2, t4 = lane & 3;
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t fr[32];
        tmem_ld_16x256b_x8(tbase + (static_cast<uint32_t>(quad * 32 + hh * 16) << 16) + C_S + half * 64, fr);
        tc_wait_ld();
        pin16(reinterpret_cast<uint32_t (&)[16]>(fr[0]));
        pin16(reinterpret_cast<uint32_t (&)[16]>(fr[16]));
        const int vr = quad * 32 + hh * 16 + g4;
        float* dst = p.k_first ? p.ht + (static_cast<size_t>(bh) * D + half * 64 + t4 * 2) * D + vr
                               : p.ht + (static_cast<size_t>(bh) * D + vr) * D + half * 64 + t4 * 2;
#pragma unroll
        for (int n8 = 0; n8 < 8; ++n8) {
          if (p.k_first) {
            float* c0 = dst + n8 * 8 * D;
            c0[0] = __uint_as_float(fr[n8 * 4]); c0[D] = __uint_as_float(fr[n8 * 4 + 1]);
            c0[8] = __uint_as_float(fr[n8 * 4 + 2]); c0[D + 8] = __uint_as_float(fr[n8 * 4 + 3]);
          } else {
            *reinterpret_cast<float2*>(dst + n8 * 8) = make_float2(__uint_as_float(fr[n8 * 4]), __uint_as_float(fr[n8 * 4 + 1]));
            *reinterpret_cast<float2*>(dst + 8 * D + n8 * 8) =
                make_float2(__uint_as_float(fr[n8 * 4 + 2]), __uint_as_float(fr[n8 * 4 + 3]));
          }
        }
      }
    }
    if (!ok) give_up();
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*sAbort != 0 && tid == 0) {
    // give copies that are still in flight a bounded chance to land before the shared memory goes
    const int issued = *sIssued;
    for (int n = max(0, issued - KT_STAGES); n < issued; ++n)
      mbar_wait_bounded(full(n % KT_STAGES), (n / KT_STAGES) & 1, nullptr);
  } else if (*sAbort == 0 && tid < KT_STAGES && tid < NT) {
    // the last stages' way back: an arrival that nobody waits for could still be under way when the shared memory goes
    // (left out behind a comparison in the issuing loop instead: K2 alone T8192 H96 430.5 -> 432.4 us)
    mbar_wait_bounded(empty(tid), ((NT - 1 - tid) / KT_STAGES) & 1, nullptr);
  }
  __syncthreads();
  if (warp == KT_EPI_WARPS + 1)
    tmem_dealloc(tbase, C_TOTAL);
  if (p.progress != nullptr || (p.long_len > 0 && blockIdx.x == gridDim.x - 1)) grid_dep_wait();   // this grid ends after K1, or the 16-row launch
}

}  // namespace

cudaError_t launch_k2t(const K2Params& p, cudaStream_t stream) {
  static std::atomic<bool> configured[64];   // set after the attributes, also for other threads
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kda_k2t_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         T_TOTAL > ONE_CTA_SMEM ? T_TOTAL : ONE_CTA_SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kda_k2t_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int nblocks = p.n_chains > 0 ? p.n_chains : (p.seq_table != nullptr ? p.n_seqs : p.B) * p.H;
  return launch_dep(kda_k2t_kernel, nblocks, KT_THREADS, k2_smem(p, T_TOTAL), stream, p.pdl, p);
}

}  // namespace kda
