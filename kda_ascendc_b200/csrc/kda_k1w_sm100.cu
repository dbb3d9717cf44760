// K1 for wide records: the state-independent work of 64 tokens of one head per item, on the tensor cores.  sm_100a.
//
// Same arithmetic as kda_k1_sm100.cu (which replaces kda_bt16_kernel_k1 of the reference,
// src/kda_bt16/kernels.py:53-184) over chunks of 64 tokens, with the inverse applied to the right (kda_wide.cuh):
//   1. l2-norm of q and k (rounded to bf16), gate, cumulative log2 gate G over the 64 tokens
//   2. Grams Akk, Aqk of all token pairs: D = L R^T, rows of L = khat, qhat times 2^(G - c), rows of R = khat
//      2^(c - G), hi/lo bf16 splits, three tcgen05.mma products with fp32 accumulation (as before, ~2^-16 relative)
//   3. X = (I + Akk)^-1: four 16 x 16 inverses by fp32 column sweeps, joined to 32 x 32 and 64 x 64 by X10 = -X11 A10 X00
//      (mma.sync, hi/lo splits of both sides; the accumulators of one product are the A operand of the next)
//   4. kx = X^T kg and ax = Aqk X, three split products each; kb, qg (bf16), dec and beta
//
// Exponent range: one centre c for all 64 tokens would overflow, so the rows of L are centred per block of tokens
// (NB blocks, centre in the middle of the block) and R exists once per block i: tokens of the blocks 0..i with
// 2^(c_i - G).  For pairs of different blocks that exponent is <= 0; inside a block both factors stay inside
// 2^+-(64 / NB / 2 * |gate|).  NB = 2 (centred over +-16 tokens) is finite while 16 |lower_bound| log2 e <= 116,
// e.g. the production -5; NB = 4 (+-8 tokens) for any lower bound and for sums made by the caller, the range
// of the reference (src/kda_bt16/kernels.py:129-139).  The R tile of the last block, scaled per column by
// 2^(G_last - c), is kg: as A operand of kx^T = R^T X the column becomes the accumulator's lane, so the scale is
// applied to the result.
//
// One persistent CTA per SM, roles: warps 0-15 gate / operands (lane = 8 columns x 2 rows), warps 16-19 (TMEM lane
// quarters) masks, solve and outputs, warp 20 MMA issue, warp 21 copies.  The operands and Grams of item n+1 run while
// item n is solved, and its outputs leave under the solve of item n+1.
//
// What bounds it: about 17,000 warp instructions and 700 KB of shared-memory traffic an item (the Grams read each
// operand tile from there), sixteen operand warps against one solving warp per scheduler.  B1 T8192 H32 (4,096 items):
// 182 us for 515 MB, against 152 us of the 16-token K1 for 643 MB; on the way 258 (one item in flight), 220 (16 operand
// warps, mma.sync solve), 182 (Grams ahead, registers moved to the solving warps).  It pays through K2.
#include <cuda.h>

#include "kda_common.cuh"
#include "kda_kernels.h"
#include "kda_tc.cuh"
#include "kda_wide.cuh"

namespace kda {

namespace {

constexpr int W1_EW = 16, W1_SW = 4;
constexpr int W1_THREADS = (W1_EW + W1_SW + 4) * 32;   // MMA issue and copies: a warp each, in a warpgroup of their own
// Registers: 24 warps are launched with 80 each; the last warpgroup hands 56 of its own to the solving one, so that the
// sum stays that of the launch (512 x 80 + 128 x 136 + 128 x 24 = 768 x 80).
constexpr int W1_SOLVE_REGS = 112, W1_ISSUE_REGS = 48;
static_assert(W1_EW * 32 * 80 + W1_SW * 32 * W1_SOLVE_REGS + 4 * 32 * W1_ISSUE_REGS <= W1_THREADS * 80, "register pool of the CTA");
constexpr int W1_ER = WT / W1_EW;   // rows of an operand warp
constexpr float W1_RANGE = 116.f;   // largest |log2| sum over half a block of 32 tokens (2^126 bounds the factors, and |X| grows them)
constexpr int W1_SLOTS = 4;         // per-item small values: an item's are rewritten four items later

template <int NB>
struct W1Smem {
  // with room for it, the R tile that the last product reads exists twice and X and -Akk have places of their own: the
  // operands of an item are then written, and its Grams taken, while the one before it is solved
  static constexpr bool AHEAD = NB == 2;
  static constexpr int BLK = WT / NB;
  static constexpr int R_ROWS = BLK * NB * (NB + 1) / 2;      // rows of all R tiles together
  static constexpr int R_LAST = WT * D * 4;                   // bytes of the last one, hi and lo
  static constexpr int QK = 0;                                // q, k as they arrive, then the p1 tile
  static constexpr int LH = QK + WREC_P1_BYTES;               // [2 halves][k 0..63, q 64..127][128 B]
  static constexpr int LL = LH + 32768;
  static constexpr int R = LL + 32768;                        // per block i: hi, lo, each [2 halves][BLK (i+1) rows][128 B]
  static constexpr int X = AHEAD ? R + R_ROWS * D * 4 + R_LAST : R;   // X^T hi, lo [64 s][64 t]; else over the first R tiles
  static constexpr int R_END = R + R_ROWS * D * 4 + (AHEAD ? R_LAST + 16384 : 0);
  // -Akk: diagonal 16 x 16 blocks fp32, rows of 20; blocks 10 and 32 hi, lo, rows of 24 bf16; rows 32..63 x columns
  // 0..31 hi, lo, rows of 40 bf16 (the paddings make row accesses conflict-free)
  static constexpr int AD = AHEAD ? R_END : LH;
  static constexpr int AO1 = AD + 4 * 16 * 80;
  static constexpr int AO2 = AO1 + 4 * 16 * 48;
  static constexpr int A_BYTES = 4 * 16 * 80 + 4 * 16 * 48 + 2 * 32 * 80;
  // fp32 [16 warps][128]: the sums of a warp's rows, then G before a warp's rows from its block's centre
  static constexpr int TOT = R_END + (AHEAD ? A_BYTES : 0);
  static constexpr int FAC = TOT + W1_EW * D * 4;             // fp32 [2 NB - 1][128]: 2^(c_b / 2); 2^((c_b+1 - c_b) / 2)
  static constexpr int BETA = FAC + (2 * NB - 1) * D * 4;     // fp32 [slot][64]
  static constexpr int SCALE = BETA + W1_SLOTS * WT * 4;      // fp32 [slot][128] 2^(G_last - c_last)
  static constexpr int STARTS = SCALE + W1_SLOTS * D * 4;     // packed: first wide chunk per sequence
  static constexpr int BARS = STARTS + (WIDE_MAX_SEQS + 2) * 4;
  static constexpr int SLOT = BARS + 10 * 8;
  static constexpr int TOTAL = SLOT + 16;
  static_assert(16384 <= R_ROWS * D * 4 - R_LAST, "X lies below the last R tile");
  static_assert(TOTAL <= 232448, "shared memory of an SM");
  __host__ __device__ static constexpr int r_tile(int i) { return R + BLK * i * (i + 1) / 2 * D * 4; }
};

// TMEM columns
// D: the Gram accumulators (NB = 2: 96 columns, of two items; NB = 4: 160 columns); AQ: Aqk hi, lo of two items
constexpr uint32_t W1_D = 0, W1_D_ITEM = 96, W1_AQ = 192, W1_KX = 320, W1_AX = 384, W1_COLS = 512;

struct W1Item { int b, h, hq, t0, nvalid; size_t rec_idx; };

__device__ __forceinline__ W1Item w1_item(const K1Params& p, const int* starts, int id) {
  W1Item w;
  const int bn = static_cast<int>(p.div_h.div(id));
  w.h = id - bn * p.H;
  w.hq = static_cast<int>(p.div_g.div(w.h));
  if (p.seq_table != nullptr) {   // the sequence of wide chunk bn: the last that starts at or before it
    int lo = 0, hi = p.n_seqs;
    while (hi - lo > 1) {
      const int m = (lo + hi) >> 1;
      if (starts[m] <= bn) lo = m; else hi = m;
    }
    const int first = starts[lo], n = bn - first;
    const int4 e = __ldg(p.seq_table + lo);
    w.b = 0;
    w.t0 = e.x + n * WT;
    w.nvalid = min(WT, e.w - n * WT);
    w.rec_idx = static_cast<size_t>(first) * p.H + static_cast<size_t>(w.h) * (starts[lo + 1] - first) + n;
    return w;
  }
  w.b = static_cast<int>(p.div_nt.div(bn));
  const int n = bn - w.b * p.NT;
  w.t0 = n * WT;
  w.nvalid = min(WT, p.T - w.t0);
  w.rec_idx = (static_cast<size_t>(w.b) * p.H + w.h) * p.NT + n;
  return w;
}

// barrier over n threads that gives all of them the same "some thread failed"
__device__ __forceinline__ bool bar_or(int id, int n, bool fail) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(n), "r"(static_cast<uint32_t>(fail))
      : "memory");
  return r != 0;
}

template <bool G_BF16, int NB>
__global__ void __launch_bounds__(W1_THREADS, 1) kda_k1w_kernel(const __grid_constant__ K1Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using SM = W1Smem<NB>;
  constexpr int BLK = SM::BLK, WPB = W1_EW / NB;   // WPB: operand warps per block
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + SM::BARS;
  // bar_gram, bar_d, bar_kx: one per parity of the item, since the roles may be two items apart
  const uint32_t bar_qk = bar0, bar_ops = bar0 + 8, bar_x = bar0 + 16;
  auto bar_gram = [&](int it) { return bar0 + 24 + (it & 1) * 8; };
  auto bar_d = [&](int it) { return bar0 + 40 + (it & 1) * 8; };
  auto bar_kx = [&](int it) { return bar0 + 56 + (it & 1) * 8; };
  auto par2 = [](int it) { return static_cast<uint32_t>((it >> 1) & 1); };
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + SM::SLOT);
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + SM::SLOT + 4);
  int* starts = reinterpret_cast<int*>(smem + SM::STARTS);
  grid_dep_launch();   // the next kernel may be set up beside this one's last items
  if (p.redo) {        // the same items over 16-token blocks, if their sums were out of the other form's range
    grid_dep_wait();
    if (*static_cast<volatile int*>(p.status + HDR_RANGE) == 0) return;
  } else if (blockIdx.x == 0 && tid == 0) {
    *reinterpret_cast<int2*>(p.status) = make_int2(ST_OK, ST_OK);
  }

  if (tid == 0) {
    mbar_init(bar_qk, 1);
    mbar_init(bar_ops, W1_EW);   // its operand tiles and its p1 tile are written
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_gram(i), 2);   // the products, and the issuing thread: what the operand warps wrote besides is visible too
      mbar_init(bar_d(i), W1_SW);  // the Grams have been read
      mbar_init(bar_kx(i), 1);
    }
    mbar_init(bar_x, W1_SW);       // X and Aqk are operands
    *sAbort = 0;
    fence_mbar_init();
  }
  if (warp == W1_EW + W1_SW) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(W1_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 0 && p.seq_table != nullptr) wide_seq_starts(p.seq_table, p.n_seqs, starts);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *slot;
  const int n_items = (p.seq_table != nullptr ? starts[p.n_seqs] : p.B * p.NT) * p.H;

  auto give_up = [&]() {
    if (*sAbort == 0) {
      *sAbort = 1;
      atomicExch(p.status, ST_K1_LOAD_TIMEOUT);
      p.status[HDR_K1_STATUS] = ST_K1_LOAD_TIMEOUT;
    }
  };

  if (warp < W1_EW) {
    // ------------------------------ gate and operands -----------------------
    const int u = lane & 15, hr = lane >> 4;    // 16-byte unit (8 columns), upper / lower two rows of the warp
    const int c0 = u * 8, row0 = warp * W1_ER + hr * 2;
    const int blk = warp / WPB;
    float* sTot = reinterpret_cast<float*>(smem + SM::TOT);
    float* sFac = reinterpret_cast<float*>(smem + SM::FAC);
    const bool use_gate = (p.flags & 1u) != 0, use_l2 = (p.flags & 2u) != 0;
    auto ld_pairs = [&](const float* at, float2 (&x)[4]) {   // this thread's eight columns of a row of 128
      const float4 a = *reinterpret_cast<const float4*>(at + c0), b = *reinterpret_cast<const float4*>(at + c0 + 4);
      x[0] = make_float2(a.x, a.y); x[1] = make_float2(a.z, a.w);
      x[2] = make_float2(b.x, b.y); x[3] = make_float2(b.z, b.w);
    };
    int it = 0;
    for (int id = blockIdx.x; id < n_items; ++it, id += gridDim.x) {
      const int slot4 = it & (W1_SLOTS - 1);
      const W1Item cur = w1_item(p, starts, id);
      const int nvalid = cur.nvalid;
      // per-item parameters; these warps have the time to wait for them
      const float a_log = use_gate ? ldg_pinned(p.A_log + cur.h) : 0.f;
      float2 bias[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        bias[c] = (use_gate && p.dt_bias != nullptr) ? ldg_pinned2(p.dt_bias + cur.h * D + c0 + 2 * c) : make_float2(0.f, 0.f);
      const int brow = warp * W1_ER + (lane & (W1_ER - 1));
      float bact = brow < nvalid ? ldg_pinned(p.beta + cur.b * p.beta_s[0] + static_cast<int64_t>(cur.t0 + brow) * p.beta_s[1] + cur.h * p.beta_s[2]) : 0.f;
      bool ok = true;

      // ---- gate: running sums over this thread's two rows, then over the warp's four ----
      float2 gv[2][4];   // [row][column pair]
      // the gate goes from global memory to registers: every element is read once, by one thread
      const int64_t g0 = cur.b * p.g_s[0] + static_cast<int64_t>(cur.t0) * p.g_s[1] + cur.h * p.g_s[2] + c0;
      auto ld_g = [&](int r, float2 (&x)[4]) {
        if (G_BF16) {
          const uint4 w = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.g) + g0 + r * p.g_s[1]));
          const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int c = 0; c < 4; ++c) x[c] = make_float2(bf16_lo_to_f32(a[c]), bf16_hi_to_f32(a[c]));
        } else {
          const float4* at = reinterpret_cast<const float4*>(static_cast<const float*>(p.g) + g0 + r * p.g_s[1]);
          const float4 a = __ldg(at), b = __ldg(at + 1);
          x[0] = make_float2(a.x, a.y); x[1] = make_float2(a.z, a.w);
          x[2] = make_float2(b.x, b.y); x[3] = make_float2(b.z, b.w);
        }
      };
      if (use_gate) {
        const float nA = -expf(a_log) * 1.4426950408889634f;   // exp(-z) = 2^(nA x + nA bias)
        const float2 nA2 = make_float2(nA, nA), one2 = make_float2(1.f, 1.f);
        const float lbr = p.lower_bound * RCP_LN2;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float2 x[4] = {};
          if (row0 + i < nvalid) ld_g(row0 + i, x);
          const float lb_r = row0 + i < nvalid ? lbr : 0.f;   // rows past the end add nothing
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float2 z = __ffma2_rn(x[c], nA2, make_float2(nA * bias[c].x, nA * bias[c].y));
            const float2 den = __fadd2_rn(make_float2(ex2f(z.x), ex2f(z.y)), one2);
            const float2 gate = __fmul2_rn(make_float2(rcpf(den.x), rcpf(den.y)), make_float2(lb_r, lb_r));
            gv[i][c] = i == 0 ? gate : __fadd2_rn(gv[0][c], gate);
          }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {   // the lower two rows follow the upper two
          float2 up;
          up.x = __shfl_up_sync(0xffffffffu, gv[1][c].x, 16);
          up.y = __shfl_up_sync(0xffffffffu, gv[1][c].y, 16);
          if (hr == 1) {
            gv[0][c] = __fadd2_rn(gv[0][c], up);
            gv[1][c] = __fadd2_rn(gv[1][c], up);
          }
        }
      } else {
        // g holds the log2 sums of every 16 tokens; rows past the end repeat the last valid one
        const int sub = (row0 >> 4) * 16;
        auto at = [&](int r, float2 (&x)[4]) {   // a row of the 16 tokens, or the last valid one before it
          if (sub >= nvalid) {
#pragma unroll
            for (int c = 0; c < 4; ++c) x[c] = make_float2(0.f, 0.f);
          } else {
            ld_g(min(r, nvalid - 1), x);
          }
        };
        float2 off[4];   // the sum before this warp's rows
#pragma unroll
        for (int c = 0; c < 4; ++c) off[c] = make_float2(0.f, 0.f);
        if (warp * W1_ER > sub) at(warp * W1_ER - 1, off);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float2 x[4];
          at(row0 + i, x);
#pragma unroll
          for (int c = 0; c < 4; ++c) gv[i][c] = make_float2(x[c].x - off[c].x, x[c].y - off[c].y);
        }
      }
      // every warp is done with its row of the previous item's table
      if (it > 0) ok = mbar_wait_parked(bar_ops, (it - 1) & 1, sAbort) && ok;
      if (hr == 1) {
        float4* t = reinterpret_cast<float4*>(sTot + warp * D + c0);
        t[0] = make_float4(gv[1][0].x, gv[1][0].y, gv[1][1].x, gv[1][1].y);
        t[1] = make_float4(gv[1][2].x, gv[1][2].y, gv[1][3].x, gv[1][3].y);
      }

      // ---- q, k: this thread's units, normalised and rounded to bf16; zero past the end ----
      ok = mbar_wait_parked(bar_qk, it & 1, sAbort) && ok;
      uint32_t qk[4][4];   // q rows, k rows
      const uint8_t* qt = smem + SM::QK;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 a = *reinterpret_cast<const uint4*>(qt + (j >> 1) * (WT * 256) + (row0 + (j & 1)) * 256 + u * 16);
        if (row0 + (j & 1) >= nvalid) a = make_uint4(0, 0, 0, 0);
        qk[j][0] = a.x; qk[j][1] = a.y; qk[j][2] = a.z; qk[j][3] = a.w;
      }
      if (use_l2) {
        float sq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 a = make_float2(0.f, 0.f);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float2 x = make_float2(bf16_lo_to_f32(qk[j][c]), bf16_hi_to_f32(qk[j][c]));
            a = __ffma2_rn(x, x, a);
          }
          sq[j] = a.x + a.y;
        }
        // four sums over the sixteen lanes of a row half: the first two exchanges halve the values a lane carries
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int n = 2 >> d, m = 8 >> d;
          const bool up = (lane & m) != 0;
#pragma unroll
          for (int j = 0; j < 2; ++j)
            if (j < n) {
              const float mine = up ? sq[j + n] : sq[j], other = up ? sq[j] : sq[j + n];
              sq[j] = mine + __shfl_xor_sync(0xffffffffu, other, m);
            }
        }
        sq[0] += __shfl_xor_sync(0xffffffffu, sq[0], 2);
        sq[0] += __shfl_xor_sync(0xffffffffu, sq[0], 1);
        const float rn = rsqrtf(sq[0] + L2NORM_EPS);
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // value j went to the lanes whose bits 3, 2 are bits 1, 0 of j
          const float f = __shfl_sync(0xffffffffu, rn, (lane & 16) | (j << 2));
#pragma unroll
          for (int c = 0; c < 4; ++c) qk[j][c] = pack_bf16(bf16_lo_to_f32(qk[j][c]) * f, bf16_hi_to_f32(qk[j][c]) * f);
        }
      }
      if (p.flags & 4u) bact = 1.0f / (1.0f + __expf(-bact));
      if (brow >= nvalid) bact = 0.f;
      if (lane < W1_ER) {
        reinterpret_cast<float*>(smem + SM::BETA)[slot4 * WT + brow] = bact;
        reinterpret_cast<float*>(p.rec + cur.rec_idx * WREC_BYTES + WREC_BETA)[brow] = bact;
      }

      // all of q, k, g is in registers and the warps' sums are published
      if (bar_or(1, W1_EW * 32, !ok || *sAbort != 0)) { give_up(); break; }
      if (tid < D) {
        // one column a thread: G before every warp's rows from the centre of its block (summed outwards from there, so
        // that the exponents stay as small as they are), the factors between centres, and the chunk's decay.  Factors
        // come as two equal ones: a single 2^c can underflow where its product with the other operand does not.
        float total = 0.f, since = 0.f;   // before the last centre; since then
        float widest = 0.f;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          float t[WPB];
#pragma unroll
          for (int w = 0; w < WPB; ++w) t[w] = sTot[(b * WPB + w) * D + tid];
          float acc = 0.f;
#pragma unroll
          for (int w = WPB / 2 - 1; w >= 0; --w) { acc -= t[w]; sTot[(b * WPB + w) * D + tid] = acc; }
          widest = fmaxf(widest, fabsf(acc));
          const float step = since - acc;           // from the last centre (or the start) to this one
          if (b > 0) sFac[(NB + b - 1) * D + tid] = ex2f(0.5f * step);
          total += step;
          sFac[b * D + tid] = ex2f(0.5f * total);
          since = 0.f;
#pragma unroll
          for (int w = WPB / 2; w < WPB; ++w) { sTot[(b * WPB + w) * D + tid] = since; since += t[w]; }
          widest = fmaxf(widest, fabsf(since));
        }
        if (NB == 2 && p.check_range && !(widest <= W1_RANGE)) p.status[HDR_RANGE] = 1;
        reinterpret_cast<float*>(smem + SM::SCALE)[slot4 * D + tid] = ex2f(since);
        reinterpret_cast<float*>(p.rec + cur.rec_idx * WREC_BYTES + WREC_DEC)[tid] = ex2f(total + since);
      }
      asm volatile("bar.sync 1, 512;" ::: "memory");

      // the previous item's Grams have read L and R; where -Akk and X lie over them, its last product is done too
      if (it > 0 && !mbar_wait_parked(SM::AHEAD ? bar_gram(it - 1) : bar_kx(it - 1), par2(it - 1), sAbort)) give_up();
      uint8_t* p1 = smem + SM::QK;
      const int atom = u >> 3;
      float2 t4[4];
      ld_pairs(sTot + warp * D, t4);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) gv[i][c] = __fadd2_rn(gv[i][c], t4[c]);   // G - c_blk
      ld_pairs(sFac + blk * D, t4);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = row0 + i;
        const uint32_t l_off = atom * 16384 + r * 128 + static_cast<uint32_t>(((u & 7) ^ (r & 7)) << 4);
        const float br = __shfl_sync(0xffffffffu, bact, hr * 2 + i);
        float2 e[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) e[c] = make_float2(ex2f(gv[i][c].x), ex2f(gv[i][c].y));
#pragma unroll
        for (int x = 0; x < 2; ++x) {   // k, then q
          uint32_t hi[4], lo[4], pp[4];
          const float f = x == 0 ? br : p.scale;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint32_t w = qk[(1 - x) * 2 + i][c];
            const float2 l = __fmul2_rn(make_float2(bf16_lo_to_f32(w), bf16_hi_to_f32(w)), e[c]);
            split_pack2(l, hi[c], lo[c]);
            const float2 g = __fmul2_rn(__fmul2_rn(__fmul2_rn(l, t4[c]), t4[c]), make_float2(f, f));
            pp[c] = pack_bf16(g.x, g.y);
          }
          *reinterpret_cast<uint4*>(smem + SM::LH + l_off + x * WT * 128) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(smem + SM::LL + l_off + x * WT * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          *reinterpret_cast<uint4*>(p1 + l_off + x * WT * 128) = make_uint4(pp[0], pp[1], pp[2], pp[3]);
        }
      }
      // the last R tile two items ago was the operand of that item's last product
      if (SM::AHEAD && it > 1 && !mbar_wait_parked(bar_kx(it - 2), par2(it - 2), sAbort)) give_up();
#pragma unroll
      for (int i = 0; i < 2; ++i) {   // khat 2^(c_blk - G), then version by version 2^(c_v - G)
        const int r = row0 + i;
        const uint32_t un = static_cast<uint32_t>(((u & 7) ^ (r & 7)) << 4);
        float2 kR[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t w = qk[2 + i][c];
          kR[c] = __fmul2_rn(make_float2(bf16_lo_to_f32(w), bf16_hi_to_f32(w)), make_float2(ex2f(-gv[i][c].x), ex2f(-gv[i][c].y)));
        }
#pragma unroll
        for (int v = 0; v < NB; ++v) {
          if (v < blk) continue;
          if (v > blk) {
            float2 f[4];
            ld_pairs(sFac + (NB + v - 1) * D, f);
#pragma unroll
            for (int c = 0; c < 4; ++c) kR[c] = __fmul2_rn(__fmul2_rn(kR[c], f[c]), f[c]);
          }
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) split_pack2(kR[c], hi[c], lo[c]);
          const int rows_b = BLK * 128 * (v + 1);   // bytes of one half of the tile
          uint8_t* t = smem + SM::r_tile(v) + (SM::AHEAD && v == NB - 1 ? (it & 1) * SM::R_LAST : 0) + atom * rows_b + r * 128 + un;
          *reinterpret_cast<uint4*>(t) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(t + 2 * rows_b) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ops);
    }
  } else if (warp < W1_EW + W1_SW) {
    // ------------------------------ masks, solve, outputs -------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(W1_SOLVE_REGS));
    const int quad = warp & 3, st = quad * 32 + lane;        // TMEM lane = thread of this role
    const uint32_t tl = tbase + (static_cast<uint32_t>(quad * 32) << 16);
    const int row = st & 63;                                 // token row: k rows in lanes 0..63, q rows in 64..127
    const int g4 = lane >> 2, t4 = lane & 3;
    uint8_t* sX = smem + SM::X;
    // byte offset of unit un (8 tokens t) of X^T row s_
    auto x_off = [](int s_, int un) { return static_cast<uint32_t>(s_ * 128 + ((un ^ (s_ & 7)) << 4)); };
    auto split8 = [](const float* x, uint4& hi, uint4& lo) {
      uint32_t h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split_pack2(make_float2(x[2 * j], x[2 * j + 1]), h[j], l[j]);
      hi = make_uint4(h[0], h[1], h[2], h[3]);
      lo = make_uint4(l[0], l[1], l[2], l[3]);
    };
    // two products of 16-row tiles on mma.sync, hi/lo splits of both sides: acc += a b
    auto mma3 = [](float (&acc)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4], const uint32_t* bh, const uint32_t* bl) {
      mma_bf16(acc, ah, bh[0], bh[1]);
      mma_bf16(acc, al, bh[0], bh[1]);
      mma_bf16(acc, ah, bl[0], bl[1]);
    };
    // operand fragments: rows of X^T (A, row-major), rows of X^T as k (B, transposing load)
    auto lda_x = [&](uint32_t lo_off, int s0, int un, uint32_t (&a)[4]) {
      const int r = s0 + (lane & 7) + ((lane >> 3) & 1) * 8;
      ldsm_x4(sbase + SM::X + lo_off + x_off(r, un + (lane >> 4)), a[0], a[1], a[2], a[3]);
    };
    auto ldb_x = [&](uint32_t lo_off, int m0, int un, uint32_t (&b)[4]) {
      const int r = m0 + (lane & 7) + ((lane >> 3) & 1) * 8;
      ldsm_x4_t(sbase + SM::X + lo_off + x_off(r, un + (lane >> 4)), b[0], b[1], b[2], b[3]);
    };
    auto frag = [](const float (&c0)[4], const float (&c1)[4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {   // accumulators as A operand
      split_pack2(make_float2(c0[0], c0[1]), hi[0], lo[0]);
      split_pack2(make_float2(c0[2], c0[3]), hi[1], lo[1]);
      split_pack2(make_float2(c1[0], c1[1]), hi[2], lo[2]);
      split_pack2(make_float2(c1[2], c1[3]), hi[3], lo[3]);
    };
    auto put_tile = [&](int s0, int un, const float (&c)[4]) {   // rows s0 + g4, + 8 of X^T, two tokens of unit un
      uint32_t hi, lo;
      split_pack2(make_float2(c[0], c[1]), hi, lo);
      *reinterpret_cast<uint32_t*>(sX + x_off(s0 + g4, un) + t4 * 4) = hi;
      *reinterpret_cast<uint32_t*>(sX + 8192 + x_off(s0 + g4, un) + t4 * 4) = lo;
      split_pack2(make_float2(c[2], c[3]), hi, lo);
      *reinterpret_cast<uint32_t*>(sX + x_off(s0 + 8 + g4, un) + t4 * 4) = hi;
      *reinterpret_cast<uint32_t*>(sX + 8192 + x_off(s0 + 8 + g4, un) + t4 * 4) = lo;
    };
    const bool upper = lane >= 16;
    // kx and ax of item `it` to its record; the products have been waited for
    auto outputs = [&](int id, int it) {
      tc_fence_after();
      const W1Item w = w1_item(p, starts, id);
      uint8_t* rec = p.rec + w.rec_idx * WREC_BYTES;
      const float ks = reinterpret_cast<const float*>(smem + SM::SCALE)[(it & (W1_SLOTS - 1)) * D + st];
#pragma unroll
      for (int half = 0; half < 2; ++half) {   // kx^T: lane = k, columns = tokens
        uint32_t d[32];
        tmem_ld32(tl + W1_KX + half * 32, d);
        tc_wait_ld();
        pin32(d);
#pragma unroll
        for (int un = 0; un < 4; ++un) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            split_pack2(make_float2(__uint_as_float(d[un * 8 + 2 * j]) * ks, __uint_as_float(d[un * 8 + 2 * j + 1]) * ks), hi[j], lo[j]);
          const int off = (half * 4 + un) * 2048 + st * 16;
          *reinterpret_cast<uint4*>(rec + WREC_KXH + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(rec + WREC_KXL + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      if (quad >= 2) {   // ax: lane = token row, columns = tokens up to its own
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (half == 1 && quad == 2) continue;
          uint32_t d[32];
          tmem_ld32(tl + W1_AX + half * 32, d);
          tc_wait_ld();
          pin32(d);
#pragma unroll
          for (int un = 0; un < 4; ++un) {
            const int c = half * 2 + (un >> 1);   // column panel of 16 tokens
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              split_pack2(make_float2(__uint_as_float(d[un * 8 + 2 * j]), __uint_as_float(d[un * 8 + 2 * j + 1])), hi[j], lo[j]);
            if (row >= 16 * c) {
              uint8_t* dst = rec + WREC_AX + ax_panel(c) + (un & 1) * (WT - 16 * c) * 16 + (row - 16 * c) * 16;
              *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
              *reinterpret_cast<uint4*>(dst + WREC_AX_BYTES) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
          }
        }
      }
    };
    int it = 0;
    bool ok = true;
    for (int id = blockIdx.x; id < n_items; id += gridDim.x, ++it) {
      const int slot4 = it & (W1_SLOTS - 1);
      ok = mbar_wait_parked(bar_gram(it), par2(it), sAbort) && ok;
      tc_fence_after();

      // ---- the row of this lane, 16 columns at a time: block b of the rows lies in accumulator D_b ----
      const float f = quad < 2 ? -reinterpret_cast<const float*>(smem + SM::BETA)[slot4 * WT + row] : p.scale;
      const uint32_t dcol = tl + W1_D + (SM::AHEAD ? (it & 1) * W1_D_ITEM : 0), aq = tl + W1_AQ + (it & 1) * 64;
      auto chunk = [&](int ch, uint32_t (&d)[16]) {   // columns 16 ch .. 16 ch + 15 of the row
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const bool keep = quad < 2 ? ch * 16 + j < row : ch * 16 + j <= row;
          x[j] = keep ? __uint_as_float(d[j]) * f : 0.f;   // what is masked may be anything, infinities included
        }
        uint4 h0, l0, h1, l1;
        split8(x, h0, l0);
        split8(x + 8, h1, l1);
        if (quad >= 2) {
          const uint32_t hi[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
          const uint32_t lo[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
          tmem_st8(aq + ch * 8, hi);
          tmem_st8(aq + 32 + ch * 8, lo);
        } else if (quad == 1 && ch < 2) {      // rows 32..63, columns 0..31
          uint8_t* t = smem + SM::AO2 + lane * 80 + ch * 32;
          *reinterpret_cast<uint4*>(t) = h0; *reinterpret_cast<uint4*>(t + 16) = h1;
          *reinterpret_cast<uint4*>(t + 32 * 80) = l0; *reinterpret_cast<uint4*>(t + 32 * 80 + 16) = l1;
        } else if ((ch & 1) == (upper ? 1 : 0)) {   // a diagonal block
          float4* t = reinterpret_cast<float4*>(smem + SM::AD + ((quad * 2 + (lane >> 4)) * 16 + (lane & 15)) * 80);
#pragma unroll
          for (int j = 0; j < 4; ++j) t[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        } else if (upper) {                          // block 10 or 32
          uint8_t* t = smem + SM::AO1 + quad * (2 * 16 * 48) + (lane & 15) * 48;
          *reinterpret_cast<uint4*>(t) = h0; *reinterpret_cast<uint4*>(t + 16) = h1;
          *reinterpret_cast<uint4*>(t + 16 * 48) = l0; *reinterpret_cast<uint4*>(t + 16 * 48 + 16) = l1;
        }
      };
      // two chunks at a time: this warp shares its scheduler with four busy ones and lives on independent instructions
      auto chunks = [&](int ch) {
        uint32_t d0[16], d1[16];
        if (NB == 2) {
          tmem_ld16(dcol + ((quad & 1) ? 32 : 0) + ch * 16, d0);
          tmem_ld16(dcol + ((quad & 1) ? 32 : 0) + ch * 16 + 16, d1);
          tc_wait_ld();
          pin16(d0);
          pin16(d1);
        } else {
          // lanes 0..15 of the quarter hold rows of block 2 (quad & 1), lanes 16..31 of the next; the accumulators have
          // 16, 32, 48, 64 columns, and what is read past an accumulator's end is masked
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t a[16], c[16];
            tmem_ld16(dcol + ((quad & 1) ? 48 : 0) + (ch + e) * 16, a);
            tmem_ld16(dcol + ((quad & 1) ? 96 : 16) + (ch + e) * 16, c);
            tc_wait_ld();
            pin16(a);
            pin16(c);
#pragma unroll
            for (int j = 0; j < 16; ++j) (e == 0 ? d0 : d1)[j] = upper ? c[j] : a[j];
          }
        }
        chunk(ch, d0);
        chunk(ch + 1, d1);
      };
      chunks(0);
      if (quad & 1) {
        chunks(2);
      } else if (quad == 2) {   // tokens 32..63 are not before rows 0..31
        const uint32_t z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        tmem_st8(aq + 16, z);
        tmem_st8(aq + 24, z);
        tmem_st8(aq + 48, z);
        tmem_st8(aq + 56, z);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_d(it));

      // ---- the outputs of the item before; after its products X may be rewritten ----
      if (it > 0) {
        if (mbar_wait_parked(bar_kx(it - 1), par2(it - 1), sAbort)) outputs(id - static_cast<int>(gridDim.x), it - 1);
        else ok = false;
      }
      if (quad >= 2) tc_wait_st();
      __syncwarp();
      if (quad < 2) {
        // ---- two diagonal 16 x 16 inverses, lane = column of one: column sweep, -A read four columns at a time ----
        const float* sL = reinterpret_cast<const float*>(smem + SM::AD + (quad * 2 + (lane >> 4)) * 16 * 80);
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = i == (lane & 15) ? 1.f : 0.f;
#pragma unroll
        for (int mb = 0; mb < 4; ++mb) {
#pragma unroll
          for (int i = mb * 4 + 1; i < 16; ++i) {
            const float4 l4 = *reinterpret_cast<const float4*>(sL + i * 20 + mb * 4);
            const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int mm = 0; mm < 4; ++mm)
              if (mb * 4 + mm < i) x[i] = fmaf(lv[mm], x[mb * 4 + mm], x[i]);
          }
        }
        const int s_ = quad * 32 + lane;
        const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint4 hi, lo;
          split8(x + 8 * e, hi, lo);
          *reinterpret_cast<uint4*>(sX + x_off(s_, quad * 4 + (lane >> 4) * 2 + e)) = hi;
          *reinterpret_cast<uint4*>(sX + 8192 + x_off(s_, quad * 4 + (lane >> 4) * 2 + e)) = lo;
          if (upper) {   // tokens before the row's own block
            *reinterpret_cast<uint4*>(sX + x_off(s_, quad * 4 + e)) = z;
            *reinterpret_cast<uint4*>(sX + 8192 + x_off(s_, quad * 4 + e)) = z;
          }
        }
        if (quad == 1) {
#pragma unroll
          for (int un = 0; un < 4; ++un) {
            *reinterpret_cast<uint4*>(sX + x_off(s_, un)) = z;
            *reinterpret_cast<uint4*>(sX + 8192 + x_off(s_, un)) = z;
          }
        }
        __syncwarp();
        // ---- 32 x 32: X10^T = (X00^T (-A10)^T) X11^T; the first product's accumulators are the second's A operand ----
        uint32_t ah[4], al[4], bh[4], bl[4];
        const int n0 = quad * 32, un0 = quad * 4;
        lda_x(0, n0, un0, ah);
        lda_x(8192, n0, un0, al);
        const uint32_t ao = sbase + SM::AO1 + quad * (2 * 16 * 48) + ((lane & 7) + ((lane >> 4) & 1) * 8) * 48 + ((lane >> 3) & 1) * 16;
        ldsm_x4(ao, bh[0], bh[1], bh[2], bh[3]);
        ldsm_x4(ao + 16 * 48, bl[0], bl[1], bl[2], bl[3]);
        float y[2][4] = {};
#pragma unroll
        for (int j = 0; j < 2; ++j) mma3(y[j], ah, al, bh + 2 * j, bl + 2 * j);
        frag(y[0], y[1], ah, al);
        ldb_x(0, n0 + 16, un0 + 2, bh);
        ldb_x(8192, n0 + 16, un0 + 2, bl);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float c[4] = {};
          mma3(c, ah, al, bh + 2 * j, bl + 2 * j);
          put_tile(n0, un0 + 2 + j, c);
        }
      }
      if (bar_or(2, W1_SW * 32, !ok || *sAbort != 0)) { give_up(); break; }
      {
        // ---- 64 x 64, the same: this warp's 16 columns s, all 32 rows m between, 16 of the rows t ----
        const int s0 = (quad & 1) * 16, th = quad >> 1;
        uint32_t ah[2][4], al[2][4];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          lda_x(0, s0, kk * 2, ah[kk]);
          lda_x(8192, s0, kk * 2, al[kk]);
        }
        float c[2][4] = {};
#pragma unroll
        for (int mp = 0; mp < 2; ++mp) {   // 16 of the rows m: accumulators y, then a k-step of the second product
          float y[2][4] = {};
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            uint32_t bh[4], bl[4];
            const uint32_t ao = sbase + SM::AO2 + (mp * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * 80 + kk * 32 + ((lane >> 3) & 1) * 16;
            ldsm_x4(ao, bh[0], bh[1], bh[2], bh[3]);
            ldsm_x4(ao + 32 * 80, bl[0], bl[1], bl[2], bl[3]);
#pragma unroll
            for (int j = 0; j < 2; ++j) mma3(y[j], ah[kk], al[kk], bh + 2 * j, bl + 2 * j);
          }
          uint32_t yh[4], yl[4], bh[4], bl[4];
          frag(y[0], y[1], yh, yl);
          ldb_x(0, 32 + mp * 16, 4 + th * 2, bh);
          ldb_x(8192, 32 + mp * 16, 4 + th * 2, bl);
#pragma unroll
          for (int j = 0; j < 2; ++j) mma3(c[j], yh, yl, bh + 2 * j, bl + 2 * j);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) put_tile(s0, 4 + th * 2 + j, c[j]);
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_x);
    }
    if (it > 0 && ok && *sAbort == 0) {
      if (mbar_wait_parked(bar_kx(it - 1), par2(it - 1), sAbort)) outputs(blockIdx.x + (it - 1) * static_cast<int>(gridDim.x), it - 1);
      else give_up();
    }
  } else {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(W1_ISSUE_REGS));
   if (warp == W1_EW + W1_SW) {
    // ------------------------------ MMA issue -------------------------------
    const int mine = n_items > static_cast<int>(blockIdx.x) ? (n_items - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    auto grams = [&](int it) -> bool {
      constexpr int ND = SM::AHEAD ? 2 : 1;   // items whose accumulators exist
      if (!mbar_wait_parked(bar_ops, it & 1, sAbort)) return false;
      if (it >= ND && !mbar_wait_parked(bar_d(it - ND), par2(it - ND), sAbort)) return false;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll 1
        for (int v = 0; v < NB; ++v) {
          const int rows_b = BLK * 128 * (v + 1), rt = SM::r_tile(v) + (SM::AHEAD && v == NB - 1 ? (it & 1) * SM::R_LAST : 0);
          const uint32_t dcol = tbase + W1_D + (SM::AHEAD ? (it & 1) * W1_D_ITEM : 0) + BLK * v * (v + 1) / 2;
          const uint32_t idesc = instr_desc(128, BLK * (v + 1), 0);
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            const uint64_t dlh = smem_desc(sbase + SM::LH + half * 16384, 16, 1024, 2), dll = smem_desc(sbase + SM::LL + half * 16384, 16, 1024, 2);
            const uint64_t drh = smem_desc(sbase + rt + half * rows_b, 16, 1024, 2), drl = smem_desc(sbase + rt + (2 + half) * rows_b, 16, 1024, 2);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              umma_ss(dcol, dlh + 2 * ks, drh + 2 * ks, idesc, half + ks != 0);
              umma_ss(dcol, dll + 2 * ks, drh + 2 * ks, idesc, 1);
              umma_ss(dcol, dlh + 2 * ks, drl + 2 * ks, idesc, 1);
            }
          }
        }
        umma_commit(bar_gram(it));
        mbar_arrive(bar_gram(it));
      }
      __syncwarp();
      return true;
    };
    auto right = [&](int it) -> bool {   // kx^T and ax
      if (!mbar_wait_parked(bar_x, it & 1, sAbort)) return false;
      tc_fence_after();
      if (elect_one()) {
        const int rt = SM::r_tile(NB - 1) + (SM::AHEAD ? (it & 1) * SM::R_LAST : 0);
        const uint32_t aq = tbase + W1_AQ + (it & 1) * 64;
#pragma unroll 1
        for (int c = 3; c >= 0; --c) {   // 16 tokens t: X[t][s] is zero beyond s = 16 c + 15
          const uint32_t id_kx = instr_desc(128, 16 * (c + 1), 0, 1), id_ax = instr_desc(128, 16 * (c + 1), 0);
          const uint64_t dah = smem_desc(sbase + rt + c * 2048, 8192, 1024, 2), dal = smem_desc(sbase + rt + 16384 + c * 2048, 8192, 1024, 2);
          const uint64_t dxh = smem_desc(sbase + SM::X + c * 32, 16, 1024, 2), dxl = smem_desc(sbase + SM::X + 8192 + c * 32, 16, 1024, 2);
          umma_ss(tbase + W1_KX, dah, dxh, id_kx, c != 3);
          umma_ss(tbase + W1_KX, dal, dxh, id_kx, 1);
          umma_ss(tbase + W1_KX, dah, dxl, id_kx, 1);
          // lanes 64..127 of A are Aqk; the others are not read from the result
          umma_ts(tbase + W1_AX, aq + c * 8, dxh, id_ax, c != 3);
          umma_ts(tbase + W1_AX, aq + 32 + c * 8, dxh, id_ax, 1);
          umma_ts(tbase + W1_AX, aq + c * 8, dxl, id_ax, 1);
        }
        umma_commit(bar_kx(it));
      }
      __syncwarp();
      return true;
    };
    // the Grams of the next item go before the products that wait for this one's solve; where the next item's operands
    // take the place of this one's, after them
    for (int it = 0; it <= mine; ++it) {
      const bool good = SM::AHEAD ? (it == mine || grams(it)) && (it == 0 || right(it - 1))
                                  : (it == 0 || right(it - 1)) && (it == mine || grams(it));
      if (!good) { give_up(); break; }
    }
   } else if (warp == W1_EW + W1_SW + 1) {
    // ------------------------------ copies ----------------------------------
    if (lane == 0) {
      constexpr uint32_t ROW_BYTES = D * 2;
      const int step = gridDim.x;
      auto load_qk = [&](int id) {
        const W1Item w = w1_item(p, starts, id);
        mbar_arrive_expect_tx(bar_qk, 2 * WT * ROW_BYTES);
        tma_load_4d(sbase + SM::QK, &p.tm_q, 0, w.hq, w.t0, w.b, bar_qk);
        tma_load_4d(sbase + SM::QK + WT * ROW_BYTES, &p.tm_k, 0, w.hq, w.t0, w.b, bar_qk);
      };
      // the next item's inputs come into L2 while this one is worked on; q and k go to their place once the p1 tile has left it
      auto prefetch = [&](int id) {
        const W1Item w = w1_item(p, starts, id);
        tma_prefetch_l2_4d(&p.tm_q, 0, w.hq, w.t0, w.b);
        tma_prefetch_l2_4d(&p.tm_k, 0, w.hq, w.t0, w.b);
        tma_prefetch_l2_4d(&p.tm_g, 0, w.h, w.t0, w.b);
      };
      int id = blockIdx.x, it = 0, qk_issued = 0;
      if (id < n_items) {
        load_qk(id);
        qk_issued = 1;
      }
      for (; id < n_items; id += step, ++it) {
        const W1Item w = w1_item(p, starts, id);
        const bool more = id + step < n_items;
        if (more) prefetch(id + step);
        if (!mbar_wait_parked(bar_ops, it & 1, sAbort)) { give_up(); break; }
        bulk_s2g(p.rec + w.rec_idx * WREC_BYTES + WREC_P1, sbase + SM::QK, WREC_P1_BYTES);
        bulk_commit();
        bulk_wait_read_all();
        if (more) { load_qk(id + step); qk_issued = it + 2; }
      }
      bulk_wait_read_all();
      // a copy still in flight gets a bounded chance to land before the shared memory goes
      if (*sAbort != 0 && qk_issued > 0) mbar_wait_parked(bar_qk, (qk_issued - 1) & 1, nullptr);
    }
    __syncwarp();
   }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == W1_EW + W1_SW)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(W1_COLS) : "memory");
}

template <bool G_BF16, int NB>
cudaError_t launch_k1w_t(const K1Params& p, cudaStream_t stream) {
  constexpr int smem_bytes = W1Smem<NB>::TOTAL;
  static std::atomic<int> sms_of[64];   // per device, published after the attribute is set
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64) return cudaErrorInvalidDevice;
  int sms = sms_of[dev].load(std::memory_order_acquire);
  if (sms == 0) {
    auto kern = kda_k1w_kernel<G_BF16, NB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    sms_of[dev].store(sms, std::memory_order_release);
  }
  // packed: the number of wide chunks is known on the device only; it is at most that of chunks of 16
  const long long n_items = (p.seq_table != nullptr ? static_cast<long long>(p.n_chunks) : static_cast<long long>(p.B) * p.NT) * p.H;
  const int grid = static_cast<int>(n_items < sms ? n_items : sms);
  return launch_dep(kda_k1w_kernel<G_BF16, NB>, grid, W1_THREADS, smem_bytes, stream, p.redo, p);
}

}  // namespace

cudaError_t launch_k1w(const K1Params& p, bool g_bf16, bool two_blocks, cudaStream_t stream) {
  if (g_bf16) return two_blocks ? launch_k1w_t<true, 2>(p, stream) : launch_k1w_t<true, 4>(p, stream);
  return two_blocks ? launch_k1w_t<false, 2>(p, stream) : launch_k1w_t<false, 4>(p, stream);
}

}  // namespace kda
