// The wide K1 -> K2 contract: one record per (batch, head, 64 tokens).  sm_100a only.
//
// Within a chunk of C = 64 tokens, with G the cumulative log2 gate (G_t <= 0), X = (I + Akk)^-1 and
// r_t = beta_t v_t - kb_t S^T, the chunk's work on the state S [V][K] is
//   S' = S diag(dec) + r^T kx          kb = beta khat 2^G,  kx = X^T (khat 2^(G_last - G)),  dec = 2^G_last
//   o  = qg S^T + ax r                 qg = scale qhat 2^G, ax = (scale tril(qhat khat^T 2^(G_i - G_j))) X
// i.e. the reference's w = X kb, u = X (beta v), v_new = u - w S^T with the inverse moved from the left of the
// state products to their right.  u does not travel: K2 reads v itself, exact in bf16.
//
//   offset  bytes   contents
//   0       32768   p1: bf16 [2 halves of 64 k][128 rows: kb 0..63, qg 64..127][64 k], the eight 16-byte units of a
//                   128-byte row XOR-permuted by row & 7 (the tensor core's 128-byte swizzle)
//   32768   16384   kx hi \ bf16 [8 units of 8 tokens][128 k][8 tokens]: 8 x 16-byte core matrices, K-major in tokens
//   49152   16384   kx lo /
//   65536   5120    ax hi \ lower block triangle by 16-token column panels: panel c holds rows 16c..63 as
//   70656   5120    ax lo /   [2 units of 8 tokens][64 - 16 c rows][8 tokens]
//   75776   512     dec fp32 [128]
//   76288   256     beta fp32 [64] (activated; 0 past the end)
// 76,544 bytes per 64 tokens against 4 x 26,112 of the 16-token records.
#pragma once
#include "kda_common.cuh"

namespace kda {

constexpr int WT = 64;                 // tokens of a wide chunk
constexpr int WREC_P1 = 0;
constexpr int WREC_P1_BYTES = 32768;
constexpr int WREC_KXH = 32768;
constexpr int WREC_KXL = 49152;
constexpr int WREC_AX = 65536;
constexpr int WREC_AX_BYTES = 5120;    // one of hi, lo
constexpr int WREC_DEC = 75776;
constexpr int WREC_BETA = 76288;
constexpr int WREC_SMALL_BYTES = 768;  // dec and beta
constexpr int WREC_BYTES = 76544;
__host__ __device__ constexpr int ax_panel(int c) { return 32 * (64 * c - 8 * c * (c - 1)); }   // byte offset of column panel c
static_assert(ax_panel(4) == WREC_AX_BYTES && ax_panel(1) == 2048 && ax_panel(2) == 3584, "panels of 64, 48, 32, 16 rows");
static_assert(WREC_BYTES % 256 == 0, "bulk copies and swizzled atoms want aligned records");

// Packed sequences: first wide chunk of every sequence, [n_seqs + 1], by one warp.
constexpr int WIDE_MAX_SEQS = 256;
__device__ __forceinline__ void wide_seq_starts(const int4* seq_table, int n_seqs, int* starts) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int j = 0; j < n_seqs; j += 32) {
    const int n = j + lane < n_seqs ? (__ldg(&seq_table[j + lane].w) + WT - 1) / WT : 0;
    int sum = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += up;
    }
    if (j + lane < n_seqs) starts[j + lane] = base + sum - n;
    base += __shfl_sync(0xffffffffu, sum, 31);
  }
  if (lane == 0) starts[n_seqs] = base;
}

}  // namespace kda
