// Shared device helpers and the K1 -> K2 chunk-record contract (sm_100a only).
//
// A "chunk record" is the 26,112-byte block K1 writes and K2 reads for one
// (batch, head, chunk-of-16-tokens).  Records are chunk-major:
//   record index c = (b * H + h) * NT + n        (same order as the reference's
//   chunk-major packing, python/kda_ascendc_v1/layout.py:17-25)
// so the stream one (b, h) recurrence walks is contiguous in HBM and every
// stage is one bulk (TMA) copy.
//
//   offset  bytes  contents
//   0       8192   -w, qg    bf16, two halves of 64 k: [half][-w, qg][16 tok][64 k], the eight 16-byte units of a
//                            128-byte row XOR-permuted by the row index (wq_off)
//   8192    4096   kg_h      bf16 [2 token halves][128 k][8 tok] \ hi/lo split of khat * 2^(g_last - g),
//   12288   4096   kg_l      bf16 [2][128][8]                    / transposed (kg_off)
//   16384   1024   Aqk       bf16 [2 column halves][hi, lo][16 i][8 j]: hi/lo split of the scaled lower triangle
//                            incl. diagonal (aq_off)
//   17408   512    dec       fp32 [128]      = 2^(g_last)
//   17920   512    Xb_h      bf16 [2 column halves][16 i][8 j] \ hi/lo split of X diag(beta), X = (I + Akk)^-1
//   18432   512    Xb_l      bf16 [2][16][8]                   / (xb_off)
//   18944   512    dec       fp32 again, in the order in which the 8-row K2's lanes read it (dec_lane_off)
//   19456   4096   v         bf16 [2 halves of 64 columns][16 tok][64], 16-byte units permuted as in w (v_off)
// (23,552 of the 26,112 bytes; a record that held u as fp32 used them all)
//
// with qg = bf16(qhat * 2^g).  u = X diag(beta) v is not stored: K2 adds it up from Xb and v, which is exact in bf16, on
// the accumulator of -w h (2.5 KiB less to write and to read, and K1 computes nothing with v).  After a plain bulk copy into shared memory (1024-byte aligned) every part is a tensor-core
// operand as it stands: [w; qg] is a 32-row K-major operand in the 128-byte swizzle of tcgen05 (8-row groups 1024
// bytes apart), kg^T and Aqk are 8x8 core matrices of 128 contiguous bytes (K-major without swizzle).  tcgen05.mma
// reads them by descriptor, and every 8x8 matrix of an ldmatrix is free of bank conflicts, most of them at
// an immediate offset.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace kda {

constexpr int BT = 16;
constexpr int D = 128;
constexpr int TILE_BYTES = BT * D * 2;  // 4096
constexpr int REC_W = 0;         // w of half hf at REC_W + hf * REC_HALF, qg at REC_QG + hf * REC_HALF
constexpr int REC_QG = 2048;
constexpr int REC_HALF = 4096;
constexpr int REC_KGH = 8192;
constexpr int REC_KGL = 12288;
constexpr int REC_AQK = 16384;   // hi; lo at REC_AQL
constexpr int REC_AQL = 16640;
constexpr int REC_DEC = 17408;
constexpr int REC_XBH = 17920;
constexpr int REC_XBL = 18432;
constexpr int REC_DEC2 = 18944;
constexpr int REC_V = 19456;             // 64 columns of v at REC_V + half * REC_V_HALF
constexpr int REC_V_HALF = 2048;
constexpr int REC_SHARED_BYTES = 19456;  // everything every V-slice needs
constexpr int REC_USED_BYTES = 23552;
// From record to record.  kda_fwd_workspace_bytes and the problems that the fixed scratch holds follow from it, and callers have
// sized their buffers by it; records 23,552 bytes apart take the same time (T8192 H32 327.8 us either way, H96 634, T65536 H16 1,731).
constexpr int REC_BYTES = 26112;
constexpr int WS_HEADER_BYTES = 256;     // status block at the start of the workspace
// Header words: 0 = status; HDR_K1_STATUS = K1's own code, which no later kernel overwrites (K2 waits for K1, so a K1
// that gave up makes K2's waits run out after it; a first-one-wins exchange in K2 instead costs its 8-row form 0.7 %:
// T8192 H32 411.7 -> 414.5 us); for a K2 that runs beside K1 (zeroed before K1 starts; unused
// otherwise) HDR_TICKET = K1 items handed out, HDR_ARRIVED = K1 CTAs that have started, HDR_PROGRESS .. = finished K1 items
// per window of chunks
constexpr int HDR_K1_STATUS = 1;
constexpr int HDR_TICKET = 2;
constexpr int HDR_ARRIVED = 3;
constexpr int HDR_PROGRESS = 4;
constexpr int MAX_WINDOWS = WS_HEADER_BYTES / 4 - HDR_PROGRESS;

// status codes written to workspace[0] by a kernel that gave up on a wait
constexpr int ST_OK = 0;
constexpr int ST_K1_LOAD_TIMEOUT = 1;
constexpr int ST_K2_FULL_TIMEOUT = 2;
constexpr int ST_K2_EMPTY_TIMEOUT = 3;
constexpr int ST_K1_WINDOW_TIMEOUT = 8;   // K2 beside K1: a window of chunks was not finished in time
constexpr int ST_PEER_TIMEOUT = 7;   // a flag from another GPU did not arrive in time (sequence-split exchange)

constexpr float RCP_LN2 = 1.44269504089f;  // literal of tests/test_torch_reference.py:87
constexpr float L2NORM_EPS = 1e-6f;

// one second is plenty for a copy that normally takes a microsecond
constexpr unsigned long long WAIT_LIMIT_NS = 1000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Swizzled bf16 tile of K1: element (r, c) of a [16][128] tile, the eight 16-byte units of each 128-byte half row
// XOR-permuted by the row index, so that every ldmatrix (8 rows, same column unit) is free of bank conflicts.
__device__ __forceinline__ uint32_t swz_off(int r, int c) {
  return static_cast<uint32_t>(r * 256 + ((((c >> 3) ^ (r & 7)) << 4) | ((c & 7) << 1)));
}

// the record's tiles: element offsets in bytes (w / qg relative to their part of half 0, see above)
__device__ __forceinline__ uint32_t wq_off(int r, int c) {
  return static_cast<uint32_t>((c >> 6) * REC_HALF + r * 128 + (((((c >> 3) & 7) ^ (r & 7)) << 4) | ((c & 7) << 1)));
}
__device__ __forceinline__ uint32_t kg_off(int tok, int k) {
  return static_cast<uint32_t>((tok >> 3) * 2048 + k * 16 + (tok & 7) * 2);
}
__device__ __forceinline__ uint32_t aq_off(int i, int j) {
  return static_cast<uint32_t>((j >> 3) * 512 + i * 16 + (j & 7) * 2);
}

__device__ __forceinline__ uint32_t xb_off(int i, int j) {
  return static_cast<uint32_t>((j >> 3) * 256 + i * 16 + (j & 7) * 2);
}
__device__ __forceinline__ uint32_t v_off(int tok, int v) {
  return static_cast<uint32_t>((v >> 6) * REC_V_HALF + tok * 128 + (((((v >> 3) & 7) ^ (tok & 7)) << 4) | ((v & 7) << 1)));
}
// lane (g = lane / 4) of the 8-row K2 holds k = 16 m + g and 16 m + 8 + g, m = 0..7: four 16-byte loads
__device__ __forceinline__ uint32_t dec_lane_off(int k) {
  return static_cast<uint32_t>((k >> 5) * 128 + (k & 7) * 16 + ((k >> 3) & 3) * 4);
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One lane of a converged warp, chosen by the hardware.  Measured: eight tcgen05.mma M128 N32 issue in 37 cycles behind
// elect.sync and in 402 behind `lane == 0`, presumably because only the former tells the compiler that one thread is there.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// ---- mbarrier ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after WAIT_LIMIT_NS (or as soon as *abort_flag is set by
// another warp of the CTA) and returns false; the caller records a status code and
// unwinds.  Never spins forever.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity,
                                                  volatile int* abort_flag) {
  if (mbar_test_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (abort_flag != nullptr && *abort_flag != 0) return false;
    if (globaltimer_ns() - t0 > WAIT_LIMIT_NS) return false;
  }
}

// ---- flags between GPUs (peer memory) ------------------------------------------
// A flag is an int32 epoch counter in the waiting GPU's own memory; a peer raises it with a
// system-scope release store after its data stores, the owner polls it with system-scope acquire
// loads.  Bounded like every other wait: false after WAIT_LIMIT_NS.
__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(int* p, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ bool flag_wait_bounded(const int* flag, int epoch) {
  if (ld_acquire_sys(flag) - epoch >= 0) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (ld_acquire_sys(flag) - epoch >= 0) return true;
    if (globaltimer_ns() - t0 > WAIT_LIMIT_NS) return false;
  }
}

// ---- K1 -> K2 hand-over on one GPU ------------------------------------------------
// Programmatic dependent launch: K1 lets the next kernel of the stream start early, K2 waits for the
// whole of K1 before it reads what K1 wrote.  Both are no-ops in an ordinary launch.
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// fence between the generic and the async proxy for every state space (the plain form above covers
// shared memory only): global memory written with plain stores and read by bulk copies, or the reverse
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void red_release_gpu(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// A K2 that runs beside K1: waits until the K1 items of a window of chunks are all finished, then makes
// their records readable by this thread's bulk copies.  Bounded; *abort_flag ends it early.
__device__ __forceinline__ bool window_wait_bounded(const int* progress, int target, volatile int* abort_flag) {
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i) {
      int v;
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(progress) : "memory");
      if (v >= target) {
        fence_proxy_async_all();
        return true;
      }
      __nanosleep(64);
    }
    if (*abort_flag != 0 || globaltimer_ns() - t0 > WAIT_LIMIT_NS) return false;
  }
}

// Chains of packed sequences in order of length, longest sequence first (ties by index): the chain
// (sequence * H + head) at place `place`.  Called by every thread of the CTA; one warp works it out, bit by bit: the
// length at a place is the largest that more than `place` sequences reach.
constexpr int MAX_SORTED_SEQS = 256;
__device__ __forceinline__ int chain_by_length(const int4* seq_table, int n_seqs, int H, int place) {
  __shared__ int chosen;
  if (threadIdx.x < 32) {
    constexpr int PER_LANE = MAX_SORTED_SEQS / 32;
    const int lane = threadIdx.x, pos = place / H;
    int len[PER_LANE], longest = 0;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      len[j] = j * 32 + lane < n_seqs ? __ldg(&seq_table[j * 32 + lane].y) : 0;   // every sequence has a chunk
      longest = max(longest, len[j]);
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    int at = 0, above = 0;
    for (int bit = 31 - __clz(longest); bit >= 0; --bit) {
      const int t = at | (1 << bit);
      int n = 0;
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j) n += len[j] >= t ? 1 : 0;
      if (__reduce_add_sync(0xffffffffu, n) > pos) at = t;
    }
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) above += len[j] > at ? 1 : 0;
    int k = pos - __reduce_add_sync(0xffffffffu, above);   // place among the sequences of this length
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const unsigned same = __ballot_sync(0xffffffffu, len[j] == at);
      if (len[j] == at && __popc(same & ((1u << lane) - 1)) == k) chosen = j * 32 + lane;
      k -= __popc(same);
    }
  }
  __syncthreads();
  return chosen * H + place % H;
}

// ---- bulk (TMA, untiled) copies ---------------------------------------------
// global -> shared, completion counted in bytes on an mbarrier.  Both addresses
// 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t dst_smem, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_smem),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// tiled TMA load of one box of a 4-D tensor map (coordinates innermost first)
__device__ __forceinline__ void tma_load_4d(uint32_t dst_smem, const void* tmap, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::
          "r"(dst_smem), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src_smem), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// ---- shared-memory loads pinned where they are written ------------------------------
__device__ __forceinline__ float2 lds_f32x2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 lds_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

__device__ __forceinline__ uint4 lds_u32x4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// a 4-byte global store by the lanes for which c holds, without a branch
__device__ __forceinline__ void stg_u32_if(void* p, uint32_t v, bool c) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.u32 [%0], %1;\n\t}" ::"l"(p), "r"(v),
               "r"(static_cast<int>(c))
               : "memory");
}

// ---- ldmatrix / mma ---------------------------------------------------------
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// four 8x8 b16 matrices in fragment layout, transposed: lane 8 i + r gives the address of row r of matrix i^T
__device__ __forceinline__ void stsm_x4_t(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2),
               "r"(r3)
               : "memory");
}
// transpose an 8x8 b16 matrix held as one register per lane (fragment layout) inside the warp
__device__ __forceinline__ uint32_t movmatrix_t(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ void ldsm_x2_t(uint32_t addr, uint32_t& r0, uint32_t& r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}
// D(16x8,f32) += A(16x16,bf16,row) * B(16x8,bf16,col)
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// same instruction, but pinned in program order (used where independent loads and stores are
// deliberately interleaved with a long MMA sequence so that their latency is covered)
__device__ __forceinline__ void mma_bf16_v(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// D = A * B with a zero accumulator: the first MMA of a chain needs no register initialisation
__device__ __forceinline__ void mma_bf16_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// Read-only global loads pinned where they are written: used to fetch per-item parameters a whole
// iteration before their use, which the compiler would otherwise sink next to the use.
__device__ __forceinline__ float ldg_pinned(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 ldg_pinned2(const float* p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// ---- bf16 helpers -----------------------------------------------------------
// pack two floats (round to nearest even) into one register: lo -> bits 0..15
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float bf16_lo_to_f32(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bf16_hi_to_f32(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ unsigned short bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
// hi/lo split of two floats: hi = bf16(x), lo = bf16(x - hi)
__device__ __forceinline__ void split_pack(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x0, x1);
  lo = pack_bf16(x0 - bf16_lo_to_f32(hi), x1 - bf16_hi_to_f32(hi));
}
// packed variant on a float2 (one f32x2 FMA for the residual)
__device__ __forceinline__ void split_pack2(float2 x, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x.x, x.y);
  const float2 r = __ffma2_rn(make_float2(bf16_lo_to_f32(hi), bf16_hi_to_f32(hi)), make_float2(-1.f, -1.f), x);
  lo = pack_bf16(r.x, r.y);
}
// u + (a + b) of two neighbours of an accumulator fragment, as a hi/lo pair
__device__ __forceinline__ void split_pack_sum(const float* u, const float* a, const float* b, uint32_t& hi, uint32_t& lo) {
  const float2 s = __fadd2_rn(make_float2(a[0], a[1]), make_float2(b[0], b[1]));
  split_pack2(__fadd2_rn(make_float2(u[0], u[1]), s), hi, lo);
}
__device__ __forceinline__ float rcpf(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

}  // namespace kda
