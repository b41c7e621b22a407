// Exact mod-2^16 dot products of u16 share matrices on tcgen05 INT8 tensor cores.
//
// Replaces the reference's three cublasGemmEx int8 limb GEMMs plus the
// matmul_correct_and_reduce kernel (iris-mpc-gpu/src/dot/share_db.rs:62-112,
// 800-905; iris-mpc-gpu/src/dot/kernel.cu:16-28).  Each u16 is split into two
// unsigned bytes (lo, hi); since
//     d*q mod 2^16 = dlo*qlo + 2^8 * (dlo*qhi + dhi*qlo)   (mod 2^16)
// one pass over K issues three u8 x u8 -> s32 MMAs per K step into two TMEM
// accumulators: acc0 += Dlo.Qlo and acc1 += Dlo.Qhi + Dhi.Qlo.  The epilogue
// forms (acc0 + (acc1 << 8)) mod 2^16, multiplies by the engine multiplier
// (2 for trimmed masks), adds the zero-share mask ks_own - ks_prev computed in
// registers with ChaCha12, and stores u16 dot shares.  Unsigned limbs need no
// sum correction (the reference's signed limbs do).
//
// Layouts: DB limb planes [entries][K] u8, query limb planes [rows][K] u8
// (both K-major, K a multiple of 128), output [entries][n_pad] u16 with the
// query row fastest.  Keystream u16 of element (entry m, row n) sits at index
// m * n_pad + n of the engine's stream (32 u16 per ChaCha block).
//
// Kernel structure (one CTA per SM, persistent over tiles of 128 entries x BN
// rows): warp 0 issues TMA loads (128B swizzle) into a STAGES-deep ring,
// warp 1 allocates TMEM and issues the MMAs from one thread, warps 2..9 drain
// the accumulators (tcgen05.ld), release TMEM to the next tile and then run
// the ChaCha mask and the stores while the next tile's MMAs proceed.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <algorithm>
#include "common.cuh"
#include "gemm_limb.h"
#include "quad_gemm.h"
#include "tc_sm100.cuh"
#include "tc_pair.cuh"
#include "launch_attr.cuh"

namespace irs {

namespace {

constexpr int kThreads = 320;

template <int BN>
struct Cfg {
  static constexpr int kStageBytes = 2 * kBM * kBK + 2 * BN * kBK;
  static constexpr int kStages = (196608 / kStageBytes) > 6 ? 6 : (196608 / kStageBytes);
  static constexpr int kTmemCols = 2 * BN;  // acc0 | acc1
  static constexpr int kColsPerThread = BN / 2;  // two epilogue warps per TMEM lane quadrant
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/;
};

struct Tile {
  int prob, m_tile, n_tile;
};

__device__ __forceinline__ bool tile_of(const GemmParams& P, int t, Tile& out) {
  for (int i = 0; i < P.n_prob; i++) {
    const int nt = (int)(P.prob[i].tiles_m * P.prob[i].tiles_n);
    if (t < nt) {
      out.prob = i;
      out.m_tile = t / (int)P.prob[i].tiles_n;
      out.n_tile = t % (int)P.prob[i].tiles_n;
      return true;
    }
    t -= nt;
  }
  return false;
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) limb_gemm_kernel(const __grid_constant__ GemmParams P) {
  using C = Cfg<BN>;
  if (P.skip.n && P.skip.all_set()) return;  // the quad GEMM runs
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a_lo = smem;
  uint8_t* a_hi = a_lo + C::kStages * kBM * kBK;
  uint8_t* b_lo = a_hi + C::kStages * kBM * kBK;
  uint8_t* b_hi = b_lo + C::kStages * BN * kBK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(b_hi + C::kStages * BN * kBK);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* acc_full = bars + 2 * C::kStages;
  uint64_t* acc_empty = acc_full + 1;
  uint64_t* done_bar = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 3);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int* err = P.err;
  // The MMA's wait for a TMA stage has the launch's limit; every other wait
  // (which in a failing launch only follows that one) twice as long, so the
  // first expiry names the stage that never arrived.
  const uint64_t lim = P.wait_timeout_ns, lim2 = 2 * P.wait_timeout_ns;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 8);  // one arrive per epilogue warp
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)C::kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued_phase[8];
      bool issued[8];
      for (int s = 0; s < C::kStages; s++) issued[s] = false;
      bool ok = true;
      const bool hinted = P.l2_hint != 0;
      const uint64_t pol_a = (P.l2_hint & 2u) ? policy_evict_first() : policy_evict_normal();
      const uint64_t pol_b = (P.l2_hint & 1u) ? policy_evict_last() : policy_evict_normal();
      // Test hook (GemmParams::test_stall): CTA 0 issues no loads at all, so
      // its MMA's first stage wait runs out.  Nothing is in flight to drain.
      if (P.test_stall && blockIdx.x == 0) ok = false;
      for (int k = 0; ok && k * (int)gridDim.x < P.total_tiles; k++) {
        Tile tl;
        if (!tile_of(P, tile_index(k, blockIdx.x, gridDim.x), tl)) continue;
        const GemmProblem& pr = P.prob[tl.prob];
        const int ya = (int)pr.m0 + tl.m_tile * kBM;
        const int yb = tl.n_tile * BN;
        const bool rev = P.serpentine && (k & 1);
        for (uint32_t ki = 0; ki < pr.k_iters; ki++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, err, kErrTimeoutEmpty, lim2)) { ok = false; break; }
          mbar_expect_tx(&full_bar[stage], (uint32_t)C::kStageBytes);
          const int x = (int)(rev ? pr.k_iters - 1 - ki : ki) * kBK;
          if (hinted) {
            tma_load_2d_hint(a_lo + stage * kBM * kBK, &pr.tm_a_lo, &full_bar[stage], x, ya, pol_a);
            tma_load_2d_hint(a_hi + stage * kBM * kBK, &pr.tm_a_hi, &full_bar[stage], x, ya, pol_a);
            tma_load_2d_hint(b_lo + stage * BN * kBK, &pr.tm_b_lo, &full_bar[stage], x, yb, pol_b);
            tma_load_2d_hint(b_hi + stage * BN * kBK, &pr.tm_b_hi, &full_bar[stage], x, yb, pol_b);
          } else {
            tma_load_2d(a_lo + stage * kBM * kBK, &pr.tm_a_lo, &full_bar[stage], x, ya);
            tma_load_2d(a_hi + stage * kBM * kBK, &pr.tm_a_hi, &full_bar[stage], x, ya);
            tma_load_2d(b_lo + stage * BN * kBK, &pr.tm_b_lo, &full_bar[stage], x, yb);
            tma_load_2d(b_hi + stage * BN * kBK, &pr.tm_b_hi, &full_bar[stage], x, yb);
          }
          issued[stage] = true;
          issued_phase[stage] = (int)phase;
          if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
        }
      }
      // Exit: make sure no copy into this CTA's shared memory is still in flight.
      for (int s = 0; s < C::kStages; s++)
        if (issued[s]) mbar_wait_drain(&full_bar[s], (uint32_t)issued_phase[s], err, lim2);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      constexpr uint32_t idesc = idesc_u8(BN);
      for (int k = 0; ok && k * (int)gridDim.x < P.total_tiles; k++) {
        Tile tl;
        if (!tile_of(P, tile_index(k, blockIdx.x, gridDim.x), tl)) continue;
        const GemmProblem& pr = P.prob[tl.prob];
        if (!mbar_wait(acc_empty, acc_phase ^ 1u, err, kErrTimeoutAccEmpty, lim2)) { ok = false; break; }
        acc_phase ^= 1u;
        tc_fence_after();
        for (uint32_t ki = 0; ki < pr.k_iters; ki++) {
          if (!mbar_wait(&full_bar[stage], phase, err, kErrTimeoutFull, lim)) { ok = false; break; }
          tc_fence_after();
          const uint64_t dal = smem_desc(a_lo + stage * kBM * kBK);
          const uint64_t dah = smem_desc(a_hi + stage * kBM * kBK);
          const uint64_t dbl = smem_desc(b_lo + stage * BN * kBK);
          const uint64_t dbh = smem_desc(b_hi + stage * BN * kBK);
#pragma unroll
          for (int kk = 0; kk < kBK / 32; kk++) {
            const uint32_t acc = (ki > 0 || kk > 0) ? 1u : 0u;
            const uint64_t o = (uint64_t)(2 * kk);  // 32 bytes along K, in 16-byte units
            mma_u8(tmem, dal + o, dbl + o, idesc, acc);
            mma_u8(tmem + BN, dal + o, dbh + o, idesc, acc);
            mma_u8(tmem + BN, dah + o, dbl + o, idesc, 1u);
          }
          mma_commit(&empty_bar[stage]);
          if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
        }
        if (ok) mma_commit(acc_full);
      }
      // Exit: wait until every MMA issued by this thread has completed.
      mma_commit(done_bar);
      mbar_wait_drain(done_bar, 0, err, lim2);
    }
  } else {
    // ---------------- Epilogue (warps 2..9) ----------------
    const int quad = warp & 3;                 // TMEM lanes 32*quad .. 32*quad+31
    const int half = (warp - 2) >> 2;          // column half of the tile
    const int row = quad * 32 + lane;          // entry within the tile
    constexpr int kCols = C::kColsPerThread;
    uint32_t acc_phase = 0;
    for (int k = 0; k * (int)gridDim.x < P.total_tiles; k++) {
      Tile tl;
      if (!tile_of(P, tile_index(k, blockIdx.x, gridDim.x), tl)) continue;
      const GemmProblem& pr = P.prob[tl.prob];
      if (!mbar_wait(acc_full, acc_phase, err, kErrTimeoutAccFull, lim2)) break;
      acc_phase ^= 1u;
      tc_fence_after();
      uint32_t packed[kCols / 2];
      const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * kCols);
#pragma unroll
      for (int c = 0; c < kCols / 32; c++) {
        uint32_t r0[32], r1[32];
        tmem_ld32(tbase + (uint32_t)(c * 32), r0);
        tmem_ld32(tbase + (uint32_t)(BN + c * 32), r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const uint32_t lo = (r0[2 * j] + (r1[2 * j] << 8)) & 0xFFFFu;
          const uint32_t hi = (r0[2 * j + 1] + (r1[2 * j + 1] << 8)) << 16;
          packed[c * 16 + j] = lo | hi;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);

      const uint32_t m_local = (uint32_t)(tl.m_tile * kBM + row);
      if (m_local < pr.m_len) {
        const uint64_t m_global = (uint64_t)pr.m0 + m_local;
        uint16_t* out_row = pr.out + (size_t)m_local * pr.n_pad;
#pragma unroll
        for (int c = 0; c < kCols / 32; c++) {
          const uint32_t n = (uint32_t)(tl.n_tile * BN + half * kCols + c * 32);
          if (n >= pr.n_pad) break;  // part-filled last tile
          uint32_t v[16];
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const uint32_t x = packed[c * 16 + j];
            v[j] = (pr.mult == 1) ? x : (((x & 0xFFFFu) * pr.mult) & 0xFFFFu) | (((x >> 16) * pr.mult) << 16);
          }
          if (pr.mask_on) {
            const uint64_t blk = (m_global * pr.n_pad + n) >> 5;
            const uint64_t batch = pr.batch_dev ? *pr.batch_dev : pr.batch;
            uint32_t ks[32];
            chacha12_pair(&pr.key_own, &pr.key_prev, counter_of(batch, blk), pr.nonce, ks);
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = sub2(add2(v[j], ks[j]), ks[16 + j]);
          }
          uint4* dst = reinterpret_cast<uint4*>(out_row + n);
#pragma unroll
          for (int q = 0; q < 4; q++) dst[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)C::kTmemCols));
  }
}

// ---------------------------------------------------------------------------
// Two-SM variant: a cluster of two CTAs computes a 256-entry x 256-row tile
// with tcgen05.mma.cta_group::2 (M = 256).  Each CTA loads its own 128 entries
// (A) and half of the 256 query rows (B); the leader CTA (rank 0) issues the
// MMAs, which read the A and B halves from both CTAs' shared memory, and each
// CTA's TMEM receives the accumulator rows of its own entries.  Per SM this
// halves the B bytes written into and read from shared memory, which is what
// bounds the one-SM kernel (about 156 of 128 B/clk at full MMA rate).
// TMA completions of both CTAs land on the leader's stage barriers; stage and
// accumulator barriers are released to both CTAs with multicast commits; the
// follower's epilogue releases the accumulator on the leader's barrier.
// ---------------------------------------------------------------------------
// Tiles are 64 to 256 rows wide, in multiples of 64 (an epilogue half then holds
// whole keystream blocks), a problem's as equal as that allows.
constexpr int kPairRoom = 225 * 1024;  // shared memory for the stages
constexpr int kPairMaxStages = 5;
constexpr int kPairMaxN = 256;
constexpr int kPairSmem = kPairRoom + 1024 /*align*/ + 256 /*barriers*/;
constexpr int pair_stage_bytes(int bn) { return 2 * 128 * kBK + 2 * (bn / 2) * kBK; }  // per CTA

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    limb_gemm_pair_kernel(const __grid_constant__ GemmParams P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int n_stages = P.pair_stages;
  const int b_bytes = P.pair_n / 2 * kBK;  // one limb of a CTA's half of the query rows
  uint8_t* a_lo = smem;
  uint8_t* a_hi = a_lo + n_stages * 128 * kBK;
  uint8_t* b_lo = a_hi + n_stages * 128 * kBK;
  uint8_t* b_hi = b_lo + n_stages * b_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPairRoom);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kPairMaxStages;
  uint64_t* acc_full = bars + 2 * kPairMaxStages;
  uint64_t* acc_empty = acc_full + 1;
  uint64_t* done_bar = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 3);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int cluster = blockIdx.x >> 1;
  const int n_clusters = gridDim.x >> 1;
  // A problem's rows, in units of 64, dealt out over its tiles: the first
  // `wider` are pair_n rows, the others 64 fewer.
  auto tile_width = [&](const Tile& tl) { return P.pair_n - (tl.n_tile < P.pair_wider ? 0 : 64); };
  auto tile_row = [&](const Tile& tl) {
    return tl.n_tile * P.pair_n - (tl.n_tile > P.pair_wider ? 64 * (tl.n_tile - P.pair_wider) : 0);
  };
  int* err = P.err;
  const uint64_t lim = P.wait_timeout_ns, lim2 = 2 * P.wait_timeout_ns;

  if (P.skip.n && cluster_reads(P.skip, tmem_slot)) return;  // the quad GEMM runs
  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 16);  // 8 epilogue warps in each CTA
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // peer barriers initialised before any remote arrive
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t issued_phase = 0, issued = 0;  // bit s: stage s
      bool ok = true;
      for (int k = 0; ok && k * n_clusters < P.total_tiles; k++) {
        Tile tl;
        if (!tile_of(P, tile_index(k, cluster, n_clusters), tl)) continue;
        const GemmProblem& pr = P.prob[tl.prob];
        const int ya = (int)pr.m0 + tl.m_tile * kBM2 + (int)rank * 128;
        const int yb = tile_row(tl) + (int)rank * (tile_width(tl) / 2);
        const bool rev = P.serpentine && (k & 1);
        for (uint32_t ki = 0; ki < pr.k_iters; ki++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, err, kErrTimeoutEmpty, lim2)) { ok = false; break; }
          if (leader) mbar_expect_tx(&full_bar[stage], (uint32_t)(2 * pair_stage_bytes(P.pair_n)));
          const uint32_t fb = map_to_rank(&full_bar[stage], 0);
          const int x = (int)(rev ? pr.k_iters - 1 - ki : ki) * kBK;
          tma_load_2d_pair(a_lo + stage * 128 * kBK, &pr.tm_a_lo, fb, x, ya);
          tma_load_2d_pair(a_hi + stage * 128 * kBK, &pr.tm_a_hi, fb, x, ya);
          tma_load_2d_pair(b_lo + stage * b_bytes, &pr.tm_b_lo, fb, x, yb);
          tma_load_2d_pair(b_hi + stage * b_bytes, &pr.tm_b_hi, fb, x, yb);
          issued |= 1u << stage;
          issued_phase = (issued_phase & ~(1u << stage)) | phase << stage;
          if (++stage == n_stages) { stage = 0; phase ^= 1u; }
        }
      }
      // Exit: the leader's stage barriers complete only when both CTAs' copies
      // of that stage have landed.
      if (leader)
        for (int s = 0; s < n_stages; s++)
          if ((issued >> s) & 1u) mbar_wait_drain(&full_bar[s], (issued_phase >> s) & 1u, err, lim2);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (lane == 0 && leader) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int k = 0; ok && k * n_clusters < P.total_tiles; k++) {
        Tile tl;
        if (!tile_of(P, tile_index(k, cluster, n_clusters), tl)) continue;
        const GemmProblem& pr = P.prob[tl.prob];
        const uint32_t idesc = idesc_u8_m256(tile_width(tl));
        if (!mbar_wait(acc_empty, acc_phase ^ 1u, err, kErrTimeoutAccEmpty, lim2)) { ok = false; break; }
        acc_phase ^= 1u;
        tc_fence_after();
        for (uint32_t ki = 0; ki < pr.k_iters; ki++) {
          if (!mbar_wait(&full_bar[stage], phase, err, kErrTimeoutFull, lim)) { ok = false; break; }
          tc_fence_after();
          const uint64_t dal = smem_desc(a_lo + stage * 128 * kBK);
          const uint64_t dah = smem_desc(a_hi + stage * 128 * kBK);
          const uint64_t dbl = smem_desc(b_lo + stage * b_bytes);
          const uint64_t dbh = smem_desc(b_hi + stage * b_bytes);
#pragma unroll
          for (int kk = 0; kk < kBK / 32; kk++) {
            const uint32_t acc = (ki > 0 || kk > 0) ? 1u : 0u;
            const uint64_t o = (uint64_t)(2 * kk);
            mma_u8_pair(tmem, dal + o, dbl + o, idesc, acc);
            mma_u8_pair(tmem + kPairMaxN, dal + o, dbh + o, idesc, acc);
            mma_u8_pair(tmem + kPairMaxN, dah + o, dbl + o, idesc, 1u);
          }
          mma_commit_pair(&empty_bar[stage]);
          if (++stage == n_stages) { stage = 0; phase ^= 1u; }
        }
        if (ok) mma_commit_pair(acc_full);
      }
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(done_bar))
                   : "memory");
      mbar_wait_drain(done_bar, 0, err, lim2);
    }
  } else {
    // ---------------- Epilogue (warps 2..9, both CTAs) ----------------
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    constexpr int kCols = kPairMaxN / 2;  // at most
    const uint32_t acc_empty_leader = map_to_rank(acc_empty, 0);
    uint32_t acc_phase = 0;
    for (int k = 0; k * n_clusters < P.total_tiles; k++) {
      Tile tl;
      if (!tile_of(P, tile_index(k, cluster, n_clusters), tl)) continue;
      const GemmProblem& pr = P.prob[tl.prob];
      const int cols = tile_width(tl) / 2;  // this half's query rows, a multiple of 32
      if (!mbar_wait(acc_full, acc_phase, err, kErrTimeoutAccFull, lim2)) break;
      acc_phase ^= 1u;
      tc_fence_after();
      uint32_t packed[kCols / 2];
      const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * cols);
#pragma unroll
      for (int c = 0; c < kCols / 32; c++) {
        if (c * 32 >= cols) break;
        uint32_t r0[32], r1[32];
        tmem_ld32(tbase + (uint32_t)(c * 32), r0);
        tmem_ld32(tbase + (uint32_t)(kPairMaxN + c * 32), r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const uint32_t lo = (r0[2 * j] + (r1[2 * j] << 8)) & 0xFFFFu;
          const uint32_t hi = (r0[2 * j + 1] + (r1[2 * j + 1] << 8)) << 16;
          packed[c * 16 + j] = lo | hi;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty_leader);

      const uint32_t m_local = (uint32_t)(tl.m_tile * kBM2 + (int)rank * 128 + row);
      if (m_local < pr.m_len) {
        const uint64_t m_global = (uint64_t)pr.m0 + m_local;
        uint16_t* out_row = pr.out + (size_t)m_local * pr.n_pad;
#pragma unroll
        for (int c = 0; c < kCols / 32; c++) {
          const uint32_t n = (uint32_t)(tile_row(tl) + half * cols + c * 32);
          if (c * 32 >= cols || n >= pr.n_pad) break;
          uint32_t v[16];
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const uint32_t x = packed[c * 16 + j];
            v[j] = (pr.mult == 1) ? x : (((x & 0xFFFFu) * pr.mult) & 0xFFFFu) | (((x >> 16) * pr.mult) << 16);
          }
          if (pr.mask_on) {
            const uint64_t blk = (m_global * pr.n_pad + n) >> 5;
            const uint64_t batch = pr.batch_dev ? *pr.batch_dev : pr.batch;
            uint32_t ks[32];
            chacha12_pair(&pr.key_own, &pr.key_prev, counter_of(batch, blk), pr.nonce, ks);
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = sub2(add2(v[j], ks[j]), ks[16 + j]);
          }
          uint4* dst = reinterpret_cast<uint4*>(out_row + n);
#pragma unroll
          for (int q = 0; q < 4; q++) dst[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while its peer may still touch its memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// ---------------------------------------------------------------------------
// Few tiles: a tile's K loop is a chain of pipeline round trips (about 0.6 us
// per 128-byte block), and with fewer tiles than SMs most of the GPU has none.
// Here a cluster of S CTAs (4 or 8) shares a tile, each taking its part of the K
// blocks, and the partial sums meet over distributed shared memory: CTA r of
// the cluster adds up columns [32 r, 32 r + 32) of the tile (mod 2^16), adds
// the mask and stores them (CTAs past BN / 32 only send).  One tile per
// cluster, not persistent.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void st_cluster(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

template <int BN, int S>
__global__ void __cluster_dims__(S, 1, 1) __launch_bounds__(kThreads, 1)
    limb_gemm_split_kernel(const __grid_constant__ GemmParams P) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a_lo = smem;
  uint8_t* a_hi = a_lo + C::kStages * kBM * kBK;
  uint8_t* b_lo = a_hi + C::kStages * kBM * kBK;
  uint8_t* b_hi = b_lo + C::kStages * BN * kBK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(b_hi + C::kStages * BN * kBK);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* acc_full = bars + 2 * C::kStages;
  uint64_t* done_bar = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 2);
  uint32_t* recv = reinterpret_cast<uint32_t*>(smem);  // [sender][word of 2 columns][row], over the stages

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  int* err = P.err;
  const uint64_t lim = P.wait_timeout_ns, lim2 = 2 * P.wait_timeout_ns;
  Tile tl;
  tile_of(P, blockIdx.x / S, tl);  // one cluster per tile
  const GemmProblem& pr = P.prob[tl.prob];
  const uint32_t k_begin = pr.k_iters * (uint32_t)rank / S, k_end = pr.k_iters * (uint32_t)(rank + 1) / S;

  if (P.skip.n && cluster_reads(P.skip, tmem_slot)) return;  // the quad GEMM runs
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)C::kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  constexpr int kCols = C::kColsPerThread;  // of one epilogue thread
  const int quad = warp & 3;
  const int half = (warp - 2) >> 2;
  const int row = quad * 32 + lane;
  uint32_t packed[kCols / 2];
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      int issued_phase[C::kStages];
      bool issued[C::kStages];
      for (int s = 0; s < C::kStages; s++) issued[s] = false;
      int stage = 0;
      uint32_t phase = 0;
      const int ya = (int)pr.m0 + tl.m_tile * kBM, yb = tl.n_tile * BN;
      for (uint32_t ki = k_begin; ki < k_end; ki++) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u, err, kErrTimeoutEmpty, lim2)) break;
        mbar_expect_tx(&full_bar[stage], (uint32_t)C::kStageBytes);
        const int x = (int)ki * kBK;
        tma_load_2d(a_lo + stage * kBM * kBK, &pr.tm_a_lo, &full_bar[stage], x, ya);
        tma_load_2d(a_hi + stage * kBM * kBK, &pr.tm_a_hi, &full_bar[stage], x, ya);
        tma_load_2d(b_lo + stage * BN * kBK, &pr.tm_b_lo, &full_bar[stage], x, yb);
        tma_load_2d(b_hi + stage * BN * kBK, &pr.tm_b_hi, &full_bar[stage], x, yb);
        issued[stage] = true;
        issued_phase[stage] = (int)phase;
        if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
      }
      // no copy into the stages may be in flight when they become the receive buffer
      for (int s = 0; s < C::kStages; s++)
        if (issued[s]) mbar_wait_drain(&full_bar[s], (uint32_t)issued_phase[s], err, lim2);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      constexpr uint32_t idesc = idesc_u8(BN);
      for (uint32_t ki = k_begin; ki < k_end; ki++) {
        if (!mbar_wait(&full_bar[stage], phase, err, kErrTimeoutFull, lim)) { ok = false; break; }
        tc_fence_after();
        const uint64_t dal = smem_desc(a_lo + stage * kBM * kBK);
        const uint64_t dah = smem_desc(a_hi + stage * kBM * kBK);
        const uint64_t dbl = smem_desc(b_lo + stage * BN * kBK);
        const uint64_t dbh = smem_desc(b_hi + stage * BN * kBK);
#pragma unroll
        for (int kk = 0; kk < kBK / 32; kk++) {
          const uint32_t acc = (ki > k_begin || kk > 0) ? 1u : 0u;
          const uint64_t o = (uint64_t)(2 * kk);
          mma_u8(tmem, dal + o, dbl + o, idesc, acc);
          mma_u8(tmem + BN, dal + o, dbh + o, idesc, acc);
          mma_u8(tmem + BN, dah + o, dbl + o, idesc, 1u);
        }
        mma_commit(&empty_bar[stage]);
        if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
      }
      if (ok) mma_commit(acc_full);
      mma_commit(done_bar);
      mbar_wait_drain(done_bar, 0, err, lim2);
    }
  } else {
    ok = mbar_wait(acc_full, 0, err, kErrTimeoutAccFull, lim2);
    if (ok) {
      tc_fence_after();
      const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * kCols);
#pragma unroll
      for (int c = 0; c < kCols / 32; c++) {
        uint32_t r0[32], r1[32];
        tmem_ld32(tbase + (uint32_t)(c * 32), r0);
        tmem_ld32(tbase + (uint32_t)(BN + c * 32), r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const uint32_t lo = (r0[2 * j] + (r1[2 * j] << 8)) & 0xFFFFu;
          const uint32_t hi = (r0[2 * j + 1] + (r1[2 * j + 1] << 8)) << 16;
          packed[c * 16 + j] = lo | hi;
        }
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  cluster_sync_all();  // every CTA's stages are free
  if (warp >= 2 && ok) {
#pragma unroll
    for (int c = 0; c < kCols / 32; c++) {
      const int to = half * (kCols / 32) + c;
      if (to == rank) continue;
      const uint32_t dst = map_to_rank(recv + (rank * 16) * kBM + row, (uint32_t)to);
#pragma unroll
      for (int j = 0; j < 16; j++) st_cluster(dst + (uint32_t)(j * kBM * 4), packed[c * 16 + j]);
    }
  }
  cluster_sync_all();  // the partial sums have arrived
  const uint32_t m_local = (uint32_t)(tl.m_tile * kBM + row);
  const uint32_t n = (uint32_t)(tl.n_tile * BN + rank * 32);
  if (warp >= 2 && half == rank / (kCols / 32) && m_local < pr.m_len && n < pr.n_pad && !has_error(err)) {
    uint32_t v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
      uint32_t x = packed[j];
#pragma unroll
      for (int c = 1; c < kCols / 32; c++)
        if (rank % (kCols / 32) == c) x = packed[c * 16 + j];
#pragma unroll
      for (int s = 0; s < S; s++)
        if (s != rank) x = add2(x, recv[(s * 16 + j) * kBM + row]);
      v[j] = (pr.mult == 1) ? x : (((x & 0xFFFFu) * pr.mult) & 0xFFFFu) | (((x >> 16) * pr.mult) << 16);
    }
    if (pr.mask_on) {
      const uint64_t blk = (((uint64_t)pr.m0 + m_local) * pr.n_pad + n) >> 5;
      const uint64_t batch = pr.batch_dev ? *pr.batch_dev : pr.batch;
      uint32_t ks[32];
      chacha12_pair(&pr.key_own, &pr.key_prev, counter_of(batch, blk), pr.nonce, ks);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = sub2(add2(v[j], ks[j]), ks[16 + j]);
    }
    uint4* dst = reinterpret_cast<uint4*>(pr.out + (size_t)m_local * pr.n_pad + n);
#pragma unroll
    for (int q = 0; q < 4; q++) dst[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)C::kTmemCols));
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

}  // namespace

int make_tmap_plane(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (k % 16) || box_rows > 256) return -2;
  cuuint64_t dims[2] = {k, rows};
  cuuint64_t strides[1] = {k};
  cuuint32_t box[2] = {(cuuint32_t)kBK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

int make_tmap_u8(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows) {
  return k % kBK ? -2 : make_tmap_plane(map, base, rows, k, box_rows);
}

template <int BN>
static cudaError_t launch_bn(const GemmParams& P, int n_sms, cudaStream_t stream) {
  using C = Cfg<BN>;
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = smem_limit_once(limb_gemm_kernel<BN>, C::kSmemBytes, attr_done);
  if (e != cudaSuccess) return e;
  const int grid = P.total_tiles < n_sms ? P.total_tiles : n_sms;
  if (grid <= 0) return cudaSuccess;
  limb_gemm_kernel<BN><<<grid, kThreads, C::kSmemBytes, stream>>>(P);
  return cudaGetLastError();
}

template <int BN, int S>
static cudaError_t launch_split(const GemmParams& P, cudaStream_t stream) {
  using C = Cfg<BN>;
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = smem_limit_once(limb_gemm_split_kernel<BN, S>, C::kSmemBytes, attr_done);
  if (e != cudaSuccess) return e;
  limb_gemm_split_kernel<BN, S><<<S * P.total_tiles, kThreads, C::kSmemBytes, stream>>>(P);
  return cudaGetLastError();
}

static cudaError_t launch_pair(const GemmParams& P, int n_sms, cudaStream_t stream) {
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = smem_limit_once(limb_gemm_pair_kernel, kPairSmem, attr_done);
  if (e != cudaSuccess) return e;
  const int clusters = P.total_tiles < n_sms / 2 ? P.total_tiles : n_sms / 2;
  if (clusters <= 0) return cudaSuccess;
  limb_gemm_pair_kernel<<<2 * clusters, kThreads, kPairSmem, stream>>>(P);
  return cudaGetLastError();
}

// The pair kernel reaches a higher MAC rate per clock but, at the B200's
// 1000 W limit, pulls the SM clock down with it: up to 768 query rows it gains
// all the same, above that the one-SM kernel is the default for long launches
// and the batch autotuner decides per batch shape (irs_sharedb_set_pair).
bool gemm_pair_applies(bool pair, uint32_t n_pad) { return pair && n_pad >= 128; }

int gemm_pair_n(uint32_t n_pad) {
  const uint32_t tiles = (n_pad + kPairMaxN - 1) / kPairMaxN;
  return (int)(((n_pad + tiles - 1) / tiles + 63) / 64 * 64);
}

// Measured on 65,536-entry chunks of the six engines: up to 768 query rows
// the 128-row tile (3 pipeline stages) beats the 256-row tile (2 stages) by
// 5-20%, since the pass is still close to streaming the DB; from 1024 rows,
// and on whole-DB passes, the 256-row tile wins (1024 rows: 66.8 against
// 76.9 ms on 524,288 entries).  Row counts that are no multiple of the tile
// part-fill the last one: the 64-row tile that would divide them runs at half
// the rate (960 rows x 32,768 entries, one engine: 1.51 ms, against 0.81).
// 832 and 896 rows (where the query capacity leaves no room for 1024) would fill
// three quarters and less of a fourth 256-row tile: 896 rows, six engines x
// 32,279 entries, 3.38 ms on four, 3.10 on seven of 128.
int gemm_block_n_for(uint32_t n_pad) {
  if (n_pad == 0 || n_pad % 64) return 0;
  return n_pad <= 64 ? 64 : n_pad <= 896 ? 128 : 256;
}

// L2 policy of the one-SM kernel's loads (GemmParams::l2_hint), opt-in through
// IRS_GEMM_L2HINT.  Measured at 524,288 entries x 2048 query rows: the query
// planes are re-read from DRAM once per sweep of the 148 CTAs over the DB
// (about 1.8x the algorithmic bytes in all), but DRAM runs at ~16% of its
// bandwidth under this tensor-bound kernel, and keeping the queries with
// evict_last saved 2% of the traffic while slowing the GEMM by 3% and the
// following threshold kernel by 18% (the pinned lines outlive the GEMM).
// Marking the streaming DB evict_first (value 2) instead tripled the reads
// on 65,536-entry chunks (31-48 GB against 13.7 GB per launch: each DB tile
// is read by the wave's 8 query-tile CTAs, and the hint drops it between
// them), and under the power cap the clock fell from 1567 to ~1365 MHz, 14%
// slower per batch.
static uint32_t gemm_l2_hint() {
  static const uint32_t hint = [] {
    const char* e = getenv("IRS_GEMM_L2HINT");
    return e ? (uint32_t)atoi(e) & 3u : 0u;
  }();
  return hint;
}

// CTAs that share a tile's K loop (1: the persistent kernel).  Six engines, cold
// caches, persistent / four / eight: 64 entries x 64 rows (6 tiles) 62 / 25.6 /
// 21.5 us; 64 x 256 (12) 71 / 29.8 / 25.6; 500 x 32 (24) 64 / 29.7 / 33.8; 1000 x
// 32 (48) 66 / 46; 700 x 256 (72) 77 / 67; 2000 x 32 (96) 75 / 73.  One engine
// (tiles of one length, so the persistent kernel has no short ones to wait
// with): 39 tiles 13.2 / 14.3, 68 tiles 40 / 50.  Eight pay while all tiles run
// at once; four while the longest do, and the shorter ones add at most half as
// much again.
static int gemm_k_split(const uint32_t* k_iters, const uint32_t* tiles, int n_prob, int block_n, int n_sms) {
  uint32_t least = ~0u, most = 0, total = 0;
  for (int i = 0; i < n_prob; i++) {
    least = std::min(least, k_iters[i]);
    most = std::max(most, k_iters[i]);
    total += tiles[i];
  }
  if (block_n > 128 || least < 8) return 1;
  if (8 * total <= (uint32_t)n_sms && least >= 16) return 8;
  uint64_t longest = 0, blocks = 0;
  for (int i = 0; i < n_prob; i++) {
    if (k_iters[i] == most) longest += tiles[i];
    blocks += (uint64_t)tiles[i] * k_iters[i];
  }
  return 4 * longest <= (uint64_t)n_sms && 8 * blocks <= 3ull * (uint64_t)n_sms * most ? 4 : 1;
}

double last_done(const uint32_t* tiles, const double* cost, int n_prob, int units) {
  double total = 0;
  uint32_t count = 0;
  for (int i = 0; i < n_prob; i++) {
    total += tiles[i] * cost[i];
    count += tiles[i];
  }
  constexpr int kMostUnits = 512;
  // many rounds: the last one does not matter
  if (count > 16u * (uint32_t)units || units > kMostUnits) return total / units;
  double busy[kMostUnits] = {};
  int k = 0, u = 0;
  for (int i = 0; i < n_prob; i++)
    for (uint32_t t = 0; t < tiles[i]; t++) {
      busy[(size_t)((k & 1) ? units - 1 - u : u)] += cost[i];
      if (++u == units) { u = 0; k++; }
    }
  return *std::max_element(busy, busy + units);
}

int few_rounds_tile(const uint32_t* K, int n_prob, uint32_t m_len, uint32_t n_pad, int n_sms) {
  uint32_t one[kMaxGemmProblems], two[kMaxGemmProblems], k_iters[kMaxGemmProblems], total = 0, total_64 = 0;
  double cost_one[kMaxGemmProblems], cost_two[kMaxGemmProblems];
  for (int i = 0; i < n_prob; i++) {
    const uint32_t m = (m_len + 127) / 128;
    one[i] = m * ((n_pad + 127) / 128);
    two[i] = (m_len + kBM2 - 1) / kBM2 * ((n_pad + kPairMaxN - 1) / kPairMaxN);
    k_iters[i] = K[i] / 128;
    cost_one[i] = k_iters[i] * kOneSmStep + 1000;
    cost_two[i] = k_iters[i] * plain_pair_step(n_pad) + 1000;
    total += one[i];
    total_64 += m * (n_pad / 64);
  }
  if (total_64 <= (uint32_t)n_sms && gemm_k_split(k_iters, one, n_prob, 128, n_sms) == 1) return 64;
  if (total <= (uint32_t)n_sms) return 128;
  if (total > 4u * (uint32_t)n_sms) return 0;
  return last_done(one, cost_one, n_prob, n_sms) < 0.97 * last_done(two, cost_two, n_prob, n_sms / 2) ? 128 : 0;
}

cudaError_t launch_limb_gemm(GemmParams& P, int block_n, bool pair, int n_sms, cudaStream_t stream) {
  if (P.wait_timeout_ns == 0) P.wait_timeout_ns = kGemmWaitTimeoutNs;
  P.l2_hint = gemm_l2_hint();
  // Serpentine K order (GemmParams::serpentine), on unless IRS_GEMM_SERPENTINE=0.
  // Measured with the query planes re-read once per wave: DRAM reads per
  // 65,536-entry one-SM launch 11.46 GB against 13.2-13.9 GB in K order, per
  // 32,768-entry two-SM launch 11.1-11.6 against 11.8-12.2 GB on the same
  // GPU; batch times unchanged (within 0.3%), results identical.
  static const uint32_t serp = [] {
    const char* e = getenv("IRS_GEMM_SERPENTINE");
    return e ? (uint32_t)(atoi(e) != 0) : 1u;
  }();
  P.serpentine = serp;
  const uint32_t bm = pair ? (uint32_t)kBM2 : (uint32_t)kBM;
  if (pair) {
    P.pair_n = gemm_pair_n(P.prob[0].n_pad);
    const int units = (int)P.prob[0].n_pad / 64, tiles = (int)(P.prob[0].n_pad + kPairMaxN - 1) / kPairMaxN;
    // Tiles of unequal length drift apart and share less of L2, equal ones pad
    // the rows.  32,768 entries, unequal / equal, one engine and six: 704 rows
    // (padded by 1/11) 0.622 / 0.623 and 2.60 / 2.63 ms, 896 (2/14) 0.709 / 0.753
    // and 3.09 / 3.37, 960 (1/15) 0.798 / 0.763 and 3.72 / 3.62, 1216 (1/19) 0.972
    // / 0.962 and 4.36 / 4.61, 1984 (1/31) 1.503 / 1.467 and 7.59 / 8.16, in long
    // runs 8.50 / 7.96.  From a fifteenth down they are as good or better.
    const int spare = P.pair_n / 64 * tiles - units;  // units of padding if all tiles were as wide
    P.pair_wider = 15 * spare <= units ? tiles : units % tiles;
    block_n = kPairMaxN;  // the tiles of a problem: as many as 256-row ones
    P.pair_stages = std::min(kPairMaxStages, kPairRoom / pair_stage_bytes(P.pair_n));
  }
  P.total_tiles = 0;
  uint32_t tiles[kMaxGemmProblems], k_iters[kMaxGemmProblems];
  for (int i = 0; i < P.n_prob; i++) {
    GemmProblem& pr = P.prob[i];
    pr.tiles_m = (pr.m_len + bm - 1) / bm;
    pr.tiles_n = (pr.n_pad + (uint32_t)block_n - 1) / (uint32_t)block_n;
    tiles[i] = pr.tiles_m * pr.tiles_n;
    k_iters[i] = pr.k_iters;
    P.total_tiles += (int)tiles[i];
  }
  if (pair) return launch_pair(P, n_sms, stream);
  switch (P.test_stall ? 1 : gemm_k_split(k_iters, tiles, P.n_prob, block_n, n_sms)) {
    case 4: return block_n == 64 ? launch_split<64, 4>(P, stream) : launch_split<128, 4>(P, stream);
    case 8: return block_n == 64 ? launch_split<64, 8>(P, stream) : launch_split<128, 8>(P, stream);
  }
  switch (block_n) {
    case 256: return launch_bn<256>(P, n_sms, stream);
    case 128: return launch_bn<128>(P, n_sms, stream);
    case 64: return launch_bn<64>(P, n_sms, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace irs
