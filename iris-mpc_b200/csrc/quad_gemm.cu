// Limb GEMM over rotation-structured query rows, with 9/16 of the products.
//
// The rotations of a query are shifts of one vector along the 200 columns, so
// the 31 x K query matrix of a slot is a Toeplitz matrix in (rotation, column)
// and its product with a DB record is a short correlation.  Two levels of the
// two-way split of a Toeplitz product (S. Winograd's minimal filtering
// F(2, 2): three products for two outputs and two taps instead of four) give
// four rotations of a query from nine products of a quarter of K:
//
// Let rows i and i + D of a slot hold rotations D apart and let the columns
// split into c and c + D (bit D of the column index clear or set), d0 and d1
// the record's coefficients there.  With f(t) the query at column offset t =
// c - i: row i reads x0 = f(t) against d0 and x1 = f(t + D) against d1, row
// i + D reads y0 = f(t - D) against d0 and y1 = f(t) against d1.  So
//     P2 = (d0 + d1) . f,  Px = d1 . (f(t + D) - f),  Py = d0 . (f(t - D) - f)
//     row i = P2 + Px,     row i + D = P2 + Py       (mod 2^16, exact)
// The split is applied with D = 4 (outer) and again with D = 2 (inner): 200
// columns divide by both, and rows i, i+2, i+4, i+6 of a slot form a quad.
// The additions run in Z_2^16 before the limb split: on the DB side once per
// record (derive_sums_kernel), on the query side once per upload
// (expand_kernel), on the products in the epilogue.
//
// Every term is exact modulo 2^16, so the dot shares equal the limb GEMM's
// (gemm_limb.cu) bit for bit; the limbs, the keystream positions and the
// result layout are the same.
//
// What bounds it: the board's power limit, with the tensor pipe 78% active at
// the clock that leaves (ncu, 16,384 entries x 2048 rows; 92% of the rounds of
// tiles are full there).  Six engines over 131,072 entries x 2048 rows: 18.1 ms
// at 1530 MHz, against 30.7 ms at 1400 MHz for the two-SM limb GEMM.  The sums
// make 2.25x the DB bytes (5.5 GB read per 16,384-entry launch), which is why
// few query rows keep the plain kernel.
//
// Structure: the two-SM limb GEMM's (cluster of two CTAs, 256 entries, M = 256;
// warp 0 TMA, warp 1 MMA on the leader), except that a tile runs nine
// accumulations of K/4 and has 16 epilogue warps.  They drain each product into
// per-thread sums: a "2" product is held in registers for the two that follow
// it, the six pair sums go to thread-local memory, and a tile's rows are formed
// and written between the next tile's products (after the last product instead:
// 22.3 ms; the sums folded earlier or the mask laid down first, to keep one set
// of sums: 19.7 and 20.7 ms against 19.4).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include "common.cuh"
#include "gemm_limb.h"
#include "quad_gemm.h"
#include "tc_sm100.cuh"
#include "tc_pair.cuh"
#include "launch_attr.cuh"

namespace irs {

namespace {

constexpr int kThreads = 576;               // TMA, MMA and 16 epilogue warps
constexpr int kMaxStages = 5;
constexpr int kMaxN = 256;
constexpr int kSkew = 2;                     // blocks that go to acc0 ahead of acc1 (see the MMA issuer)
constexpr int kABytes = 128 * kBK;           // one limb of a CTA's 128 entries
constexpr int kStageRoom = 225 * 1024;        // shared memory for the stages
constexpr int kSmemBytes = kStageRoom + 1024 /*align*/ + 256 /*barriers*/;
constexpr int kTmemCols = 512;               // acc0 at 0, acc1 at 256

// Stages of 128 K bytes that fit: three for 256 quads, four up to 192, five up
// to 96 (192 quads on four stages: 2.08 to 2.18 ms per 32,768 entries against
// 2.27 to 2.30 on three).  Prefetching the DB rows of a later block into L2
// made every size slower, by 1 to 9%: the kernel is bound by what the SMs draw
// from L2, not by the latency behind it.
constexpr int stage_count(int tile_n) {
  const int s = kStageRoom / (2 * (kABytes + tile_n / 2 * kBK));
  return s < kMaxStages ? s : kMaxStages;
}

// Products in order (outer, inner) = 22 2x 2y x2 xx xy y2 yx yy: the DB plane
// and the quarter of it that each reads.
__device__ __forceinline__ int product_plane(int j) { return j % 3 == 0 ? 2 : (j < 3 ? 1 : 0); }
__device__ __forceinline__ int product_quarter(int j) {
  return (int)((0x010232110ull >> (4 * (8 - j))) & 15ull);
}

struct Tile {
  int prob, m_tile, n_tile;
};

// The t-th tile in launch order: problems in sequence, the quad tiles of one
// block of entries together.
__device__ __forceinline__ bool tile_of(const QuadParams& P, int t, Tile& out) {
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

// The 32 rows of one slot for one entry, from the s-th slot of a thread's pair
// sums f.  Out of line: one copy of its ChaCha code, with the keystream added
// from registers.
__device__ __noinline__ void put_slot(const QuadProblem& pr, uint32_t m_local, uint32_t slot,
                                      const uint32_t (*f)[kMaxN / 8], int s) {
  if (m_local >= pr.m_len || slot >= pr.n_pad / 32) return;
  const uint32_t valid = pr.row_valid[slot];
  // word q of a form holds quads 2q and 2q + 1: rows i and i + 1, so the four
  // forms' words are four consecutive words of the slot
  uint32_t v[16];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t x2 = f[0][4 * s + q], y2 = f[1][4 * s + q];
    v[4 * q + 0] = add2(x2, f[2][4 * s + q]);  // rows 8q + 0, 1
    v[4 * q + 1] = add2(y2, f[3][4 * s + q]);  // rows 8q + 2, 3
    v[4 * q + 2] = add2(x2, f[4][4 * s + q]);  // rows 8q + 4, 5
    v[4 * q + 3] = add2(y2, f[5][4 * s + q]);  // rows 8q + 6, 7
  }
#pragma unroll
  for (int w = 0; w < 16; w++) {
    // rows without a query are zero, as the plain kernel's zero rows
    const uint32_t keep = ((valid >> (2 * w)) & 1u) * 0xFFFFu + ((valid >> (2 * w + 1)) & 1u) * 0xFFFF0000u;
    const uint32_t x = v[w] & keep;
    v[w] = (pr.mult == 1) ? x : (((x & 0xFFFFu) * pr.mult) & 0xFFFFu) | (((x >> 16) * pr.mult) << 16);
  }
  if (pr.mask_on) {
    const uint64_t blk = (((uint64_t)pr.m0 + m_local) * pr.n_pad + 32ull * slot) >> 5;
    const uint64_t ctr = counter_of(pr.batch_dev ? *pr.batch_dev : pr.batch, blk);
#pragma unroll 1
    for (int side = 0; side < 2; side++) {  // + ks_own - ks_prev
      uint32_t ks[16];
      chacha_block<12>(side ? pr.key_prev : pr.key_own, ctr, pr.nonce, ks);
#pragma unroll
      for (int w = 0; w < 16; w++) v[w] = side ? sub2(v[w], ks[w]) : add2(v[w], ks[w]);
    }
  }
  uint4* dst = reinterpret_cast<uint4*>(pr.out + (size_t)m_local * pr.n_pad + 32 * slot);
#pragma unroll
  for (int q = 0; q < 4; q++) dst[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    quad_gemm_kernel(const __grid_constant__ QuadParams P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int bn = P.tile_n, half_n = bn / 2;
  const int n_stages = P.stages;
  const int b_bytes = half_n * kBK;  // one limb of a CTA's half of the quads
  uint8_t* a_lo = smem;
  uint8_t* a_hi = a_lo + n_stages * kABytes;
  uint8_t* b_lo = a_hi + n_stages * kABytes;
  uint8_t* b_hi = b_lo + n_stages * b_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStageRoom);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kMaxStages;
  uint64_t* acc_full = bars + 2 * kMaxStages;  // [2]: acc0, acc1
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint64_t* done_bar = acc_full + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 5);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int cluster = blockIdx.x >> 1;
  const int n_clusters = gridDim.x >> 1;
  int* err = P.err;
  const uint64_t lim = P.wait_timeout_ns, lim2 = 2 * P.wait_timeout_ns;

  if (P.run.n && !cluster_reads(P.run, tmem_slot)) return;
  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 32);  // 16 epilogue warps in each CTA
    }
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)kTmemCols));
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
      const uint32_t tx = (uint32_t)(2 * 2 * (kABytes + half_n * kBK));  // both CTAs, both limbs
      for (int k = 0; ok; k++) {
        const int t = tile_index(k, cluster, n_clusters);
        if (k * n_clusters >= P.total_tiles) break;
        Tile tl;
        if (t >= P.total_tiles || !tile_of(P, t, tl)) continue;
        const QuadProblem& pr = P.prob[tl.prob];
        const int ya = (int)pr.m0 + tl.m_tile * kBM2 + (int)rank * 128;
        const int quads = (int)pr.n_pad / 4;
        const int k_iters = ((int)pr.quarter + kBK - 1) / kBK;
        for (int j = 0; ok && j < kQuadProducts; j++) {
          const int plane = product_plane(j);
          const int x0 = product_quarter(j) * (int)pr.quarter;
          const int yb = j * quads + tl.n_tile * bn + (int)rank * half_n;
          for (int ki = 0; ki < k_iters; ki++) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1u, err, kErrTimeoutEmpty, lim2)) { ok = false; break; }
            if (leader) mbar_expect_tx(&full_bar[stage], tx);
            const uint32_t fb = map_to_rank(&full_bar[stage], 0);
            tma_load_2d_pair(a_lo + stage * kABytes, &pr.tm_a_lo[plane], fb, x0 + ki * kBK, ya);
            tma_load_2d_pair(a_hi + stage * kABytes, &pr.tm_a_hi[plane], fb, x0 + ki * kBK, ya);
            tma_load_2d_pair(b_lo + stage * b_bytes, &pr.tm_b_lo, fb, ki * kBK, yb);
            tma_load_2d_pair(b_hi + stage * b_bytes, &pr.tm_b_hi, fb, ki * kBK, yb);
            issued |= 1u << stage;
            issued_phase = (issued_phase & ~(1u << stage)) | phase << stage;
            if (++stage == n_stages) { stage = 0; phase ^= 1u; }
          }
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
      const uint32_t idesc = idesc_u8_m256(bn);
      for (int k = 0; ok; k++) {
        const int t = tile_index(k, cluster, n_clusters);
        if (k * n_clusters >= P.total_tiles) break;
        Tile tl;
        if (t >= P.total_tiles || !tile_of(P, t, tl)) continue;
        const QuadProblem& pr = P.prob[tl.prob];
        const int k_iters = ((int)pr.quarter + kBK - 1) / kBK;
        // 32-byte steps of the last block (the bytes past the quarter belong
        // to the next one)
        const int last_steps = ((int)pr.quarter - (k_iters - 1) * kBK) / 32;
        // The products of block ki, in stage st, into acc0 (which = 0) or acc1.
        auto issue = [&](int ki, int st, int which) {
          const uint64_t dal = smem_desc(a_lo + st * kABytes);
          const uint64_t dah = smem_desc(a_hi + st * kABytes);
          const uint64_t dbl = smem_desc(b_lo + st * b_bytes);
          const uint64_t dbh = smem_desc(b_hi + st * b_bytes);
          const int steps = ki == k_iters - 1 ? last_steps : kBK / 32;
#pragma unroll
          for (int kk = 0; kk < kBK / 32; kk++) {
            if (kk < steps) {
              const uint32_t acc = (ki > 0 || kk > 0) ? 1u : 0u;
              const uint64_t o = (uint64_t)(2 * kk);
              if (which == 0) {
                mma_u8_pair(tmem, dal + o, dbl + o, idesc, acc);
              } else {
                mma_u8_pair(tmem + kMaxN, dal + o, dbh + o, idesc, acc);
                mma_u8_pair(tmem + kMaxN, dah + o, dbl + o, idesc, 1u);
              }
            }
          }
          if (which) mma_commit_pair(&empty_bar[st]);
        };
        // Waits for the next stage and moves on; the stage, or -1.
        auto next_stage = [&] {
          const int st = stage;
          if (!mbar_wait(&full_bar[st], phase, err, kErrTimeoutFull, lim)) return -1;
          if (++stage == n_stages) { stage = 0; phase ^= 1u; }
          tc_fence_after();
          return st;
        };
        for (int j = 0; ok && j < kQuadProducts; j++) {
          // The first and the last kSkew blocks go into acc0 before any of them
          // goes into acc1, so the epilogue drains acc0 of this product during
          // the last acc1 blocks, and acc1 during the next product's first acc0
          // blocks: neither side waits for a whole drain.
          int ki = 0, st[kSkew];
#pragma unroll
          for (int i = 0; i < kSkew; i++, ki++) {
            st[i] = ok ? next_stage() : -1;
            ok = st[i] >= 0;
            if (ok && i == 0) ok = mbar_wait(&acc_empty[0], acc_phase ^ 1u, err, kErrTimeoutAccEmpty, lim2);
            if (!ok) continue;
            tc_fence_after();
            issue(ki, st[i], 0);
          }
          ok = ok && mbar_wait(&acc_empty[1], acc_phase ^ 1u, err, kErrTimeoutAccEmpty, lim2);
          if (!ok) break;
          acc_phase ^= 1u;
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < kSkew; i++) issue(i, st[i], 1);
          for (; ki < k_iters - kSkew; ki++) {
            const int s = next_stage();
            ok = s >= 0;
            if (!ok) break;
            issue(ki, s, 0);
            issue(ki, s, 1);
          }
#pragma unroll
          for (int i = 0; i < kSkew; i++) {
            st[i] = ok ? next_stage() : -1;
            ok = st[i] >= 0;
            if (ok) issue(ki + i, st[i], 0);
          }
          if (!ok) break;
          mma_commit_pair(&acc_full[0]);
#pragma unroll
          for (int i = 0; i < kSkew; i++) issue(ki + i, st[i], 1);
          mma_commit_pair(&acc_full[1]);
        }
      }
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(done_bar))
                   : "memory");
      mbar_wait_drain(done_bar, 0, err, lim2);
    }
  } else {
    // ---------------- Epilogue (warps 2..17, both CTAs) ----------------
    const int quad = warp & 3;             // TMEM lanes 32*quad .. 32*quad+31
    const int part = (warp - 2) >> 2;      // column quarter of the tile
    const int row = quad * 32 + lane;
    const int cols = bn / 4, slots = cols / 8;  // this thread's quads, and the slots they make up
    const uint32_t acc_empty_leader[2] = {map_to_rank(&acc_empty[0], 0), map_to_rank(&acc_empty[1], 0)};
    const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * cols);
    uint32_t acc_phase = 0;
    bool ok = true;
    // 2+x and 2+y of the three outer forms, of the tile that drains and of the
    // one whose rows go out (thread-local memory)
    uint32_t sums[2][6][kMaxN / 8];
    int cur = 0;

    // Waits for the next product, hands its words (two quads each) to
    // use(index, word), and releases each accumulator as it is read.
    auto drain = [&](auto use) {
      uint32_t w[kMaxN / 8];
#pragma unroll
      for (int a = 0; a < 2; a++) {
        if (!mbar_wait(&acc_full[a], acc_phase, err, kErrTimeoutAccFull, lim2)) return false;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < kMaxN / 64; c++) {
          if (c * 16 < cols) {
            uint32_t r[16];
            tmem_ld16(tbase + (uint32_t)(a * kMaxN + c * 16), r);
            tmem_wait_ld16(r);
#pragma unroll
            for (int i = 0; i < 8; i++) {
              if (a == 0) w[8 * c + i] = __byte_perm(r[2 * i], r[2 * i + 1], 0x5410);
              else use(8 * c + i, add2(w[8 * c + i], ((r[2 * i] & 0xFFu) << 8) | (r[2 * i + 1] << 24)));
            }
          } else if (a == 0) {
#pragma unroll
            for (int i = 0; i < 8; i++) w[8 * c + i] = 0;
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_leader[a]);
      }
      acc_phase ^= 1u;
      return true;
    };

    // The last tile's rows go out a slot at a time between this tile's products:
    // the keystream of a tile (the bulk of the epilogue's instructions) takes
    // longer than one product.
    int prob = -1;  // -1: none
    uint32_t m_local = 0, slot0 = 0;
    auto put = [&](int s) {
      if (prob >= 0 && s < slots) put_slot(P.prob[prob], m_local, slot0 + (uint32_t)s, sums[cur ^ 1], s);
    };
    for (int k = 0; ok; k++) {
      const int t = tile_index(k, cluster, n_clusters);
      if (k * n_clusters >= P.total_tiles) break;
      Tile tl;
      if (t >= P.total_tiles || !tile_of(P, t, tl)) continue;
#pragma unroll 1
      for (int outer = 0; ok && outer < 3; outer++) {
        uint32_t two[kMaxN / 8] = {};
        put(3 * outer);
        ok = drain([&](int i, uint32_t v) { two[i] = v; });
#pragma unroll 1
        for (int inner = 0; ok && inner < 2; inner++) {
          put(3 * outer + 1 + inner);
          ok = drain([&](int i, uint32_t v) { sums[cur][2 * outer + inner][i] = add2(two[i], v); });
        }
      }
      if (!ok) break;
      prob = tl.prob;
      m_local = (uint32_t)(tl.m_tile * kBM2 + (int)rank * 128 + row);
      slot0 = (uint32_t)(tl.n_tile * bn + part * cols) / 8;
      cur ^= 1;
    }
    if (ok)
#pragma unroll 1
      for (int s = 0; s < slots; s++) put(s);
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while its peer may still touch its memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemCols));
  }
}

}  // namespace

// Both sides by the rounds of their tiles (last_done) and measured cycles of a
// 128-byte K step (gemm_limb.h has the plain ones; the one-SM 256-row tile
// takes 2700): 1840 for 160 quads, 2070 for 192, 2530 for 256, and 1500 for the
// drain of a product's accumulators.  Both kernels have to stream their DB
// planes.  Over 2,500 launches of 1 to 6 engines x 576 to 2,304 rows x 1,024 to
// 46,000 entries the choice is more than 5% off the better of the two in 75,
// against 245 when the steps were taken for their MMAs' time (two engines, 1,088
// rows x 1,975 entries: 290 us on the quad GEMM, 148 on 128-row tiles).
int quad_width_for(const uint32_t* K, int n_prob, uint32_t m_len, uint32_t n_pad, int block_n, bool pair, int n_sms) {
  constexpr double kDrain = 1500, kHbmBytesPerCycle = 3500;
  uint32_t tiles[kMaxGemmProblems];
  double cost[kMaxGemmProblems], bytes = 0;
  const uint32_t bm = pair ? (uint32_t)kBM2 : (uint32_t)kBM, wide = pair ? 256u : (uint32_t)block_n;
  const double step = pair ? plain_pair_step(n_pad) : block_n == 256 ? 2700 : kOneSmStep;
  for (int i = 0; i < n_prob; i++) {
    bytes += 2.0 * K[i] * m_len;
    tiles[i] = (m_len + bm - 1) / bm * ((n_pad + wide - 1) / wide);
    cost[i] = K[i] / 128 * step + 1000;
  }
  const double plain = std::max(last_done(tiles, cost, n_prob, pair ? n_sms / 2 : n_sms), bytes / kHbmBytesPerCycle);
  int best = -1;
  double least = 0.97 * plain;
  for (int w = 0; w < kQuadWidths; w++) {
    const int bn = quad_tile_n(n_pad, w);
    for (int i = 0; i < n_prob; i++) {
      tiles[i] = (m_len + kBM2 - 1) / kBM2 * ((n_pad / 4 + bn - 1) / (uint32_t)bn);
      cost[i] = kQuadProducts * (K[i] / 512.0 * std::max(690 + 7.2 * bn, kOneSmStep) + kDrain);
    }
    // (narrow tiles read more of the DB side per product: in launches of several
    // rounds 128 quads take a tenth more than their step in one says)
    const double c = std::max((w ? 1.1 : 1.0) * last_done(tiles, cost, n_prob, n_sms / 2),
                              2.25 * bytes / kHbmBytesPerCycle);
    if (c < least) {
      least = c;
      best = w;
    }
  }
  return best;
}

cudaError_t launch_quad_gemm(QuadParams& P, int n_sms, cudaStream_t stream) {
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = smem_limit_once(quad_gemm_kernel, kSmemBytes, attr_done);
  if (e != cudaSuccess) return e;
  if (P.wait_timeout_ns == 0) P.wait_timeout_ns = kGemmWaitTimeoutNs;
  P.stages = stage_count(P.tile_n);
  P.total_tiles = 0;
  for (int i = 0; i < P.n_prob; i++) {
    QuadProblem& pr = P.prob[i];
    pr.tiles_m = (pr.m_len + kBM2 - 1) / kBM2;
    pr.tiles_n = (pr.n_pad / 4 + (uint32_t)P.tile_n - 1) / (uint32_t)P.tile_n;
    P.total_tiles += (int)(pr.tiles_m * pr.tiles_n);
  }
  const int clusters = P.total_tiles < n_sms / 2 ? P.total_tiles : n_sms / 2;
  if (clusters <= 0) return cudaSuccess;
  quad_gemm_kernel<<<2 * clusters, kThreads, kSmemBytes, stream>>>(P);
  return cudaGetLastError();
}

}  // namespace irs
