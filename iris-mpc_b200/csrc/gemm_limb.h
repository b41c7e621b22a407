// Launch interface of the tcgen05 limb GEMM (internal to the library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "common.cuh"

namespace irs {

// One dot-product problem: a party's DB limb planes against its query limb
// planes, for the entries [m0, m0 + m_len).
struct alignas(64) GemmProblem {
  CUtensorMap tm_a_lo;  // DB low bytes   [rows][K]
  CUtensorMap tm_a_hi;  // DB high bytes  [rows][K]
  CUtensorMap tm_b_lo;  // query low bytes  [n_pad][K]
  CUtensorMap tm_b_hi;  // query high bytes [n_pad][K]
  uint16_t* out;        // [m_len][n_pad]
  uint32_t m0;
  uint32_t m_len;
  uint32_t n_pad;
  uint32_t k_iters;     // K / 128
  uint32_t mult;        // 1 for codes, 2 for trimmed masks
  uint32_t mask_on;     // add ks_own - ks_prev
  ChaChaKey key_own;
  ChaChaKey key_prev;
  uint64_t nonce;
  uint64_t batch;
  const uint64_t* batch_dev;  // when set, the batch id is read from device memory
  uint32_t tiles_m;     // filled by launch_limb_gemm
  uint32_t tiles_n;
};

constexpr int kMaxGemmProblems = 6;
// Device words that hold the padded row count while an engine's uploaded rows
// are quads of rotations, else 0.  A captured launch holds both GEMMs, since
// later uploads decide which one a replay needs: the quad GEMM runs when all
// words are the row count it was captured for, the plain one when not.
struct QuadFlags {
  const uint32_t* word[kMaxGemmProblems];
  int n;  // 0: not captured, no check
  uint32_t rows;
#ifdef __CUDACC__
  __device__ __forceinline__ bool all_set() const {
    bool all = true;
    for (int i = 0; i < n; i++) all = all && *word[i] == rows;
    return all;
  }
#endif
};

constexpr uint64_t kGemmWaitTimeoutNs = 2000000000ull;  // default limit of a bounded wait: 2 s

struct GemmParams {
  GemmProblem prob[kMaxGemmProblems];
  QuadFlags skip;  // the launch does nothing when they are all set
  int n_prob;
  int total_tiles;
  int* err;
  // L2 eviction priority of the TMA loads: bit 0 = query planes evict_last
  // (re-read by every DB tile), bit 1 = DB planes evict_first (streamed).
  uint32_t l2_hint;
  // Limit of the MMA's wait for a TMA stage; the other waits get twice this.
  // 0 = kGemmWaitTimeoutNs.
  uint64_t wait_timeout_ns;
  // Test hook: CTA 0 issues no TMA loads, so its MMA's first stage wait runs
  // out (kErrTimeoutFull) and the kernel returns with the error word set.
  uint32_t test_stall;
  // Serpentine K order: a CTA walks K backwards on its odd tile iterations,
  // so the query K blocks the previous wave of CTAs loaded last are the first
  // this wave needs.  Integer accumulation: the result does not depend on it.
  uint32_t serpentine;
  // two-SM kernel (filled by launch_limb_gemm): the widest tile's query rows,
  // how many tiles of a problem have them, pipeline stages
  int pair_n;
  int pair_wider;
  int pair_stages;
};

// Builds a 2-D u8 tensor map (inner dim K, outer dim rows) with 128x`box_rows`
// boxes and 128-byte swizzle.  Returns 0 on success.
int make_tmap_u8(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows);

// Tile width along the query rows for n_pad of them (256, 128 or 64; 0 if n_pad
// is no multiple of 64).
int gemm_block_n_for(uint32_t n_pad);

// Whether the two-SM (cta_group::2) kernel can run n_pad query rows where it is
// asked for; its query tensor maps then use boxes of gemm_pair_n / 2 rows.
bool gemm_pair_applies(bool pair, uint32_t n_pad);
// Its widest tile for n_pad query rows (a multiple of 64, at most 256).
int gemm_pair_n(uint32_t n_pad);

// Cycles until the last of `units` SMs (or pairs) is done, tiles of the
// problems dealt out in order.
double last_done(const uint32_t* tiles, const double* cost, int n_prob, int units);

// Cycles of a 128-byte K step, measured over launches of a few rounds (1.9 to 2
// GHz): of a 128-row tile on one SM, and of the two-SM kernel's tiles over n_pad
// rows (1300 for 128 rows, 1740 for 192, 2190 for 256).
constexpr double kOneSmStep = 1340;
inline double plain_pair_step(uint32_t n_pad) { return 400 + 7.0 * gemm_pair_n(n_pad); }

// The width of the tiles, one to an SM, that a launch of few rounds over m_len
// entries and n_pad rows of engines with code lengths K[0..n_prob) runs rather
// than SM pairs or 256-row tiles: 128 or 64 rows, or 0 for no such launch.  Up to
// a few rounds of tiles, what counts is how full the last round is; all in one
// round, one-SM tiles take less, and 64-row ones least where they fit it and the
// K loop of the 128-row ones would not be shared (3 engines, 1,984 rows x 89
// entries: 62.5 / 70 us).  Over 3,000 launches of 1 to 6 engines x 64 to 2,304
// rows x 32 to 23,000 entries, the choice between 128-row tiles and pairs is more
// than 5% off the better one in 21, against 400 for a limit on the tiles (one
// engine, 12,800 coefficients: 1,408 rows x 1,461 entries, 132 tiles of 128, 67 /
// 105 us; 1,536 x 1,900, 180 tiles, 121 / 105).
int few_rounds_tile(const uint32_t* K, int n_prob, uint32_t m_len, uint32_t n_pad, int n_sms);

cudaError_t launch_limb_gemm(GemmParams& P, int block_n, bool pair, int n_sms, cudaStream_t stream);

}  // namespace irs
