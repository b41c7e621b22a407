// Launch interface of the rotation-structured limb GEMM (internal to the
// library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "common.cuh"
#include "gemm_limb.h"

namespace irs {

constexpr int kQuadProducts = 9;

// One dot-product problem over quads of query rows: the entries
// [m0, m0 + m_len) of a party's DB against n_pad / 4 quads.
struct alignas(64) QuadProblem {
  // DB planes, low and high limbs: [0] the records [rows][K], [1] the outer
  // sums [rows][K/2], [2] the inner sums [rows][3K/4] (derive_sums_kernel)
  CUtensorMap tm_a_lo[3];
  CUtensorMap tm_a_hi[3];
  CUtensorMap tm_b_lo;  // query forms [9][n_pad/4][K/4] (expand_kernel)
  CUtensorMap tm_b_hi;
  uint16_t* out;        // [m_len][n_pad]
  const uint32_t* row_valid;  // [n_pad/32] rows of each slot that hold a query row
  uint32_t m0;
  uint32_t m_len;
  uint32_t n_pad;
  uint32_t quarter;     // K / 4
  uint32_t mult;        // 1 for codes, 2 for trimmed masks
  uint32_t mask_on;     // add ks_own - ks_prev
  ChaChaKey key_own;
  ChaChaKey key_prev;
  uint64_t nonce;
  uint64_t batch;
  const uint64_t* batch_dev;
  uint32_t tiles_m;     // filled by launch_quad_gemm
  uint32_t tiles_n;
};

struct QuadParams {
  QuadProblem prob[kMaxGemmProblems];
  QuadFlags run;  // the launch does nothing unless they are all set
  int n_prob;
  int total_tiles;
  int tile_n;  // quads per tile: a multiple of 32, at most 256
  int stages;  // filled by launch_quad_gemm
  int* err;
  uint64_t wait_timeout_ns;  // 0 = kGemmWaitTimeoutNs
};

// Quads per tile for n_pad query rows, in multiples of 32 (the N step of the
// two-SM i8 instruction): width 0 is equal tiles of at most 256 quads, widths
// 1 and 2 at most 128 and 64, for launches with too few tiles for the GPU.
constexpr int kQuadWidths = 3;
inline int quad_tile_n(uint32_t n_pad, int width) {
  const uint32_t quads = n_pad / 4, most = 256u >> width;
  const uint32_t tiles = (quads + most - 1) / most;
  return (int)(((quads + tiles - 1) / tiles + 31) / 32 * 32);
}

// The tile width with which a launch over m_len entries and n_pad rows of
// engines with code lengths K[0..n_prob) is expected to take least, or -1 where
// the plain limb GEMM (block_n, pair) is expected to be as fast.
int quad_width_for(const uint32_t* K, int n_prob, uint32_t m_len, uint32_t n_pad, int block_n, bool pair, int n_sms);

// Tensor map of a [rows][k] u8 plane read in boxes of 128 bytes x box_rows
// (k a multiple of 16; a box over the end of a row reads zeros there).
int make_tmap_plane(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows);

cudaError_t launch_quad_gemm(QuadParams& P, int n_sms, cudaStream_t stream);

}  // namespace irs
