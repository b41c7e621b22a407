// Launch interface of the data-preparation kernels (internal to the library).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace irs {

// One 32-row query slot: rows 0..n_rot-1 hold rotations rot_lo..rot_lo+n_rot-1
// (indices into all_rotations(), 15 = centre) of base query `src`.
struct QuerySlot {
  uint32_t src;
  uint32_t rot_lo;
  uint32_t n_rot;
  uint32_t query;  // output query index (bitmap row) the slot reports to
};

// Query forms of the rotation-structured GEMM (quad_gemm.cu) beside the planes.
struct QuadForms {
  uint8_t* lo;      // [9][n_pad/4][K/4], NULL: none
  uint8_t* hi;
  uint32_t* valid;  // [n_pad/32] rows of each slot that hold a query row
  uint32_t* flag;   // set to the padded rows the forms are for, 0 without forms (NULL: left alone)
};

struct SynthOut {
  uint8_t* code_lo[3];
  uint8_t* code_hi[3];
  uint8_t* mask_lo[3];
  uint8_t* mask_hi[3];
};

// n = rows x K coefficients; planes in quarter order (prep.cu)
cudaError_t launch_split_limbs(const uint16_t* in, uint32_t K, uint8_t* lo, uint8_t* hi, size_t n,
                               cudaStream_t stream);
// n rows of K i8 limbs to a plane; in == out where i8_plane_in_place(K)
bool i8_plane_in_place(size_t K);
cudaError_t launch_i8_plane(const uint8_t* in, uint32_t K, uint8_t* out, size_t n, cudaStream_t stream);
cudaError_t launch_derive_sums(const uint8_t* lo, const uint8_t* hi, uint32_t K, size_t n, uint8_t* outer_lo,
                               uint8_t* outer_hi, uint8_t* inner_lo, uint8_t* inner_hi, cudaStream_t stream);
// Whether the forms of queries of K coefficients can be expanded (K up to 21,600).
bool forms_fit(size_t K);
// Query planes of n_pad rows, and the query forms where quads.lo is set.
cudaError_t launch_expand_slots(const uint16_t* base, uint32_t K, const QuerySlot* slots, uint32_t n_slots,
                                uint32_t n_pad, uint8_t* lo, uint8_t* hi, const QuadForms& quads, cudaStream_t stream);
cudaError_t launch_expand_rows(const uint16_t* base, uint32_t K, const uint32_t* row_desc, uint32_t n_rows,
                               uint32_t n_pad, uint8_t* lo, uint8_t* hi, const QuadForms& quads, cudaStream_t stream);
cudaError_t launch_gather_rows(const uint8_t* src_lo, const uint8_t* src_hi, const uint32_t* ids, uint32_t n,
                               uint32_t K, uint8_t* dst_lo, uint8_t* dst_hi, cudaStream_t stream);
// K = 0: the words in sequence, else a limb plane of rows of K
cudaError_t launch_fill_random(void* p, size_t bytes, uint64_t seed, uint32_t K, cudaStream_t stream);
cudaError_t launch_synth_db(uint64_t seed, uint32_t first, uint32_t count, const SynthOut& out, cudaStream_t stream);

}  // namespace irs
