// Data-preparation kernels: u16 share records to u8 limb planes, query
// rotation expansion into 32-row slots, the i8 (byte - 128) storage limbs, and
// the seeded synthetic share database used by the benchmark workloads.
//
// Limb split: the reference stores limb_i = byte_i - 128 as i8 for cuBLAS
// (iris-mpc-gpu/src/dot/share_db.rs:45-59,620-655); the tcgen05 GEMM takes the
// unsigned bytes directly, so a stored i8 limb converts with x ^ 0x80.
// Rotations: row r of a query slot is all_rotations()[r] of the query share,
// i.e. every 800-coefficient row rotated left by 4*(15 - r) coefficients
// (iris-mpc-common/src/galois_engine.rs:42-52,197-206).
//
// Limb planes, of records and of query rows alike, hold a row's K coefficients
// as four quarters: each group of 32 consecutive coefficients (8 columns)
// gives its q-th 8 to quarter q, so quarter 2o + n holds the columns with bit 2
// (value 4) = o and bit 1 (value 2) = n, which is how the rotation-structured
// GEMM (quad_gemm.cu) splits them.  A dot product does not depend on the order.
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include "common.cuh"
#include "launch_attr.cuh"
#include "prep.h"

namespace irs {

namespace {

// Position in a plane row of the octet (8 coefficients) o of the record order.
__device__ __forceinline__ uint32_t plane_octet(uint32_t o, uint32_t K) { return (o & 3u) * (K / 32) + (o >> 2); }

// The same for a block of 4 coefficients.
__device__ __forceinline__ uint32_t plane_block(uint32_t b, uint32_t K) {
  return 2 * plane_octet(b >> 1, K) + (b & 1u);
}

// The low and the high bytes of four u16.
__device__ __forceinline__ uint32_t low_bytes(uint2 v) { return __byte_perm(v.x, v.y, 0x6420); }
__device__ __forceinline__ uint32_t high_bytes(uint2 v) { return __byte_perm(v.x, v.y, 0x7531); }

// One thread per octet of `n8` (rows of K coefficients).
__global__ void split_limbs_kernel(const uint16_t* __restrict__ in, uint32_t K, uint8_t* __restrict__ lo,
                                   uint8_t* __restrict__ hi, size_t n8) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  const uint4 v = reinterpret_cast<const uint4*>(in)[i];
  const uint2 a = make_uint2(v.x, v.y), b = make_uint2(v.z, v.w);
  const uint32_t per = K / 8;
  const size_t d = i / per * per + plane_octet((uint32_t)(i % per), K);
  reinterpret_cast<uint2*>(lo)[d] = make_uint2(low_bytes(a), low_bytes(b));
  reinterpret_cast<uint2*>(hi)[d] = make_uint2(high_bytes(a), high_bytes(b));
}

// Stored i8 limbs (byte - 128) in record order to a plane, one block per row.
// With `in_place` (in == out) the row passes through shared memory, so that
// records are written without scratch memory however full the device is.
__global__ void i8_plane_kernel(const uint8_t* in, uint32_t K, uint8_t* out, bool in_place) {
  extern __shared__ uint2 record[];
  const uint32_t per = K / 8;
  const uint2* src = reinterpret_cast<const uint2*>(in) + (size_t)blockIdx.x * per;
  uint2* dst = reinterpret_cast<uint2*>(out) + (size_t)blockIdx.x * per;
  if (in_place) {
    for (uint32_t o = threadIdx.x; o < per; o += blockDim.x) record[o] = src[o];
    __syncthreads();
    src = record;
  }
  for (uint32_t o = threadIdx.x; o < per; o += blockDim.x) {
    const uint2 v = src[o];
    dst[plane_octet(o, K)] = make_uint2(v.x ^ 0x80808080u, v.y ^ 0x80808080u);
  }
}

constexpr int kI8RowMost = 227 * 1024;  // a row of i8 limbs in shared memory

// Bytewise sums of two u16 vectors given as limb words: (al, ah) + (bl, bh).
__device__ __forceinline__ void add_limbs(uint32_t al, uint32_t ah, uint32_t bl, uint32_t bh, uint32_t& sl,
                                          uint32_t& sh) {
  sl = __vadd4(al, bl);
  const uint32_t carry = __vcmpltu4(sl, al) & 0x01010101u;
  sh = __vadd4(__vadd4(ah, bh), carry);
}
__device__ __forceinline__ void add_limbs(const uint4& al, const uint4& ah, const uint4& bl, const uint4& bh, uint4& sl,
                                          uint4& sh) {
  add_limbs(al.x, ah.x, bl.x, bh.x, sl.x, sh.x);
  add_limbs(al.y, ah.y, bl.y, bh.y, sl.y, sh.y);
  add_limbs(al.z, ah.z, bl.z, bh.z, sl.z, sh.z);
  add_limbs(al.w, ah.w, bl.w, bh.w, sl.w, sh.w);
}

// The sums of a record's quarters that the rotation-structured GEMM reads:
// outer = (q0 + q2, q1 + q3), inner = (all four, q0 + q1, q2 + q3).  One
// thread per 16 coefficients of a quarter; bound by HBM (2 bytes read and 2.5
// written per coefficient).
__global__ void derive_sums_kernel(const uint8_t* __restrict__ lo, const uint8_t* __restrict__ hi, uint32_t K, size_t n,
                                   uint8_t* __restrict__ outer_lo, uint8_t* __restrict__ outer_hi,
                                   uint8_t* __restrict__ inner_lo, uint8_t* __restrict__ inner_hi) {
  const uint32_t per = K / 64, Q = K / 4;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * per) return;
  const size_t row = i / per;
  const uint32_t x = (uint32_t)(i % per) * 16;
  uint4 l[4], h[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    l[q] = *reinterpret_cast<const uint4*>(lo + row * K + q * Q + x);
    h[q] = *reinterpret_cast<const uint4*>(hi + row * K + q * Q + x);
  }
  auto put = [&](uint8_t* pl, uint8_t* ph, size_t at, const uint4& sl, const uint4& sh) {
    *reinterpret_cast<uint4*>(pl + at) = sl;
    *reinterpret_cast<uint4*>(ph + at) = sh;
  };
  uint4 s0l, s0h, s1l, s1h, tl, th;
  add_limbs(l[0], h[0], l[2], h[2], s0l, s0h);
  add_limbs(l[1], h[1], l[3], h[3], s1l, s1h);
  put(outer_lo, outer_hi, row * 2 * Q + x, s0l, s0h);
  put(outer_lo, outer_hi, row * 2 * Q + Q + x, s1l, s1h);
  add_limbs(s0l, s0h, s1l, s1h, tl, th);
  put(inner_lo, inner_hi, row * 3 * Q + x, tl, th);
  add_limbs(l[0], h[0], l[1], h[1], tl, th);
  put(inner_lo, inner_hi, row * 3 * Q + Q + x, tl, th);
  add_limbs(l[2], h[2], l[3], h[3], tl, th);
  put(inner_lo, inner_hi, row * 3 * Q + 2 * Q + x, tl, th);
}

// The query source of a row: base query, mirror bit, rotation index into
// all_rotations() (15 = centre).
struct RowSource {
  uint32_t src;
  bool mirror, live;
  int rot;
};

// Row sources of a slot list: slot s row r holds rotation rot_lo[s] + r of
// query src[s] for r < n_rot[s]; other rows are zero.
struct SlotRows {
  const QuerySlot* slots;
  uint32_t n_slots;
  __device__ RowSource operator()(uint32_t row) const {
    const uint32_t s = row / kSlotRows, r = row % kSlotRows;
    if (s >= n_slots || r >= slots[s].n_rot) return {0u, false, false, 0};
    return {slots[s].src, false, true, (int)(slots[s].rot_lo + r)};
  }
};

// Row sources of a row table: desc[r] = (src << 8) | mirror << 7 | rot puts
// rotation `rot` (0..30) of base query `src` in row r, of its mirrored form
// when the mirror bit is set; 0xFFFFFFFF leaves the row zero.  Lets a batch
// pack queries with different rotation counts densely (no 32-row slot per
// query).
struct TableRows {
  const uint32_t* desc;
  uint32_t n_rows;
  __device__ RowSource operator()(uint32_t row) const {
    const uint32_t d = row < n_rows ? desc[row] : 0xFFFFFFFFu;
    if (d == 0xFFFFFFFFu) return {0u, false, false, 0};
    return {d >> 8, (d & 0x80u) != 0, true, (int)(d & 0x7Fu)};
  }
};

// Column `col` (any integer above -400) of 800-coefficient row `row800` of the
// row source's query, rotation not applied.
//
// Mirror (mirrored_code / mirrored_mask of the query share,
// iris-mpc-common/src/galois_engine.rs:218-225,520-543): 4-coefficient
// column c of each 800-coefficient row moves to 99 - c (c < 100) or 299 - c
// (c >= 100), and a code share's imaginary half (rows 8..15) is negated.
// The column map is its own inverse.
__device__ __forceinline__ uint2 query_column(const uint16_t* __restrict__ base, uint32_t K, const RowSource& q,
                                              uint32_t row800, int col) {
  uint32_t c = (uint32_t)(col + 400) % 200u;
  if (q.mirror) c = c < 100 ? 99 - c : 299 - c;
  uint2 v = *reinterpret_cast<const uint2*>(base + (size_t)q.src * K + (size_t)row800 * kRowLen + (size_t)c * 4);
  if (q.mirror && row800 >= 8) v = make_uint2(sub2(0u, v.x), sub2(0u, v.y));  // only code shares reach it
  return v;
}

__device__ __forceinline__ void put_octet(uint8_t* lo, uint8_t* hi, size_t at, uint2 a, uint2 b) {
  reinterpret_cast<uint2*>(lo)[at] = make_uint2(low_bytes(a), low_bytes(b));
  reinterpret_cast<uint2*>(hi)[at] = make_uint2(high_bytes(a), high_bytes(b));
}

// The query planes of n_pad rows and, when `quads.lo` is set, the query forms
// of the rotation-structured GEMM beside them: one block per row (the first
// n_pad) or quad.
//
// Planes: a rotated row's column c reads base column c + 15 - rot (mod 200).
//
// Forms (quad_gemm.cu): planes [9 products][n_pad / 4 quads][K / 4].  Quad s of
// a slot is rows i, i + 2, i + 4, i + 6 with i = 16 s2 + 8 s1 + s0 (the bits of
// s); its live rows are rotations of one query that keep their distance (the
// caller checked), so row i stands for rotation `rot` even where it is not live
// itself.  With f(k) the query at column offset c - rot shifted by 2k columns
// (column c of quarter 0), the forms are the outer and inner differences x:
// f(+D) - f, y: f(-D) - f at D = 4 and D = 2, "2": f itself.  Quads without a
// live row are zero.
//
// Bound by the strided half of the transfer: planes read the query in order and
// write 64-byte runs of each quarter (reading with a stride to write in order
// was a third slower), forms read it from shared memory.  64 queries of a code,
// planes and forms (82 MB written, cold): 32 us, against 46 us with a thread per
// octet of the whole grid and every division it takes.
template <class Rows>
__global__ void expand_kernel(const uint16_t* __restrict__ base, uint32_t K, Rows rows, uint32_t n_pad,
                              uint8_t* __restrict__ lo, uint8_t* __restrict__ hi, QuadForms quads) {
  const uint32_t per_quarter = K / 32;
  if (blockIdx.x < n_pad) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && quads.flag) *quads.flag = quads.lo ? n_pad : 0u;
    const uint32_t row = blockIdx.x;
    const RowSource src = rows(row);
    for (uint32_t o = threadIdx.x; o < 4 * per_quarter; o += blockDim.x) {
      uint2 a = make_uint2(0u, 0u), b = a;
      if (src.live) {
        const int col = (int)(o % 100) * 2 + 15 - src.rot;
        a = query_column(base, K, src, o / 100, col);
        b = query_column(base, K, src, o / 100, col + 1);
      }
      put_octet(lo, hi, (size_t)row * 4 * per_quarter + plane_octet(o, K), a, b);
    }
    return;
  }
  const uint32_t n_quads = n_pad / 4, p = blockIdx.x - n_pad;
  if (threadIdx.x < 32 && (p & 7u) == 0) {  // the rows of this slot that hold a query row
    const uint32_t bits = __ballot_sync(0xFFFFFFFFu, rows((p >> 3) * kSlotRows + threadIdx.x).live);
    if (threadIdx.x == 0) quads.valid[p >> 3] = bits;
  }
  const uint32_t row0 = (p >> 3) * kSlotRows + ((p >> 2) & 1u) * 16 + ((p >> 1) & 1u) * 8 + (p & 1u);
  RowSource src{0u, false, false, 0};
#pragma unroll
  for (int m = 3; m >= 0; m--) {
    const RowSource r = rows(row0 + 2 * m);
    if (r.live) src = {r.src, r.mirror, true, r.rot - 2 * m};
  }
  // The query, rotated by `rot` columns, in shared memory: column c of a row at
  // c + c / 8, so that threads eight columns apart read different banks.
  extern __shared__ uint2 query[];
  for (uint32_t i = threadIdx.x; src.live && i < K / 4; i += blockDim.x) {
    const uint32_t row800 = i / 200, c = i % 200;
    query[row800 * 225 + c + c / 8] = query_column(base, K, src, row800, (int)c + 15 - src.rot);
  }
  __syncthreads();
  for (uint32_t g = threadIdx.x; g < per_quarter; g += blockDim.x) {
    uint2 f[7][2];  // f(k - 3), the octet's two columns
#pragma unroll
    for (int k = 0; k < 7; k++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const uint32_t col = ((g % 25) * 8 + (uint32_t)(c + 2 * (k - 3) + 200)) % 200;
        f[k][c] = src.live ? query[g / 25 * 225 + col + col / 8] : make_uint2(0u, 0u);
      }
#pragma unroll
    for (int j = 0; j < 9; j++) {
      // terms of product j (outer, inner) = 22 2x 2y x2 xx xy y2 yx yy
      const int o = j / 3 == 0 ? 0 : (j / 3 == 1 ? 2 : -2), n = j % 3 == 0 ? 0 : (j % 3 == 1 ? 1 : -1);
      auto form = [&](auto at) {  // at(k) = f(k)
        uint32_t v = at(0);
        if (n) v = sub2(at(n), v);
        if (o) v = sub2(n ? sub2(at(o + n), at(o)) : at(o), v);
        return v;
      };
      uint2 w[2];
#pragma unroll
      for (int c = 0; c < 2; c++)
        w[c] = make_uint2(form([&](int k) { return f[k + 3][c].x; }), form([&](int k) { return f[k + 3][c].y; }));
      put_octet(quads.lo, quads.hi, ((size_t)j * n_quads + p) * per_quarter + g, w[0], w[1]);
    }
  }
}

// Copies DB rows ids[k] of (src_lo, src_hi) into rows k of (dst_lo, dst_hi),
// 16 bytes per thread (prefetch_subset, iris-mpc-gpu/src/dot/share_db.rs:344-407,
// done device-to-device because the DB is resident).
__global__ void gather_rows_kernel(const uint8_t* __restrict__ src_lo, const uint8_t* __restrict__ src_hi,
                                   const uint32_t* __restrict__ ids, uint32_t n, uint32_t K, uint8_t* __restrict__ dst_lo,
                                   uint8_t* __restrict__ dst_hi) {
  const uint32_t per_row = K / 16;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)n * per_row) return;
  const uint32_t k = (uint32_t)(i / per_row), c = (uint32_t)(i % per_row);
  const size_t s = (size_t)ids[k] * K + (size_t)c * 16, d = (size_t)k * K + (size_t)c * 16;
  *reinterpret_cast<uint4*>(dst_lo + d) = *reinterpret_cast<const uint4*>(src_lo + s);
  *reinterpret_cast<uint4*>(dst_hi + d) = *reinterpret_cast<const uint4*>(src_hi + s);
}

// ---------------- synthetic share database ----------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t rng64(uint64_t seed, uint64_t ctr) {
  return mix64(seed + (ctr + 1) * 0x9E3779B97F4A7C15ull);
}
__device__ __forceinline__ int remap_new_to_old(int i) {
  const int b = i / 6400, w = i % 6400 / 3200, r1 = i % 3200 / 800, c = i % 800 / 4, r2 = i % 4;
  return 800 * (r2 * 4 + r1) + c * 4 + w * 2 + b;
}
__device__ __forceinline__ void gr4_mul(const uint32_t a[4], const uint32_t b[4], uint32_t o[4]) {
  const uint32_t d4 = a[1] * b[3] + a[2] * b[2] + a[3] * b[1];
  const uint32_t d5 = a[2] * b[3] + a[3] * b[2];
  const uint32_t d6 = a[3] * b[3];
  o[0] = a[0] * b[0] + d4;
  o[1] = a[0] * b[1] + a[1] * b[0] + d4 + d5;
  o[2] = a[0] * b[2] + a[1] * b[1] + a[2] * b[0] + d5 + d6;
  o[3] = a[0] * b[3] + a[1] * b[2] + a[2] * b[1] + a[3] * b[0] + d6;
}

// Seeded uniform bytes (splitmix64 of the 8-byte word index): random shares
// for benchmark buffers whose values do not matter, only their bit activity.
__global__ void fill_random_kernel(uint64_t* __restrict__ p, size_t n_words, uint64_t seed) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_words; i += (size_t)gridDim.x * blockDim.x)
    p[i] = rng64(seed, i);
}
// The same words, in record order, for a limb plane of `rows` rows of K: a thread
// takes four consecutive words, one for each quarter.
__global__ void fill_random_plane_kernel(uint64_t* __restrict__ p, size_t rows, uint64_t seed, uint32_t K) {
  const uint32_t quarter = K / 32;  // words
  const size_t n = rows * quarter;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const size_t r = n >> 32 ? t / quarter : (uint32_t)t / quarter;
    uint64_t* out = p + r * 4 * quarter + (t - r * quarter);
#pragma unroll
    for (int q = 0; q < 4; q++) out[q * quarter] = rng64(seed, 4 * t + q);
  }
}

// One CTA per entry.  Mirrors the synthetic generator and the degree-1 Shamir
// encoding the CPU oracle defines (iris bits from rng64, mask pairs kept with
// probability 0.9, share randomness r = rng64(share seed, block)).
__global__ void synth_db_kernel(uint64_t seed, uint32_t first, uint32_t count, SynthOut out) {
  __shared__ uint64_t code[200], mask[200];
  const uint32_t e = first + blockIdx.x;
  if (blockIdx.x >= count) return;
  const uint64_t s = mix64(seed ^ ((uint64_t)e * 0xD1B54A32D192ED03ull));
  for (int w = threadIdx.x; w < 200; w += blockDim.x) {
    code[w] = rng64(s, (uint64_t)w);
    uint64_t m = 0;
    for (int q = 0; q < 32; q++) {
      const int p = w * 32 + q;  // pair index
      const uint64_t r = rng64(s ^ 0x5bd1e995ull, (uint64_t)(p >> 1));
      const uint32_t v = (p & 1) ? (uint32_t)(r >> 32) : (uint32_t)r;
      if (v < 3865470566u) m |= 3ull << (2 * q);
    }
    mask[w] = m;
  }
  __syncthreads();
  const uint64_t share_seed = rng64(seed ^ 0x5EEDull, e);
  const uint32_t S[4][4] = {{1, 0, 0, 0}, {58082, 1, 0, 0}, {60579, 25194, 1, 0}, {17325, 51956, 57011, 1}};
  const uint32_t BP[3][4] = {{1, 0, 0, 0}, {0, 1, 0, 0}, {1, 1, 0, 0}};
  for (int blk = threadIdx.x; blk < 3200; blk += blockDim.x) {
    const int i = blk * 4;
    uint32_t vc[4], vm[4];
    for (int k = 0; k < 4; k++) {
      const int o = remap_new_to_old(i + k);
      const uint32_t mb = (uint32_t)((mask[o >> 6] >> (o & 63)) & 1);
      const uint32_t cb = (uint32_t)((code[o >> 6] >> (o & 63)) & 1);
      vc[k] = (mb - 2u * (cb & mb)) & 0xFFFFu;
      vm[k] = mb;
    }
    for (int which = 0; which < 2; which++) {
      if (which == 1 && i >= kMaskCodeLength) break;  // trimmed mask
      const uint32_t* v = which == 0 ? vc : vm;
      uint32_t sm[4];
      for (int r = 0; r < 4; r++) sm[r] = S[r][0] * v[0] + S[r][1] * v[1] + S[r][2] * v[2] + S[r][3] * v[3];
      const uint64_t rr = rng64(which == 0 ? share_seed : (share_seed ^ 0xabcdef12345ull), (uint64_t)blk);
      const uint32_t rv[4] = {(uint32_t)(rr & 0xFFFF), (uint32_t)((rr >> 16) & 0xFFFF), (uint32_t)((rr >> 32) & 0xFFFF),
                              (uint32_t)(rr >> 48)};
      for (int p = 0; p < 3; p++) {
        uint32_t t[4];
        gr4_mul(rv, BP[p], t);
        uint32_t lo = 0, hi = 0;
        for (int k = 0; k < 4; k++) {
          const uint32_t x = (sm[k] + t[k]) & 0xFFFFu;
          lo |= (x & 0xFFu) << (8 * k);
          hi |= (x >> 8) << (8 * k);
        }
        const size_t K = which == 0 ? (size_t)kIrisCodeLength : (size_t)kMaskCodeLength;
        uint8_t* plo = which == 0 ? out.code_lo[p] : out.mask_lo[p];
        uint8_t* phi = which == 0 ? out.code_hi[p] : out.mask_hi[p];
        const uint32_t at = plane_block((uint32_t)blk, (uint32_t)K);
        reinterpret_cast<uint32_t*>(plo + (size_t)e * K)[at] = lo;
        reinterpret_cast<uint32_t*>(phi + (size_t)e * K)[at] = hi;
      }
    }
  }
}

}  // namespace

cudaError_t launch_split_limbs(const uint16_t* in, uint32_t K, uint8_t* lo, uint8_t* hi, size_t n,
                               cudaStream_t stream) {
  if (n % 8) return cudaErrorInvalidValue;
  const size_t n8 = n / 8;
  if (!n8) return cudaSuccess;
  split_limbs_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, stream>>>(in, K, lo, hi, n8);
  return cudaGetLastError();
}

bool i8_plane_in_place(size_t K) { return K <= kI8RowMost; }

cudaError_t launch_i8_plane(const uint8_t* in, uint32_t K, uint8_t* out, size_t n, cudaStream_t stream) {
  if (!n) return cudaSuccess;
  const bool in_place = in == out;
  if (in_place && !i8_plane_in_place(K)) return cudaErrorInvalidValue;
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = smem_limit_once(i8_plane_kernel, kI8RowMost, attr_done);
  if (e != cudaSuccess) return e;
  i8_plane_kernel<<<(unsigned)n, 256, in_place ? K : 0, stream>>>(in, K, out, in_place);
  return cudaGetLastError();
}

cudaError_t launch_derive_sums(const uint8_t* lo, const uint8_t* hi, uint32_t K, size_t n, uint8_t* outer_lo,
                               uint8_t* outer_hi, uint8_t* inner_lo, uint8_t* inner_hi, cudaStream_t stream) {
  if (K % 64) return cudaErrorInvalidValue;
  const size_t total = n * (K / 64);
  if (!total) return cudaSuccess;
  derive_sums_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(lo, hi, K, n, outer_lo, outer_hi, inner_lo,
                                                                          inner_hi);
  return cudaGetLastError();
}

bool forms_fit(size_t K) { return K / kRowLen * 225 * sizeof(uint2) <= 48 * 1024; }

template <class Rows>
static cudaError_t launch_expand(const uint16_t* base, uint32_t K, Rows rows, uint32_t n_pad, uint8_t* lo, uint8_t* hi,
                                 const QuadForms& quads, cudaStream_t stream) {
  if (!n_pad) return cudaSuccess;
  const size_t smem = quads.lo ? (size_t)K / kRowLen * 225 * sizeof(uint2) : 0;  // 28,800 bytes for a code
  if (quads.lo && !forms_fit(K)) return cudaErrorInvalidValue;
  expand_kernel<<<n_pad + (quads.lo ? n_pad / 4 : 0), 256, smem, stream>>>(base, K, rows, n_pad, lo, hi, quads);
  return cudaGetLastError();
}

cudaError_t launch_expand_slots(const uint16_t* base, uint32_t K, const QuerySlot* slots, uint32_t n_slots,
                                uint32_t n_pad, uint8_t* lo, uint8_t* hi, const QuadForms& quads, cudaStream_t stream) {
  return launch_expand(base, K, SlotRows{slots, n_slots}, n_pad, lo, hi, quads, stream);
}

cudaError_t launch_expand_rows(const uint16_t* base, uint32_t K, const uint32_t* row_desc, uint32_t n_rows,
                               uint32_t n_pad, uint8_t* lo, uint8_t* hi, const QuadForms& quads, cudaStream_t stream) {
  return launch_expand(base, K, TableRows{row_desc, n_rows}, n_pad, lo, hi, quads, stream);
}

cudaError_t launch_gather_rows(const uint8_t* src_lo, const uint8_t* src_hi, const uint32_t* ids, uint32_t n,
                               uint32_t K, uint8_t* dst_lo, uint8_t* dst_hi, cudaStream_t stream) {
  const size_t total = (size_t)n * (K / 16);
  if (!total) return cudaSuccess;
  gather_rows_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(src_lo, src_hi, ids, n, K, dst_lo, dst_hi);
  return cudaGetLastError();
}

cudaError_t launch_fill_random(void* p, size_t bytes, uint64_t seed, uint32_t K, cudaStream_t stream) {
  const size_t n = bytes / 8, threads = K ? n / 4 : n;
  if (n) {
    const unsigned blocks = (unsigned)std::min<size_t>((threads + 255) / 256, 148 * 16);
    if (K) fill_random_plane_kernel<<<blocks, 256, 0, stream>>>(static_cast<uint64_t*>(p), n / (K / 8), seed, K);
    else fill_random_kernel<<<blocks, 256, 0, stream>>>(static_cast<uint64_t*>(p), n, seed);
  }
  return cudaGetLastError();
}

cudaError_t launch_synth_db(uint64_t seed, uint32_t first, uint32_t count, const SynthOut& out, cudaStream_t stream) {
  if (!count) return cudaSuccess;
  synth_db_kernel<<<count, 128, 0, stream>>>(seed, first, count, out);
  return cudaGetLastError();
}

}  // namespace irs
