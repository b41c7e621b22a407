// Fused 3-party threshold comparison, open and rotation OR.
//
// One thread evaluates the whole Phase-2 protocol for one 32-element word of
// all three co-resident parties (circuit.cuh): the lift of the mask dot
// shares from Z_2^16 to Z_2^32, the bit injection of the two lift carries,
// mask*A - code*2^16 - 1, the 32-bit MSB adder, and the opening of the result.
// The per-gate "send to next party" of the reference (NCCL send/recv around
// every AND round, iris-mpc-gpu/src/threshold_ring/protocol.rs:894-1032) is the
// component store inside the thread, so the ~52 dependent rounds and ~7
// launches per round collapse into straight-line code, and HBM sees each input
// share exactly once.
//
// Modes:
//   flat   -- elements e = 0..n-1, word w = e/32 (Circuits API: results are
//             the per-party shares of the msb bit plus the opened bits);
//   bitmap -- dot shares laid out [entry][n_pad], each query iris owning a
//             32-row slot; a warp covers 32 consecutive entries of one slot,
//             the opened word OR-ed over the slot's valid rows is the match bit
//             (the rotation OR of openResults, dot/kernel.cu:54-116), written
//             with one ballot per warp, and matches are appended to a list.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include "circuit.cuh"
#include "threshold.h"
#include "threshold_emit.cuh"
#include "launch_attr.cuh"

namespace irs {

namespace {

constexpr int kThreshThreads = 128;
// Shared memory per thread of the keystream (WordRandShared): 18 prepared
// words-of-four and 48 keystream words.
constexpr int kRandSmemPerThread = 18 * 16 + 48 * 4;

template <class WR>
__device__ __forceinline__ void init_rand(WR& wr, const ThresholdParams& P, uint64_t word_id) {
#pragma unroll
  for (int s = 0; s < 3; s++) wr.key[s] = P.key[s];
  wr.nonce = P.nonce;
  wr.base = counter_of(P.batch_dev ? *P.batch_dev : P.batch, word_id * (uint64_t)kCircuitBlocksPerWord);
}

// This thread's keystream columns in the block's shared memory ([element][thread]).
template <int THREADS>
__device__ __forceinline__ void bind_rand(WordRandShared& wr) {
  extern __shared__ uint4 rand_smem[];
  wr.pre = rand_smem + threadIdx.x;
  wr.ks = reinterpret_cast<uint32_t*>(rand_smem + 18 * THREADS) + threadIdx.x;
  wr.nt = THREADS;
}

template <int STAGE>
__global__ void __launch_bounds__(kThreshThreads) threshold_flat_kernel(const ThresholdParams P) {
  const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= P.n_words) return;
  WordRandShared wr;
  bind_rand<kThreshThreads>(wr);
  init_rand(wr, P, P.word_base + w);
  const uint16_t* code[3] = {P.code[0] + 32 * w, P.code[1] + 32 * w, P.code[2] + 32 * w};
  const uint16_t* mask[3] = {P.mask[0] + 32 * w, P.mask[1] + 32 * w, P.mask[2] + 32 * w};
  Comp msb;
  const uint32_t r = threshold_word<STAGE>(code, mask, P.threshold_a, wr, msb);
  if (P.revealed) P.revealed[w] = r;
  if (P.res_comp) {
    P.res_comp[w] = msb.c0;
    P.res_comp[P.n_words + w] = msb.c1;
    P.res_comp[2 * P.n_words + w] = msb.c2;
  }
}

// The bitmap kernel indexes by global warp only, so its block size is free:
// THREADS x MIN_BLOCKS sets the resident warps per SM the registers are sized for.
template <int THREADS, int MIN_BLOCKS>
__global__ void __launch_bounds__(THREADS, MIN_BLOCKS) threshold_bitmap_kernel(const ThresholdParams P) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t gwarp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t n_groups = (P.n_entries + 31) / 32;
  const uint64_t total = (uint64_t)n_groups * P.n_slots;
  if (gwarp >= total) return;  // warp-uniform
  const uint32_t slot = (uint32_t)(gwarp % P.n_slots);
  const uint32_t group = (uint32_t)(gwarp / P.n_slots);
  const uint32_t m_local = group * 32 + lane;
  const bool valid = m_local < P.n_entries;
  const uint32_t m_read = valid ? m_local : (P.n_entries - 1);
  const uint64_t m_global = (uint64_t)P.m0 + m_local;

  WordRandShared wr;
  bind_rand<THREADS>(wr);
  init_rand(wr, P, ((uint64_t)P.m0 + m_read) * (uint64_t)(P.n_pad / 32) + slot);
  const size_t off = (size_t)m_read * P.n_pad + (size_t)slot * 32;
  uint32_t opened;
  {
    // The share pointers die here; the rare distance capture below rebuilds
    // them from `off`, which keeps 12 registers free through the circuit.
    const uint16_t* code[3] = {P.code[0] + off, P.code[1] + off, P.code[2] + off};
    const uint16_t* mask[3] = {P.mask[0] + off, P.mask[1] + off, P.mask[2] + off};
    Comp msb;
    opened = threshold_word<kStageFull>(code, mask, P.threshold_a, wr, msb);
  }
  const size_t bitmap_word = (size_t)((P.m0 + group * 32) / 32);
  // The capture rebuilds the share pointers from `off` (rare).
  emit_word(P, opened, valid, lane, slot, m_global, bitmap_word,
            [&](int p, int is_mask, int r) { return (is_mask ? P.mask[p] : P.code[p])[off + r]; });
}

// ---------------------------------------------------------------------------
// Few words: one thread per word leaves most of the GPU idle while each warp
// walks 20,000 instructions of straight-line code, once.  Here a block of eight
// warps takes one warp's 32 words and shares out what the protocol leaves
// independent, with the bit planes in shared memory ([plane][word], a warp's
// lanes side by side): the keystream blocks over all warps, the slicing, the
// lifted values and their transposes over the parties, the bit injection over
// the element pairs.  Only the two adders run on one warp, as loops.  The
// gates, their keystream words and the results are threshold_word's.
// ---------------------------------------------------------------------------
constexpr int kSplitThreads = 256;
constexpr int kSplitWarps = kSplitThreads / 32;
constexpr int kSplitKs = 3 * kCircuitBlocksPerWord * 16;           // keystream words, [(3 block + stream) 16 + j]
constexpr int kSplitRows = kSplitKs + 96 + 48 + 6;                 // + planes, lift corrections, carries
constexpr int kSplitSmem = kSplitRows * 32 * 4;                    // 68,352 bytes

struct SplitSmem {
  uint32_t* ks;     // this lane's columns, row stride 32
  uint32_t* plane;  // [3][16] mask planes, then [3][32] planes of the lifted value
  uint32_t* corr;   // [3][16]
  uint32_t* carry;  // c1 (3 components), c2
  // gate word j of block b, stream s
  __device__ uint32_t k(int b, int s, int j) const { return ks[((3 * b + s) * 16 + j) * 32]; }
  __device__ Comp gate(Comp x, Comp y, int b, int j) const { return cand(x, y, k(b, 0, j), k(b, 1, j), k(b, 2, j)); }
  __device__ Comp at(int stride, int i) const {
    return {plane[i * 32], plane[(stride + i) * 32], plane[(2 * stride + i) * 32]};
  }
};

// One ripple step of a 3-input adder whose inputs are the components of s
// (planes k and k + 1), its carry-save gate at word j of block b and its ripple
// gate at word j + 1.  Returns the step's carry-save bit.
__device__ __forceinline__ Comp ripple_step(const SplitSmem& m, Comp s, Comp s1, int b, int j, bool first,
                                            Comp& carry) {
  Comp c = m.gate({s.c0, 0u, s.c2}, {0u, s.c1, s.c2}, b, j);
  c.c2 ^= s.c2;
  if (first) carry = m.gate(s1, c, b, j + 1);
  else carry = cxor(carry, m.gate(cxor(s1, carry), cxor(c, carry), b, j + 1));
  return c;
}

// threshold_word of the word of lane `lane` by the whole block; the result is
// the first warp's.
template <int STAGE>
__device__ __forceinline__ uint32_t split_word(const ThresholdParams& P, const uint16_t* const code[3],
                                               const uint16_t* const mask[3], uint64_t base, Comp& msb) {
  extern __shared__ uint4 rand_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SplitSmem m;
  m.ks = reinterpret_cast<uint32_t*>(rand_smem) + lane;
  m.plane = m.ks + kSplitKs * 32;
  m.corr = m.plane + 96 * 32;
  m.carry = m.corr + 48 * 32;
  constexpr int kFirst = STAGE == kStageFull ? 0 : 2, kLast = STAGE == kStageFull ? 8 : 6;  // blocks that are drawn
  uint32_t wm[16], wc[16];  // party `warp`'s shares
  if (warp < 3) {
    load32(code[warp], wc);
    if (STAGE == kStageFull) {
      uint32_t M[16];
      load32(mask[warp], wm);
      slice16(wm, M);
#pragma unroll
      for (int k = 0; k < 16; k++) m.plane[(16 * warp + k) * 32] = M[k];
    }
  }
#pragma unroll 1
  for (int c = 3 * kFirst + warp; c < 3 * kLast; c += kSplitWarps) {
    uint32_t out[16];
    chacha_block<12>(P.key[c % 3], base + (uint64_t)(c / 3), P.nonce, out);
#pragma unroll
    for (int j = 0; j < 16; j++) m.ks[(16 * c + j) * 32] = out[j];
  }
  __syncthreads();
  if (STAGE == kStageFull) {
    if (warp == 0) {  // lift_carries
      Comp carry = {0, 0, 0}, s = m.at(16, 0);
#pragma unroll 3
      for (int k = 0; k < 15; k++) {
        const Comp s1 = m.at(16, k + 1);
        ripple_step(m, s, s1, k >> 3, 2 * (k & 7), k == 0, carry);
        s = s1;
      }
      Comp c = m.gate({s.c0, 0u, s.c2}, {0u, s.c1, s.c2}, 1, 14);
      c.c2 ^= s.c2;
      const Comp c2 = m.gate(c, carry, 1, 15), c1 = cxor(carry, c);
      m.carry[0] = c1.c0; m.carry[32] = c1.c1; m.carry[64] = c1.c2;
      m.carry[96] = c2.c0; m.carry[128] = c2.c1; m.carry[160] = c2.c2;
    }
    __syncthreads();
    uint32_t v[6];
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = unzip_bits(m.carry[32 * q]);
#pragma unroll 1
    for (int i = warp; i < 16; i += kSplitWarps) {
      uint32_t a[3], b[3];
      inject_pair((v[0] >> i) & 0x00010001u, (v[1] >> i) & 0x00010001u, (v[2] >> i) & 0x00010001u, m.k(6, 0, i),
                  m.k(6, 1, i), m.k(6, 2, i), a[0], a[1], a[2]);
      inject_pair((v[3] >> i) & 0x00010001u, (v[4] >> i) & 0x00010001u, (v[5] >> i) & 0x00010001u, m.k(7, 0, i),
                  m.k(7, 1, i), m.k(7, 2, i), b[0], b[1], b[2]);
#pragma unroll
      for (int p = 0; p < 3; p++) m.corr[(16 * p + i) * 32] = add2(a[p], (b[p] << 1) & 0xFFFEFFFEu);
    }
    __syncthreads();
  }
  if (warp < 3) {  // X_p of threshold_word, transposed
    uint32_t X[32];
    const uint32_t one = warp == 0 ? 1u : 0u;
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const uint32_t c = (wc[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
      if (STAGE == kStageFull) {
        const uint32_t mk = (wm[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
        const uint32_t cr = (m.corr[(16 * warp + (j >> 1)) * 32] >> (16 * (j & 1))) & 0xFFFFu;
        X[j] = mk * P.threshold_a - ((cr * P.threshold_a + c) << 16) - one;
      } else {
        X[j] = 0u - (c << 16) - one;
      }
    }
    transpose32(X);
#pragma unroll
    for (int k = 0; k < 32; k++) m.plane[(32 * warp + k) * 32] = X[k];
  }
  __syncthreads();
  if (warp) return 0;
  // msb_of_sum
  Comp carry = {0, 0, 0}, s = m.at(32, 0);
#pragma unroll 3
  for (int k = 0; k < 30; k++) {
    const Comp s1 = m.at(32, k + 1);
    ripple_step(m, s, s1, 2 + (k >> 3), 2 * (k & 7), k == 0, carry);
    s = s1;
  }
  Comp c = m.gate({s.c0, 0u, s.c2}, {0u, s.c1, s.c2}, 5, 12);
  c.c2 ^= s.c2;
  msb = cxor(cxor(carry, m.at(32, 31)), c);
  return msb.c0 ^ msb.c1 ^ msb.c2;
}

// The results of flat word w: the opened bits, the components, and the shares
// of each party (a = its own component, b = the previous party's).
__device__ __forceinline__ void put_flat(const ThresholdParams& P, uint64_t w, uint32_t opened, const Comp& msb) {
  if (P.revealed) P.revealed[w] = opened;
  if (P.res_comp) {
    P.res_comp[w] = msb.c0;
    P.res_comp[P.n_words + w] = msb.c1;
    P.res_comp[2 * P.n_words + w] = msb.c2;
  }
  const uint32_t c[3] = {msb.c0, msb.c1, msb.c2};
#pragma unroll
  for (int p = 0; p < 3; p++)
    if (P.res_a[p]) P.res_a[p][w] = c[p];
#pragma unroll
  for (int p = 0; p < 3; p++)
    if (P.res_b[p]) P.res_b[p][w] = c[(p + 2) % 3];
}

__device__ __forceinline__ uint64_t keystream_base(const ThresholdParams& P, uint64_t word_id) {
  return counter_of(P.batch_dev ? *P.batch_dev : P.batch, word_id * (uint64_t)kCircuitBlocksPerWord);
}

template <int STAGE>
__global__ void __launch_bounds__(kSplitThreads, 3) threshold_flat_split_kernel(const ThresholdParams P) {
  const uint64_t w = (uint64_t)blockIdx.x * 32 + (threadIdx.x & 31);
  const uint64_t rd = w < P.n_words ? w : P.n_words - 1;
  const uint16_t* code[3] = {P.code[0] + 32 * rd, P.code[1] + 32 * rd, P.code[2] + 32 * rd};
  const uint16_t* mask[3] = {P.mask[0] + 32 * rd, P.mask[1] + 32 * rd, P.mask[2] + 32 * rd};
  Comp msb;
  const uint32_t r = split_word<STAGE>(P, code, mask, keystream_base(P, P.word_base + rd), msb);
  if (threadIdx.x < 32 && w < P.n_words) put_flat(P, w, r, msb);
}

__global__ void __launch_bounds__(kSplitThreads, 3) threshold_bitmap_split_kernel(const ThresholdParams P) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t slot = blockIdx.x % P.n_slots, group = blockIdx.x / P.n_slots;
  const uint32_t m_local = group * 32 + lane;
  const bool valid = m_local < P.n_entries;
  const uint32_t m_read = valid ? m_local : (P.n_entries - 1);
  const size_t off = (size_t)m_read * P.n_pad + (size_t)slot * 32;
  const uint16_t* code[3] = {P.code[0] + off, P.code[1] + off, P.code[2] + off};
  const uint16_t* mask[3] = {P.mask[0] + off, P.mask[1] + off, P.mask[2] + off};
  Comp msb;
  const uint32_t opened = split_word<kStageFull>(
      P, code, mask, keystream_base(P, ((uint64_t)P.m0 + m_read) * (uint64_t)(P.n_pad / 32) + slot), msb);
  if (threadIdx.x >= 32) return;
  emit_word(P, opened, valid, lane, slot, (uint64_t)P.m0 + m_local, (size_t)((P.m0 + group * 32) / 32),
            [&](int p, int is_mask, int r) { return (is_mask ? P.mask[p] : P.code[p])[off + r]; });
}

__global__ void __launch_bounds__(kThreshThreads) lift_flat_kernel(const ThresholdParams P, uint16_t* corr) {
  const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= P.n_words) return;
  WordRand wr;
  init_rand(wr, P, P.word_base + w);
  const uint16_t* mask[3] = {P.mask[0] + 32 * w, P.mask[1] + 32 * w, P.mask[2] + 32 * w};
  uint16_t c1[3][32], c2[3][32];
  lift_word(mask, wr, c1, c2);
  const uint64_t n = P.n_words * 32;
#pragma unroll
  for (int p = 0; p < 3; p++) {
    uint16_t* o1 = corr + (size_t)(2 * p) * n + 32 * w;
    uint16_t* o2 = corr + (size_t)(2 * p + 1) * n + 32 * w;
#pragma unroll
    for (int j = 0; j < 32; j++) { o1[j] = c1[p][j]; o2[j] = c2[p][j]; }
  }
}

}  // namespace

constexpr int kRandSmem = kThreshThreads * kRandSmemPerThread;  // 61,440 bytes per block

template <class K>
static cudaError_t allow_rand_smem(K kernel, std::atomic<uint64_t>& done) {
  return smem_limit_once(kernel, kRandSmem, done);
}

// Most warps' worth of words (32 each) that run in the split kernels: two rounds
// of the three blocks that fit an SM, of a B200's 148.  Flat calls, split against one thread per
// word: 4,096 elements 10.5 / 25 us (cold), 454,656 18.5 / 23.5, 699,968 24.7 /
// 34.9, 1,048,576 34.0 / 34.4, 2,097,152 66 / 64, 4,194,304 123 / 104.
constexpr uint64_t kSplitMost = 2 * 3 * 148;

bool threshold_writes_shares(uint64_t n_words) { return (n_words + 31) / 32 <= kSplitMost; }

cudaError_t launch_threshold_flat(const ThresholdParams& P, int stage, cudaStream_t stream) {
  if (P.n_words == 0) return cudaSuccess;
  const uint64_t n_warps = (P.n_words + 31) / 32;
  if (n_warps <= kSplitMost) {
    static std::atomic<uint64_t> split_full{0}, split_msb{0};
    const cudaError_t e = stage == kStageFull
                              ? smem_limit_once(threshold_flat_split_kernel<kStageFull>, kSplitSmem, split_full)
                              : smem_limit_once(threshold_flat_split_kernel<kStageMsbOnly>, kSplitSmem, split_msb);
    if (e != cudaSuccess) return e;
    if (stage == kStageFull)
      threshold_flat_split_kernel<kStageFull><<<(unsigned)n_warps, kSplitThreads, kSplitSmem, stream>>>(P);
    else
      threshold_flat_split_kernel<kStageMsbOnly><<<(unsigned)n_warps, kSplitThreads, kSplitSmem, stream>>>(P);
    return cudaGetLastError();
  }
  static std::atomic<uint64_t> done_full{0}, done_msb{0};
  cudaError_t attr = allow_rand_smem(threshold_flat_kernel<kStageFull>, done_full);
  if (attr == cudaSuccess) attr = allow_rand_smem(threshold_flat_kernel<kStageMsbOnly>, done_msb);
  if (attr != cudaSuccess) return attr;
  const unsigned grid = (unsigned)((P.n_words + kThreshThreads - 1) / kThreshThreads);
  if (stage == kStageFull) threshold_flat_kernel<kStageFull><<<grid, kThreshThreads, kRandSmem, stream>>>(P);
  else threshold_flat_kernel<kStageMsbOnly><<<grid, kThreshThreads, kRandSmem, stream>>>(P);
  return cudaGetLastError();
}

cudaError_t launch_threshold_bitmap(const ThresholdParams& P, cudaStream_t stream) {
  if (P.n_entries == 0 || P.n_slots == 0) return cudaSuccess;
  const uint64_t warps = (uint64_t)((P.n_entries + 31) / 32) * P.n_slots;
  if (warps <= kSplitMost) {
    static std::atomic<uint64_t> split_bitmap{0};
    const cudaError_t e = smem_limit_once(threshold_bitmap_split_kernel, kSplitSmem, split_bitmap);
    if (e != cudaSuccess) return e;
    threshold_bitmap_split_kernel<<<(unsigned)warps, kSplitThreads, kSplitSmem, stream>>>(P);
    return cudaGetLastError();
  }
  // Resident warps per SM the kernel's registers are sized for: 12 (3 per
  // SM sub-partition, 168-register cap) measured 2-6% faster than 8 on
  // 512K-entry batches.  Other
  // counts give the same register cap as one of these two, since each
  // sub-partition holds a quarter of the register file.
  // IRS_THRESHOLD_WARPS_PER_SM=8 selects the other variant for tuning runs.
  static const bool eight = [] {
    const char* e = getenv("IRS_THRESHOLD_WARPS_PER_SM");
    return e && atoi(e) == 8;
  }();
  static std::atomic<uint64_t> done_8{0}, done_12{0};
  cudaError_t attr = eight ? allow_rand_smem(threshold_bitmap_kernel<kThreshThreads, 2>, done_8)
                           : allow_rand_smem(threshold_bitmap_kernel<kThreshThreads, 3>, done_12);
  if (attr != cudaSuccess) return attr;
  const unsigned grid = (unsigned)((warps * 32 + kThreshThreads - 1) / kThreshThreads);
  if (eight) threshold_bitmap_kernel<kThreshThreads, 2><<<grid, kThreshThreads, kRandSmem, stream>>>(P);
  else threshold_bitmap_kernel<kThreshThreads, 3><<<grid, kThreshThreads, kRandSmem, stream>>>(P);
  return cudaGetLastError();
}

cudaError_t launch_lift_flat(const ThresholdParams& P, uint16_t* corr, cudaStream_t stream) {
  if (P.n_words == 0) return cudaSuccess;
  const unsigned grid = (unsigned)((P.n_words + kThreshThreads - 1) / kThreshThreads);
  lift_flat_kernel<<<grid, kThreshThreads, 0, stream>>>(P, corr);
  return cudaGetLastError();
}

}  // namespace irs
