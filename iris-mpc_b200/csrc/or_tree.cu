// MPC OR tree over a shared bit vector (or_reduce_result / or_tree_on_gpu,
// iris-mpc-gpu/src/threshold_ring/protocol.rs:2363-2515): the three parties
// reduce all bits of a replicated-shared vector to one shared bit by AND gates
// on their own views (OR(x, y) = x ^ y ^ (x & y)), then open it.
//
// Tree shape (the reference's): at each level the first half of the words is
// combined with the second half, word i with word i + num, and an odd last
// word moves down; after the word tree, the 32 bits of the last word are
// collapsed with shifted copies of itself (16, 8, 4, 2, 1).
//
// Randomness of the AND gate of level L, index i: word 0 of the ChaCha12 block
// at counter (batch << 40) | (L << 34) | i of each party's stream, nonce
// domain 4; party p's mask is k_p ^ k_{p-1} (zero-sharing).  Word levels are
// 1.., the collapse steps 40..44.
//
// What bounds it: latency.  A gate is three ChaCha blocks and a few logic
// operations, and a launch per level spends its 5 us on the launch and on the
// three blocks one after another.  So a block here takes the whole subtree of
// one word several levels down: its threads draw the keystream of all the
// subtree's gates at once, one block each, and the levels themselves are then
// a few loads apart in shared memory.  32,770 words (2^20 elements): 2 launches
// instead of 17, and 93 us for
// the whole call with the comparison, against 177.
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include "or_tree.h"

namespace irs {

namespace {

constexpr int kMostLevels = 9;               // of one launch: 512 leaves
constexpr int kStageLevels = 7;              // of a launch that is not the last
constexpr int kMostLeaves = 1 << kMostLevels;
constexpr uint64_t kCollapseLevel = 40;

__device__ __forceinline__ void or_gate(uint32_t x[3], const uint32_t y[3], const uint32_t k[3]) {
  uint32_t z[3];
#pragma unroll
  for (int p = 0; p < 3; p++) {
    const int q = (p + 2) % 3;  // party p views (component p, component p-1)
    z[p] = (x[p] & y[p]) ^ (x[q] & y[p]) ^ (x[p] & y[q]) ^ (k[p] ^ k[q]);
  }
#pragma unroll
  for (int p = 0; p < 3; p++) x[p] = x[p] ^ y[p] ^ z[p];
}

// Words of a level below a level of n words.
__device__ __forceinline__ uint64_t halved(uint64_t n) { return (n >> 1) + (n & 1); }

// The word at position `pos` of level `level` (0 = this launch's input, n
// words) in the subtree of word `root` at level `levels`: the position's bits,
// highest first, choose between the two words i and i + num that make a word i.
// An odd level's last word has one source.  False where there is no such word.
__device__ __forceinline__ bool word_at(uint64_t n, int levels, int level, uint32_t pos, uint64_t root, uint64_t& idx) {
  uint64_t size[kMostLevels + 1];
  size[0] = n;
#pragma unroll
  for (int l = 0; l < kMostLevels; l++) size[l + 1] = halved(size[l]);
  idx = root;
  bool there = true;
#pragma unroll
  for (int l = kMostLevels - 1; l >= 0; l--) {
    if (l >= levels || l < level) continue;
    const uint64_t num = size[l] >> 1;
    const bool second = (pos >> (l - level)) & 1u;
    if (idx < num) idx += second ? num : 0;
    else { there = there && !second; idx = 2 * num; }
  }
  return there;
}

// Each block reduces the subtree of output word blockIdx.x over `levels`
// levels; with `last`, that is the whole tree, and the word collapses to one bit.
__global__ void or_subtree_kernel(const uint32_t* __restrict__ in, uint64_t in_stride, uint64_t n, int levels,
                                  uint32_t first_level, uint32_t* __restrict__ out, uint64_t out_stride, int last,
                                  const OrTreeParams P) {
  __shared__ uint32_t word[2][3][kMostLeaves];
  __shared__ uint32_t key[3][kMostLeaves + 8];
  const int leaves = 1 << levels;
  const uint64_t batch = P.batch_dev ? *P.batch_dev : P.batch;
  for (int t = threadIdx.x; t < leaves; t += blockDim.x) {
    uint64_t i;
    const bool there = word_at(n, levels, 0, (uint32_t)t, blockIdx.x, i);
#pragma unroll
    for (int p = 0; p < 3; p++) word[0][p][t] = there ? in[p * in_stride + i] : 0u;
  }
  // Gates: those of the first level (leaves / 2 of them), of the second, ...,
  // then the collapse steps; gate g's keystream word of stream s at key[s][g].
  const int gates = leaves - 1, all = gates + (last ? 5 : 0);
  for (int c = threadIdx.x; c < 3 * all; c += blockDim.x) {
    const int g = c / 3, s = c % 3;
    uint64_t gate = (kCollapseLevel + (uint64_t)(g - gates)) << 34;
    bool there = true;
    if (g < gates) {
      int l = 0, pos = g;
      for (; pos >= (leaves >> (l + 1)); l++) pos -= leaves >> (l + 1);
      uint64_t i;
      there = word_at(n, levels, l + 1, (uint32_t)pos, blockIdx.x, i);
      gate = ((uint64_t)(first_level + (uint32_t)l) << 34) | i;
    }
    if (there) {
      uint32_t blk[16];
      chacha_block<12>(P.key[s], counter_of(batch, gate), P.nonce, blk);
      key[s][g] = blk[0];
    }
  }
  __syncthreads();
  int cur = 0, first_gate = 0;
  for (int l = 0; l < levels; l++) {
    const int nodes = leaves >> (l + 1);
    for (int t = threadIdx.x; t < nodes; t += blockDim.x) {
      uint64_t i, num = n;
      for (int q = 0; q < l; q++) num = halved(num);
      num >>= 1;
      const bool there = word_at(n, levels, l + 1, (uint32_t)t, blockIdx.x, i);
      uint32_t x[3], y[3], k[3];
#pragma unroll
      for (int p = 0; p < 3; p++) {
        x[p] = word[cur][p][2 * t];
        y[p] = word[cur][p][2 * t + 1];
        k[p] = key[p][first_gate + t];
      }
      if (there && i < num) or_gate(x, y, k);
#pragma unroll
      for (int p = 0; p < 3; p++) word[cur ^ 1][p][t] = x[p];
    }
    __syncthreads();
    cur ^= 1;
    first_gate += nodes;
  }
  if (threadIdx.x) return;
  uint32_t x[3] = {word[cur][0][0], word[cur][1][0], word[cur][2][0]};
  if (!last) {
#pragma unroll
    for (int p = 0; p < 3; p++) out[p * out_stride + blockIdx.x] = x[p];
    return;
  }
  for (int j = 0; j < 5; j++) {
    const int s = 16 >> j;
    const uint32_t y[3] = {x[0] >> s, x[1] >> s, x[2] >> s};
    const uint32_t k[3] = {key[0][gates + j], key[1][gates + j], key[2][gates + j]};
    or_gate(x, y, k);
  }
  out[0] = x[0] & 1u;
  out[1] = x[1] & 1u;
  out[2] = x[2] & 1u;
  out[3] = (x[0] ^ x[1] ^ x[2]) & 1u;
  out[4] = (uint32_t)*P.err;
}

}  // namespace

cudaError_t launch_or_tree(const OrTreeParams& P, const uint32_t* comp, size_t n_words, uint32_t* scratch,
                           uint32_t* out5, cudaStream_t stream) {
  if (n_words == 0) return cudaErrorInvalidValue;
  const uint32_t* cur = comp;
  uint64_t cur_stride = n_words, num = n_words;
  uint32_t* bufs[2] = {scratch, scratch + 3 * n_words};
  int which = 0;
  uint32_t level = 1;
  while (true) {
    int levels = 0;
    uint64_t left = num;
    for (; left > 1 && levels < kMostLevels; levels++) left = (left >> 1) + (left & 1);
    const bool last = left == 1;
    if (!last) {
      left = num;
      for (levels = 0; levels < kStageLevels; levels++) left = (left >> 1) + (left & 1);
    }
    const unsigned threads = (unsigned)std::min(1024, std::max(32, 3 << levels));
    or_subtree_kernel<<<(unsigned)left, threads, 0, stream>>>(cur, cur_stride, num, levels, level,
                                                              last ? out5 : bufs[which], n_words, last, P);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || last) return e;
    cur = bufs[which];
    cur_stride = n_words;
    which ^= 1;
    num = left;
    level += (uint32_t)levels;
  }
}

}  // namespace irs
