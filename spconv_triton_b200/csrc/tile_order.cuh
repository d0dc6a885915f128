// Row order of the gather-GEMM (tile_order.cu) and the key and bucket of a row, which the kernel that
// writes the neighbour tables makes on its way.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace spc {

// Rows that one CTA sorts exactly.
constexpr int kTileOrderPiece = 8192;
// Sets of at most three of 32 offsets: 1 + 32 + 496 + 4960.
constexpr int kTileBuckets = 5489;

// Words of scratch of one order: the rows of every bucket, then how many of them have been dealt.
constexpr int kTileOrderWords = 2 * ((kTileBuckets + 63) / 64 * 64);

inline bool tile_order_needs_buckets(int64_t n) { return n > kTileOrderPiece; }

// The order the gather-GEMM wants is not the numeric order of the mask words but one in which the
// 128 rows of a tile share as many kernel offsets as possible.  Two cheap changes to the mask word
// get most of what a data-dependent order would: the offsets far from the kernel's centre (the
// corners of the window, the rarest in surface-like data) become the most significant bits, so that
// rows are grouped by their rare offsets first, and the key is Gray-decoded, so that neighbouring
// keys (hence neighbouring tiles) differ in few offsets.  On the VoxelNet-style backbone: 6 - 9 % fewer
// (tile, offset) stages on the submanifold levels, 2 - 16 % on the strided ones.
__host__ __device__ __forceinline__ uint32_t gray_decode(uint32_t key) {
  key ^= key >> 1;
  key ^= key >> 2;
  key ^= key >> 4;
  key ^= key >> 8;
  key ^= key >> 16;
  return key;
}
__host__ __device__ __forceinline__ uint32_t gray_encode(uint32_t key) { return key ^ (key >> 1); }

// Number of the set of the three highest bits of `word`, in the order of the Gray-decoded words: ascending
// in the highest bit, descending in the second (the decoded word is ones from the first down to the second,
// so a lower second bit is a larger key, and none the largest), ascending in the third.
// u(m, t) = subsets of m bits with at most t of them.
__device__ __forceinline__ int bucket_of(uint32_t word) {
  if (word == 0) return 0;
  const int a = 31 - __clz(word);
  word ^= 1u << a;
  const int upto3 = 1 + a + a * (a - 1) / 2 + a * (a - 1) * (a - 2) / 6;  // sets below bit a, up to three of them
  const int upto2 = 1 + a + a * (a - 1) / 2;                              // sets below bit a, up to two of them
  int inner = 0;
  if (word != 0) {
    const int b = 31 - __clz(word);
    word ^= 1u << b;
    const int c = 32 - __clz(word);  // one above the third bit, 0 without one
    inner = 1 + b + b * (b - 1) / 2 + (b - c);  // sets below bit b, then descending in the third bit
  }
  return upto3 + (upto2 - 1 - inner);
}

// Ascending order (as above) of `n` rows by key; kv <= 32 offsets make the keys.  `counts` (kTileOrderWords words, the
// rows per bucket made by the caller, the rest zero) and `pairs` (n entries) are used only where
// tile_order_needs_buckets(n); every word of `counts` is zero again afterwards, so that the next order of the same
// scratch can be counted into it.
int tile_order(const uint32_t* keys, int64_t n, int kv, uint32_t* counts, uint2* pairs, int32_t* order, cudaStream_t st);

}  // namespace spc
