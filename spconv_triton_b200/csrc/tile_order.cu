// Row order of the gather-GEMM: rows that share kernel offsets are brought into the same 128-row tile.
//
// The order only decides which rows share a tile, never a result, so it need not be a full sort of the
// 27-bit keys.  A library radix sort of (key, row) was 13 launches (seven of them memsets) and four
// passes of about 8 us each however few rows there were: 340 of 870 us of device time of a one-sample
// backbone pass.  Here the rows are
//   1. counted per bucket by the kernel that makes their keys (fill_kernel, rulebook.cu),
//   2. dealt to their buckets (deal_rows_kernel), and
//   3. sorted exactly inside consecutive pieces of 8192 rows, in shared memory (sort_piece_kernel).
// A bucket is the set of keys with the same three most significant offsets (bucket_of), numbered in key
// order, so the result is the exact sort except inside buckets longer than a piece: 0 - 3 % more
// (tile, offset) stages than the exact order of the tile key on every level of the backbone and UNet
// workloads (two offsets instead of three: up to 7 %; no buckets, only pieces: 100 - 500 %).
#include <cub/block/block_radix_sort.cuh>

#include "common.cuh"
#include "tile_order.cuh"

namespace spc {
namespace {

constexpr int kPieceThreads = 1024;
constexpr int kPieceItems = kTileOrderPiece / kPieceThreads;

// One CTA deals 8192 rows: counts them per bucket in shared memory, reserves that much of every bucket it
// meets with one atomic, and writes (key, row) to its places.  Rows of a bucket come in any order.
__global__ void __launch_bounds__(kPieceThreads)
deal_rows_kernel(const uint32_t* __restrict__ keys, long long n, const uint32_t* __restrict__ counts,
                 uint32_t* __restrict__ taken, uint2* __restrict__ pairs) {
  __shared__ uint32_t place[kTileBuckets];  // rows of this CTA in the bucket, then where they go
  __shared__ uint32_t warp_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int b = tid; b < kTileBuckets; b += kPieceThreads) place[b] = 0;
  __syncthreads();
  const long long first = blockIdx.x * static_cast<long long>(kTileOrderPiece);
  uint32_t key[kPieceItems];
  int bucket[kPieceItems];
  uint32_t rank[kPieceItems];
#pragma unroll
  for (int i = 0; i < kPieceItems; ++i) {
    const long long r = first + i * kPieceThreads + tid;
    key[i] = r < n ? keys[r] : 0u;
    bucket[i] = r < n ? bucket_of(gray_encode(key[i])) : -1;
  }
#pragma unroll
  for (int i = 0; i < kPieceItems; ++i) rank[i] = bucket[i] >= 0 ? atomicAdd(&place[bucket[i]], 1u) : 0u;
  // start of every bucket: exclusive sum of all rows' counts, six consecutive buckets a thread
  constexpr int kPer = (kTileBuckets + kPieceThreads - 1) / kPieceThreads;
  uint32_t mine[kPer], sum = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int b = tid * kPer + q;
    mine[q] = b < kTileBuckets ? __ldg(&counts[b]) : 0u;
    sum += mine[q];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();  // the counts in place[] are complete as well
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += warp_sum[w];
  uint32_t start = before + incl - sum;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int b = tid * kPer + q;
    if (b < kTileBuckets) {
      const uint32_t have = place[b];
      place[b] = have != 0 ? start + atomicAdd(&taken[b], have) : 0u;
    }
    start += mine[q];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kPieceItems; ++i) {
    if (bucket[i] < 0) continue;
    const long long at = static_cast<long long>(place[bucket[i]]) + rank[i];
    if (at < n) pairs[at] = make_uint2(key[i], static_cast<uint32_t>(first + i * kPieceThreads + tid));
  }
}

// order[piece] = the piece's rows in ascending key order.  `pairs` null: the rows are 0..n-1 with `keys`.
template <int ITEMS>
__global__ void __launch_bounds__(kPieceThreads)
sort_piece_kernel(const uint32_t* __restrict__ keys, const uint2* __restrict__ pairs, long long n, int key_bits,
                  int32_t* __restrict__ order) {
  using Sort = cub::BlockRadixSort<uint32_t, kPieceThreads, ITEMS, int32_t>;
  extern __shared__ __align__(16) unsigned char temp[];
  const long long first = blockIdx.x * static_cast<long long>(kPieceThreads * ITEMS);
  const long long left = n - first;
  uint32_t key[ITEMS];
  int32_t row[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int at = threadIdx.x * ITEMS + i;
    key[i] = 0xffffffffu;  // past the end: sorts behind every key and is not written
    row[i] = -1;
    if (at < left) {
      if (pairs != nullptr) {
        const uint2 p = pairs[first + at];
        key[i] = p.x;
        row[i] = static_cast<int32_t>(p.y);
      } else {
        key[i] = keys[at];
        row[i] = at;
      }
    }
  }
  Sort(*reinterpret_cast<typename Sort::TempStorage*>(temp)).SortBlockedToStriped(key, row, 0, key_bits);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int at = i * kPieceThreads + threadIdx.x;
    if (at < left) order[first + at] = row[i];
  }
}

template <int ITEMS>
int launch_sort(const uint32_t* keys, const uint2* pairs, int64_t n, int key_bits, int32_t* order, cudaStream_t st) {
  using Sort = cub::BlockRadixSort<uint32_t, kPieceThreads, ITEMS, int32_t>;
  static bool configured[kMaxDevices] = {false};
  constexpr int bytes = static_cast<int>(sizeof(typename Sort::TempStorage));
  SPC_CUDA_OK(ensure_dynamic_smem(sort_piece_kernel<ITEMS>, bytes, configured));
  const unsigned blocks = static_cast<unsigned>(ceil_div(n, kPieceThreads * ITEMS));
  sort_piece_kernel<ITEMS><<<blocks, kPieceThreads, bytes, st>>>(keys, pairs, n, key_bits, order);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace

int tile_order(const uint32_t* keys, int64_t n, int kv, const uint32_t* counts, uint32_t* taken, uint2* pairs,
               int32_t* order, cudaStream_t st) {
  // one more bit than the keys have, so that the filler of the last piece sorts behind them
  const int bits = kv < 32 ? kv + 1 : 32;
  if (!tile_order_needs_buckets(n)) {
    // one piece: exact, and no larger than it has to be (the fewer rows a thread holds, the sooner it is done)
    if (n <= kPieceThreads) return launch_sort<1>(keys, nullptr, n, bits, order, st);
    if (n <= 2 * kPieceThreads) return launch_sort<2>(keys, nullptr, n, bits, order, st);
    if (n <= 4 * kPieceThreads) return launch_sort<4>(keys, nullptr, n, bits, order, st);
    return launch_sort<kPieceItems>(keys, nullptr, n, bits, order, st);
  }
  const unsigned blocks = static_cast<unsigned>(ceil_div(n, kTileOrderPiece));
  deal_rows_kernel<<<blocks, kPieceThreads, 0, st>>>(keys, n, counts, taken, pairs);
  SPC_LAUNCH_OK();
  return launch_sort<kPieceItems>(keys, pairs, n, bits, order, st);
}

}  // namespace spc
