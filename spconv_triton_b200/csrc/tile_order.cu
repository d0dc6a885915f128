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
#include "common.cuh"
#include "tile_order.cuh"

namespace spc {
namespace {

constexpr int kDealThreads = 512;
constexpr int kDealItems = 8;
constexpr int kPieceThreads = 1024;
constexpr int kPieceWarps = kPieceThreads / 32;
constexpr int kDigitBits = 9;
constexpr int kDigits = 1 << kDigitBits;

// One CTA deals 4096 rows: counts them per bucket in shared memory, reserves that much of every bucket it
// meets with one atomic, and writes (key, row) to its places.  Rows of a bucket come in any order.
__global__ void __launch_bounds__(kDealThreads)
deal_rows_kernel(const uint32_t* __restrict__ keys, long long n, const uint32_t* __restrict__ counts,
                 uint32_t* __restrict__ taken, uint2* __restrict__ pairs) {
  __shared__ uint32_t place[kTileBuckets];  // rows of this CTA in the bucket, then where they go
  __shared__ uint32_t warp_sum[kDealThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int b = tid; b < kTileBuckets; b += kDealThreads) place[b] = 0;
  __syncthreads();
  const long long first = blockIdx.x * static_cast<long long>(kDealThreads * kDealItems);
  uint32_t key[kDealItems];
  int bucket[kDealItems];
  uint32_t rank[kDealItems];
#pragma unroll
  for (int i = 0; i < kDealItems; ++i) {
    const long long r = first + i * kDealThreads + tid;
    key[i] = r < n ? keys[r] : 0u;
    bucket[i] = r < n ? bucket_of(gray_encode(key[i])) : -1;
  }
#pragma unroll
  for (int i = 0; i < kDealItems; ++i) rank[i] = bucket[i] >= 0 ? atomicAdd(&place[bucket[i]], 1u) : 0u;
  // start of every bucket: exclusive sum of all rows' counts, eleven consecutive buckets a thread
  constexpr int kPer = (kTileBuckets + kDealThreads - 1) / kDealThreads;
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
  uint32_t have[kPer], at_least[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) have[q] = tid * kPer + q < kTileBuckets ? place[tid * kPer + q] : 0u;
#pragma unroll
  for (int q = 0; q < kPer; ++q) at_least[q] = have[q] != 0 ? atomicAdd(&taken[tid * kPer + q], have[q]) : 0u;  // all in flight
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    if (have[q] != 0) place[tid * kPer + q] = start + at_least[q];
    start += mine[q];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kDealItems; ++i) {
    if (bucket[i] < 0) continue;
    const long long at = static_cast<long long>(place[bucket[i]]) + rank[i];
    if (at < n) pairs[at] = make_uint2(key[i], static_cast<uint32_t>(first + i * kDealThreads + tid));
  }
}

// order[piece] = the piece's rows in ascending key order.  `pairs` null: the rows are 0..n-1 with `keys`.
// A least-significant-digit radix sort in shared memory: nine bits a pass, so three passes for the 27
// offsets of a 3x3x3 kernel.  A warp ranks its rows 32 at a time (lanes with the same digit find each other
// with nine ballots, the first of them adds to the warp's count of that digit), then the counts of all warps
// become places by one block-wide sum in (digit, warp) order, which keeps the sort stable.
// `used` (may be null): the bucket counts that the rows have been dealt by, zeroed for the next order.
template <int ITEMS>
__global__ void __launch_bounds__(kPieceThreads)
sort_piece_kernel(const uint32_t* __restrict__ keys, const uint2* __restrict__ pairs, long long n, int key_bits,
                  int32_t* __restrict__ order, uint32_t* __restrict__ used) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint2* item = reinterpret_cast<uint2*>(smem);                                   // [kPieceThreads * ITEMS]
  uint16_t* count = reinterpret_cast<uint16_t*>(item + kPieceThreads * ITEMS);    // [kDigits][kPieceWarps]
  __shared__ uint32_t warp_sum[kPieceWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (used != nullptr)
    for (int i = blockIdx.x * kPieceThreads + tid; i < kTileOrderWords; i += gridDim.x * kPieceThreads) used[i] = 0u;
  const long long first = blockIdx.x * static_cast<long long>(kPieceThreads * ITEMS);
  const int left = static_cast<int>(n - first < kPieceThreads * ITEMS ? n - first : kPieceThreads * ITEMS);
  uint2 mine[ITEMS];
  const int at0 = warp * 32 * ITEMS + lane;  // a warp's rows are consecutive
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int at = at0 + i * 32;
    mine[i] = make_uint2(0u, 0u);
    if (at < left) mine[i] = pairs != nullptr ? pairs[first + at] : make_uint2(keys[at], static_cast<uint32_t>(at));
  }
  for (int bit = 0; bit < key_bits; bit += kDigitBits) {
    for (int i = tid; i < kDigits * kPieceWarps / 8; i += kPieceThreads)
      reinterpret_cast<uint4*>(count)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    uint32_t rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const bool live = at0 + i * 32 < left;
      const int digit = live ? static_cast<int>((mine[i].x >> bit) & (kDigits - 1)) : kDigits;
      unsigned same = __ballot_sync(0xffffffffu, live);
#pragma unroll
      for (int b = 0; b < kDigitBits; ++b) {
        const unsigned ones = __ballot_sync(0xffffffffu, (digit >> b) & 1);
        same &= (digit >> b) & 1 ? ones : ~ones;
      }
      uint32_t before = 0;
      if (live) before = count[digit * kPieceWarps + warp];
      __syncwarp();
      if (live && __ffs(same) - 1 == lane) count[digit * kPieceWarps + warp] = static_cast<uint16_t>(before + __popc(same));
      __syncwarp();
      rank[i] = before + __popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    // exclusive sum over the counts, sixteen consecutive ones a thread
    constexpr int kEach = kDigits * kPieceWarps / kPieceThreads;
    uint32_t sum = 0;
    uint16_t c[kEach];
    static_assert(kEach == 16, "two 16-byte words of counts a thread");
    reinterpret_cast<uint4*>(c)[0] = reinterpret_cast<const uint4*>(count)[2 * tid];
    reinterpret_cast<uint4*>(c)[1] = reinterpret_cast<const uint4*>(count)[2 * tid + 1];
#pragma unroll
    for (int q = 0; q < kEach; ++q) sum += c[q];
    uint32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    uint32_t total = warp_sum[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, total, off);
      if (lane >= off) total += t;
    }
    uint32_t start = __shfl_sync(0xffffffffu, total, warp > 0 ? warp - 1 : 0);
    start = (warp > 0 ? start : 0u) + incl - sum;
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
      const uint32_t v = c[q];
      c[q] = static_cast<uint16_t>(start);
      start += v;
    }
    reinterpret_cast<uint4*>(count)[2 * tid] = reinterpret_cast<const uint4*>(c)[0];
    reinterpret_cast<uint4*>(count)[2 * tid + 1] = reinterpret_cast<const uint4*>(c)[1];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (at0 + i * 32 < left)
        item[count[((mine[i].x >> bit) & (kDigits - 1)) * kPieceWarps + warp] + rank[i]] = mine[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (at0 + i * 32 < left) mine[i] = item[at0 + i * 32];
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (at0 + i * 32 < left) order[first + at0 + i * 32] = static_cast<int32_t>(mine[i].y);
}

template <int ITEMS>
int launch_sort(const uint32_t* keys, const uint2* pairs, int64_t n, int key_bits, int32_t* order, uint32_t* used, cudaStream_t st) {
  static bool configured[kMaxDevices] = {false};
  constexpr int bytes = kPieceThreads * ITEMS * static_cast<int>(sizeof(uint2)) + kDigits * kPieceWarps * 2;
  SPC_CUDA_OK(ensure_dynamic_smem(sort_piece_kernel<ITEMS>, bytes, configured));
  const unsigned blocks = static_cast<unsigned>(ceil_div(n, kPieceThreads * ITEMS));
  sort_piece_kernel<ITEMS><<<blocks, kPieceThreads, bytes, st>>>(keys, pairs, n, key_bits, order, used);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace

int tile_order(const uint32_t* keys, int64_t n, int kv, uint32_t* counts, uint2* pairs, int32_t* order, cudaStream_t st) {
  constexpr int kItems = kTileOrderPiece / kPieceThreads;
  if (!tile_order_needs_buckets(n)) {
    // one piece: exact, and no larger than it has to be (the fewer rows a thread holds, the sooner it is done)
    if (n <= kPieceThreads) return launch_sort<1>(keys, nullptr, n, kv, order, nullptr, st);
    if (n <= 2 * kPieceThreads) return launch_sort<2>(keys, nullptr, n, kv, order, nullptr, st);
    if (n <= 4 * kPieceThreads) return launch_sort<4>(keys, nullptr, n, kv, order, nullptr, st);
    return launch_sort<kItems>(keys, nullptr, n, kv, order, nullptr, st);
  }
  // pieces of 4096 rows where they still fit one wave of CTAs: the sort is as long as one piece takes
  const bool small = n <= static_cast<int64_t>(sm_count()) * kTileOrderPiece / 2;
  const unsigned blocks = static_cast<unsigned>(ceil_div(n, kDealThreads * kDealItems));
  deal_rows_kernel<<<blocks, kDealThreads, 0, st>>>(keys, n, counts, counts + kTileOrderWords / 2, pairs);
  SPC_LAUNCH_OK();
  return small ? launch_sort<kItems / 2>(keys, pairs, n, kv, order, counts, st) : launch_sort<kItems>(keys, pairs, n, kv, order, counts, st);
}

}  // namespace spc
