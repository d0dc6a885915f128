// Point cloud voxelisation (points -> voxels) on the GPU, first come first served.
//
// Semantics follow PointToVoxel.generate_voxel_with_id,
// spconv_triton/pytorch/utils.py:72-163, which states them with torch sorts:
//   * a point's voxel is floor((p - cmin) / vsize) per axis, in the dtype of the
//     points (fp32 here: one IEEE subtraction, one IEEE division, floor);
//   * voxels are numbered in the order of their first point (utils.py:107-114);
//     only the first max_voxels voxels are kept, points of the others get id -1;
//   * inside a voxel the points keep their arrival order; the first max_points
//     are stored, the others keep the voxel id but are not stored (utils.py:129-144);
//   * num_per_voxel is the true count clamped at max_points (utils.py:119-120);
//   * voxel coordinates are written reversed (z, y, x) (utils.py:122-128);
//   * empty_mean fills the unused slots of a voxel with the mean of its stored
//     points (utils.py:146-153).
// The result is deterministic and equal to the reference's, bit for bit.
//
// How it is computed here (no sort):
//   1. quantize_insert: key per point; a hash table keeps, per key, the lowest
//      point index (one packed 64-bit atomicMin: key << 32 | index) and a count
//      that also gives the point a place among its voxel's points, in any order;
//   2. a point is "first" when the table returns its own index; the number of
//      first points before it IS its voxel's number.  count_first adds them up per
//      block and hands the total to the host, number_voxels numbers them and
//      reserves room for each voxel's points in one list;
//   3. place: every point goes to its place in its voxel's stretch of the list;
//   4. rank: a point's slot is the number of lower indices in that stretch (a few
//      points; voxels of more than 256 points take a radix sort instead);
//   5. emit: the voxel buffer and the caller's copy of it are written row by row,
//      points and zeros alike, so that nothing is cleared or copied first.
// HBM-bound; bytes per point: 4*F read + 4*F written (stored points) + 8 (voxel id)
// + the rows of the voxel buffer.  1.2 M points: the sort (three passes, a scan, nine
// memsets) and the three copies were 110 of 215 us of device time.
#include <cub/cub.cuh>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "rulebook_internal.cuh"

namespace spc {
namespace {

constexpr int kVoxThreads = 256;
constexpr int kVoxMaxDim = 4;
constexpr unsigned long long kVoxEmpty = ~0ull;
constexpr uint32_t kNoKey = 0xffffffffu;

struct VoxGeo {
  int ndim;
  float cmin[kVoxMaxDim];
  float vsize[kVoxMaxDim];
  int grid[kVoxMaxDim];  // x, y, z order, as given
};

__device__ __forceinline__ uint32_t vox_mix(uint32_t h) {
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}

inline unsigned vox_blocks(int64_t n) { return static_cast<unsigned>(ceil_div(std::max<int64_t>(n, 1), kVoxThreads)); }

// One slot of the hash table, 16 bytes so that whatever a point asks of its voxel is one sector.  While points
// are entered: key << 32 | lowest point index (all ones: free) and their count.  Once numbered: the voxel
// (-1: beyond the cap), its stretch of the list, the count.
struct alignas(16) VoxSlot {
  union {
    unsigned long long packed;
    struct {
      int voxel;
      uint32_t seg;
    };
  };
  uint32_t count, unused;
};

__global__ void __launch_bounds__(kVoxThreads)
vox_clear_kernel(uint4* __restrict__ status, uint4* __restrict__ slots, long long n_slots) {
  const long long stride = static_cast<long long>(gridDim.x) * kVoxThreads, t = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  if (t < 16) status[t] = make_uint4(0u, 0u, 0u, 0u);
  for (long long i = t; i < n_slots; i += stride) slots[i] = make_uint4(~0u, ~0u, 0u, 0u);
}

enum VoxStatus { kVoxError = 0, kVoxTotal = 1, kVoxMost = 2, kVoxTicket = 3, kVoxCursor = 4 };

__global__ void __launch_bounds__(kVoxThreads)
quantize_insert_kernel(const __grid_constant__ VoxGeo g, const float* __restrict__ points, long long n,
                       int point_stride, VoxSlot* __restrict__ slots, uint32_t cap_mask, uint32_t* __restrict__ slot_of, uint32_t* __restrict__ place,
                       int* __restrict__ status) {
  const long long i = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  if (i >= n) return;
  const float* p = points + i * point_stride;
  uint32_t key = 0;
  bool in_range = true;
  for (int d = 0; d < g.ndim; ++d) {
    const float q = floorf(__fdiv_rn(__fsub_rn(__ldg(&p[d]), g.cmin[d]), g.vsize[d]));
    // NaN and out-of-range both fail the comparison chain
    if (!(q >= 0.f && q < static_cast<float>(g.grid[d]))) {
      in_range = false;
      break;
    }
    key = key * static_cast<uint32_t>(g.grid[d]) + static_cast<uint32_t>(q);
  }
  slot_of[i] = kNoKey;
  if (!in_range) return;
  const unsigned long long packed = (static_cast<unsigned long long>(key) << 32) | static_cast<uint32_t>(i);
  uint32_t s = vox_mix(key) & cap_mask;
  for (uint32_t probe = 0; probe <= cap_mask; ++probe) {
    const unsigned long long old = atomicCAS(&slots[s].packed, kVoxEmpty, packed);
    if (old == kVoxEmpty || static_cast<uint32_t>(old >> 32) == key) {
      if (old != kVoxEmpty) atomicMin(&slots[s].packed, packed);
      slot_of[i] = s;
      place[i] = atomicAdd(&slots[s].count, 1u);
      return;
    }
    s = (s + 1) & cap_mask;
  }
  atomicExch(&status[kVoxError], SPC_ERR_HASH_TABLE_FULL);
}

constexpr int kVoxBlock = 2048;  // points a block counts and numbers
constexpr int kVoxEach = kVoxBlock / kVoxThreads;

__device__ __forceinline__ uint32_t vox_block_sum(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  __syncthreads();
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kVoxThreads / 32; ++w) {
    if (w < warp) before += warp_sums[w];
    all += warp_sums[w];
  }
  *total = all;
  return before + incl - v;  // exclusive
}

// First points: their bits, and how many a block has; the last block to finish turns the sums into starts and
// hands the number of voxels and the largest count of points in one to the host.
__global__ void __launch_bounds__(kVoxThreads)
count_first_kernel(const uint32_t* __restrict__ slot_of, long long n, const VoxSlot* __restrict__ slots, uint32_t* __restrict__ first_bits,
                   uint32_t* __restrict__ starts, int* __restrict__ status, volatile int* host_box, int ticket) {
  __shared__ uint32_t warp_sums[kVoxThreads / 32];
  __shared__ int last;
  const long long base = blockIdx.x * static_cast<long long>(kVoxBlock);
  uint32_t mine = 0, most = 0;
  uint32_t slot[kVoxEach];
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e) {
    const long long i = base + e * kVoxThreads + threadIdx.x;
    slot[e] = i < n ? slot_of[i] : kNoKey;
  }
  uint4 held[kVoxEach];  // all requested before any is used
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e)
    held[e] = slot[e] != kNoKey ? *reinterpret_cast<const uint4*>(&slots[slot[e]]) : make_uint4(kNoKey, 0u, 0u, 0u);
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e) {
    const long long i = base + e * kVoxThreads + threadIdx.x;
    const bool first = slot[e] != kNoKey && held[e].x == static_cast<uint32_t>(i);  // (the low word of `packed`)
    const unsigned bits = __ballot_sync(0xffffffffu, first);
    if ((threadIdx.x & 31) == 0) first_bits[(base + e * kVoxThreads + threadIdx.x) >> 5] = bits;
    if (!first) continue;
    ++mine;
    most = max(most, held[e].z);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(&status[kVoxMost], static_cast<int>(most));
  uint32_t total;
  vox_block_sum(mine, warp_sums, &total);
  if (threadIdx.x == 0) {
    starts[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(&status[kVoxTicket], 1) == static_cast<int>(gridDim.x) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  volatile uint32_t* st = starts;
  uint32_t carry = 0;
  for (int b0 = 0; b0 < static_cast<int>(gridDim.x); b0 += kVoxThreads) {
    const int b = b0 + threadIdx.x;
    const uint32_t v = b < static_cast<int>(gridDim.x) ? st[b] : 0u;
    uint32_t all;
    const uint32_t before = vox_block_sum(v, warp_sums, &all);
    if (b < static_cast<int>(gridDim.x)) st[b] = carry + before;
    carry += all;
  }
  if (threadIdx.x == 0) {
    status[kVoxTotal] = static_cast<int>(carry);
    host_box[1] = *reinterpret_cast<volatile int*>(&status[kVoxError]);
    host_box[2] = static_cast<int>(carry);
    host_box[3] = *reinterpret_cast<volatile int*>(&status[kVoxMost]);
    __threadfence_system();
    host_box[0] = ticket;
  }
}

// The voxel number of every first point below the cap (else -1), its stretch of the list, its coordinates and
// its count.  Only first points touch their slot, so it can take its second meaning in place.
__global__ void __launch_bounds__(kVoxThreads)
number_voxels_kernel(const __grid_constant__ VoxGeo g, const uint32_t* __restrict__ slot_of, long long n, VoxSlot* __restrict__ slots,
                     const uint32_t* __restrict__ first_bits, const uint32_t* __restrict__ starts, long long max_voxels, int max_points,
                     int* __restrict__ status, int32_t* __restrict__ indices, int32_t* __restrict__ num_per_voxel) {
  constexpr int kWords = kVoxBlock / 32;
  __shared__ uint32_t before[kWords], bits_s[kWords];
  __shared__ uint32_t points, room;
  const long long base = blockIdx.x * static_cast<long long>(kVoxBlock);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) points = 0;
  if (warp == 0) {
    static_assert(kWords == 64, "two words a lane");
    const uint32_t a = first_bits[(base >> 5) + 2 * lane], b = first_bits[(base >> 5) + 2 * lane + 1];
    uint32_t incl = __popc(a) + __popc(b);
    const uint32_t both = incl;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    bits_s[2 * lane] = a;
    bits_s[2 * lane + 1] = b;
    before[2 * lane] = incl - both;
    before[2 * lane + 1] = incl - both + __popc(a);
  }
  __syncthreads();
  const uint32_t start = starts[blockIdx.x];
  uint32_t slot[kVoxEach], at[kVoxEach];
  uint4 held[kVoxEach];
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e) {
    const bool first = (bits_s[e * (kVoxThreads / 32) + warp] >> lane) & 1u;
    slot[e] = first ? slot_of[base + e * kVoxThreads + threadIdx.x] : kNoKey;
  }
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e)
    if (slot[e] != kNoKey) held[e] = *reinterpret_cast<const uint4*>(&slots[slot[e]]);
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e)
    if (slot[e] != kNoKey) at[e] = atomicAdd(&points, held[e].z);
  __syncthreads();
  if (threadIdx.x == 0) room = atomicAdd(reinterpret_cast<uint32_t*>(&status[kVoxCursor]), points);
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kVoxEach; ++e) {
    if (slot[e] == kNoKey) continue;
    const int w = e * (kVoxThreads / 32) + warp;
    const long long vid = static_cast<long long>(start) + before[w] + __popc(bits_s[w] & ((1u << lane) - 1u));
    const bool kept = vid < max_voxels;
    *reinterpret_cast<uint4*>(&slots[slot[e]]) =
        make_uint4(kept ? static_cast<uint32_t>(vid) : 0xffffffffu, room + at[e], held[e].z, 0u);
    if (!kept) continue;
    num_per_voxel[vid] = min(static_cast<int>(held[e].z), max_points);
    // the voxel's coordinates, reversed to (z, y, x)
    uint32_t rem = held[e].y;  // the key
    for (int d = g.ndim - 1; d >= 0; --d) {
      const uint32_t gd = static_cast<uint32_t>(g.grid[d]);
      indices[vid * g.ndim + (g.ndim - 1 - d)] = static_cast<int32_t>(rem % gd);
      rem /= gd;
    }
  }
}

// pc_voxel_id, and the point's index at its place in its voxel's stretch.
__global__ void __launch_bounds__(kVoxThreads)
place_kernel(const uint32_t* __restrict__ slot_of, const uint32_t* __restrict__ place, long long n, const VoxSlot* __restrict__ slots,
             int* __restrict__ list, long long* __restrict__ pc_voxel_id) {
  const long long i = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = slot_of[i];
  const uint4 held = s == kNoKey ? make_uint4(0xffffffffu, 0u, 0u, 0u) : __ldg(reinterpret_cast<const uint4*>(&slots[s]));
  const int v = static_cast<int>(held.x);
  pc_voxel_id[i] = v;
  if (v >= 0) list[held.y + place[i]] = static_cast<int>(i);
}

// chosen[voxel, slot] = the point stored there: the slot of a point is the number of earlier points of its voxel.
__global__ void __launch_bounds__(kVoxThreads)
rank_kernel(const uint32_t* __restrict__ slot_of, long long n, const VoxSlot* __restrict__ slots, const int* __restrict__ list,
            int max_points, int* __restrict__ chosen) {
  const long long i = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = slot_of[i];
  if (s == kNoKey) return;
  const uint4 held = __ldg(reinterpret_cast<const uint4*>(&slots[s]));
  const int v = static_cast<int>(held.x);
  if (v < 0) return;
  const uint32_t c = held.z;
  int rank = 0;
  if (c > 1) {
    const int* l = list + held.y;
    for (uint32_t q = 0; q < c; ++q) rank += __ldg(&l[q]) < static_cast<int>(i);
  }
  if (rank < max_points) chosen[static_cast<long long>(v) * max_points + rank] = static_cast<int>(i);
}

// The same from the points sorted by (voxel number, index): for voxels of so many points that counting the
// earlier ones of each would take longer than the sort.
__global__ void __launch_bounds__(kVoxThreads)
sort_keys_kernel(const long long* __restrict__ pc_voxel_id, long long n, uint32_t behind, uint32_t* __restrict__ keys, int* __restrict__ vals) {
  const long long i = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  if (i >= n) return;
  const long long v = pc_voxel_id[i];
  keys[i] = v < 0 ? behind : static_cast<uint32_t>(v);
  vals[i] = static_cast<int>(i);
}
__global__ void __launch_bounds__(kVoxThreads)
choose_sorted_kernel(const uint32_t* __restrict__ keys, const int* __restrict__ vals, long long n, uint32_t behind, int max_points,
                     int* __restrict__ chosen) {
  const long long i = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  if (i >= n) return;
  const uint32_t v = keys[i];
  if (v == behind) return;
  // the slot is the distance to the first position of this voxel, if that is less than max_points
  long long lo = i - max_points < 0 ? 0 : i - max_points, hi = i;
  if (lo < i && keys[lo] == v && i - lo >= max_points) return;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (keys[mid] == v) hi = mid;
    else lo = mid + 1;
  }
  chosen[static_cast<long long>(v) * max_points + (i - lo)] = vals[i];
}

// Rows of the voxel buffer and of the caller's copies (`out` .. `num_out`, may be null).  With `clear`: every
// element of every row, zeros where there is no point; without: only the stored points.
// An element is three dependent loads.  Four a thread, their counts and point numbers on their way together, where there are
// elements enough to fill the chip all the same (the rule is at the launch).
constexpr int kEmitEach = 4;
template <int VEC, int EACH, typename Index>
__global__ void __launch_bounds__(kVoxThreads)
emit_voxels_kernel(const float* __restrict__ points, int point_stride, int num_features, const int* __restrict__ chosen,
                   const int32_t* __restrict__ num_per_voxel, const int32_t* __restrict__ indices, int ndim, Index num_voxels, Index rows,
                   int max_points, int clear, float* __restrict__ voxels, float* __restrict__ out, int32_t* __restrict__ indices_out,
                   int32_t* __restrict__ num_out) {
  struct alignas(4 * VEC) Pack { float v[VEC]; };
  const Index per = static_cast<Index>(num_features / VEC), all = rows * static_cast<Index>(max_points) * per;
  const Index first = static_cast<Index>(blockIdx.x) * (kVoxThreads * EACH) + threadIdx.x;
  Index at[EACH];   // of the element's first float
  int stored[EACH], from[EACH];
#pragma unroll
  for (int i = 0; i < EACH; ++i) {
    const Index e = first + static_cast<Index>(i * kVoxThreads), ps = e / per;  // (voxel, slot)
    at[i] = e;
    stored[i] = from[i] = 0;
    if (e < all && ps < num_voxels * static_cast<Index>(max_points)) {
      stored[i] = num_per_voxel[ps / static_cast<Index>(max_points)];
      from[i] = chosen[ps];  // (read beside the count; of no meaning from the count on)
    }
  }
#pragma unroll
  for (int i = 0; i < EACH; ++i) {
    const Index e = at[i];
    if (e >= all) break;
    const Index ps = e / per, v = ps / static_cast<Index>(max_points);
    const int c = static_cast<int>(e - ps * per) * VEC, slot = static_cast<int>(ps - v * static_cast<Index>(max_points));
    Pack x;
#pragma unroll
    for (int q = 0; q < VEC; ++q) x.v[q] = 0.f;
    if (slot < stored[i]) x = *reinterpret_cast<const Pack*>(points + static_cast<long long>(from[i]) * point_stride + c);
    const long long to = static_cast<long long>(e) * VEC;
    if (slot < stored[i] || clear) *reinterpret_cast<Pack*>(voxels + to) = x;
    if (out == nullptr || v >= num_voxels) continue;
    *reinterpret_cast<Pack*>(out + to) = x;
    if (slot == 0 && c == 0) {
      num_out[v] = stored[i];
      for (int d = 0; d < ndim; ++d) indices_out[static_cast<long long>(v) * ndim + d] = indices[static_cast<long long>(v) * ndim + d];
    }
  }
}

// One thread per (voxel, feature): unused slots take the mean of the stored points,
// summed in slot order over ALL max_points slots as the reference's sum(dim=1) does.
__global__ void __launch_bounds__(kVoxThreads)
fill_mean_kernel(float* __restrict__ voxels, const int32_t* __restrict__ num_per_voxel, long long num_voxels,
                 int max_points, int num_features) {
  const long long e = blockIdx.x * static_cast<long long>(kVoxThreads) + threadIdx.x;
  const long long v = e / num_features;
  if (v >= num_voxels) return;
  const int c = static_cast<int>(e - v * num_features);
  const int npv = num_per_voxel[v];
  float* base = voxels + (v * max_points) * num_features + c;
  float sum = 0.f;
  for (int s = 0; s < max_points; ++s) sum += base[static_cast<long long>(s) * num_features];
  const float mean = __fdiv_rn(sum, static_cast<float>(npv > 1 ? npv : 1));
  for (int s = npv; s < max_points; ++s) base[static_cast<long long>(s) * num_features] = mean;
}

uint32_t vox_pow2_at_least(int64_t v) {
  uint32_t c = 1;
  while (static_cast<int64_t>(c) < v && c < (1u << 31)) c <<= 1;
  return c;
}

// Voxels of more points than this take the radix sort: counting earlier points is quadratic in a voxel's points.
constexpr int kVoxMostRanked = 256;

struct VoxLayout {
  uint32_t cap;
  size_t off_status, off_slots, off_slot_of, off_place, off_first, off_list, off_starts, off_chosen, off_sk_a,
      off_sk_b, off_sv_a, off_sv_b, off_cub, cub_bytes, total;
};

size_t vox_sort_bytes(int64_t n) {
  static std::atomic<size_t> known[64];
  int e = 0;
  while ((1ll << e) < n) ++e;
  size_t have = known[e].load(std::memory_order_relaxed);
  if (have != 0) return have;
  cub::DeviceRadixSort::SortPairs(nullptr, have, static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  static_cast<int*>(nullptr), static_cast<int*>(nullptr), static_cast<int>(1ll << e));
  have = std::max<size_t>(have, 16);
  known[e].store(have, std::memory_order_relaxed);
  return have;
}

VoxLayout vox_layout(int64_t n, int64_t max_voxels, int max_points) {
  VoxLayout L{};
  L.cap = std::max<uint32_t>(vox_pow2_at_least(n + n / 2), 64);
  L.cub_bytes = vox_sort_bytes(std::max<int64_t>(n, 1));
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t np = static_cast<size_t>(std::max<int64_t>(n, 1));
  const size_t nv = static_cast<size_t>(std::min<int64_t>(std::max<int64_t>(max_voxels, 1), np));
  L.off_status = take(256);
  L.off_slots = take(static_cast<size_t>(L.cap) * sizeof(VoxSlot));
  L.off_first = take(static_cast<size_t>(ceil_div(static_cast<int64_t>(np), kVoxBlock)) * (kVoxBlock / 8));
  L.off_slot_of = take(np * 4);
  L.off_place = take(np * 4);
  L.off_list = take(np * 4);
  L.off_starts = take(static_cast<size_t>(ceil_div(static_cast<int64_t>(np), kVoxBlock)) * 4);
  L.off_chosen = take(nv * max_points * 4);
  L.off_sk_a = take(np * 4);
  L.off_sk_b = take(np * 4);
  L.off_sv_a = take(np * 4);
  L.off_sv_b = take(np * 4);
  L.off_cub = take(L.cub_bytes);
  L.total = off;
  return L;
}

struct VoxArgs {
  const float* points;
  int64_t n;
  int point_stride, num_features;
  int64_t max_voxels;
  int max_points;
  VoxGeo g{};
};
int vox_check(const float* points, int64_t n_points, int point_stride, int ndim, int num_features, const float* cmin, const float* vsize,
              const int32_t* grid_xyz, int64_t max_voxels, int max_points, VoxArgs* a) {
  if (!cmin || !vsize || !grid_xyz || ndim < 1 || ndim > kVoxMaxDim || num_features < 1 ||
      point_stride < std::max(ndim, num_features) || max_voxels <= 0 || max_points <= 0 || n_points < 0)
    return fail(SPC_ERR_INVALID_ARGUMENT, "voxelize: bad arguments");
  if (n_points >= (1ll << 30)) return fail(SPC_ERR_SIZE_LIMIT, "voxelize: %lld points", static_cast<long long>(n_points));
  a->points = points;
  a->n = n_points;
  a->point_stride = point_stride;
  a->num_features = num_features;
  a->max_voxels = max_voxels;
  a->max_points = max_points;
  a->g.ndim = ndim;
  double volume = 1;
  for (int d = 0; d < ndim; ++d) {
    if (grid_xyz[d] <= 0 || !(vsize[d] > 0.f)) return fail(SPC_ERR_INVALID_ARGUMENT, "voxelize: bad grid");
    a->g.cmin[d] = cmin[d];
    a->g.vsize[d] = vsize[d];
    a->g.grid[d] = grid_xyz[d];
    volume *= grid_xyz[d];
  }
  if (volume >= 4294967295.0) return fail(SPC_ERR_SIZE_LIMIT, "voxelize: grid of %.0f cells needs keys beyond 32 bits", volume);
  return SPC_OK;
}

}  // namespace
}  // namespace spc

using namespace spc;

extern "C" size_t spc_voxelize_workspace_bytes(int64_t n_points, int64_t max_voxels, int max_points) {
  if (n_points < 0 || max_voxels <= 0 || max_points <= 0 || n_points >= (1ll << 30)) return 0;
  return vox_layout(n_points, max_voxels, max_points).total;
}

extern "C" int spc_voxelize_number(const float* points, int64_t n_points, int point_stride, int ndim, int num_features, const float* cmin,
                                   const float* vsize, const int32_t* grid_xyz, int64_t max_voxels, int max_points, void* workspace,
                                   size_t workspace_bytes, int32_t* indices, int32_t* num_per_voxel, int64_t* pc_voxel_id,
                                   int64_t* num_voxels_host, int* sorted_host, void* stream) {
  VoxArgs a;
  int rc = vox_check(points, n_points, point_stride, ndim, num_features, cmin, vsize, grid_xyz, max_voxels, max_points, &a);
  if (rc != SPC_OK) return rc;
  if (!num_voxels_host || !sorted_host || !indices || !num_per_voxel || !workspace || (n_points > 0 && (!points || !pc_voxel_id)))
    return fail(SPC_ERR_INVALID_ARGUMENT, "voxelize: bad arguments");
  *num_voxels_host = 0;
  *sorted_host = 0;
  if (n_points == 0) return SPC_OK;
  const VoxLayout L = vox_layout(n_points, max_voxels, max_points);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "voxelize: workspace %zu < %zu bytes", workspace_bytes, L.total);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  int* status = reinterpret_cast<int*>(ws + L.off_status);
  VoxSlot* slots = reinterpret_cast<VoxSlot*>(ws + L.off_slots);
  uint32_t* first_bits = reinterpret_cast<uint32_t*>(ws + L.off_first);
  uint32_t* slot_of = reinterpret_cast<uint32_t*>(ws + L.off_slot_of);
  uint32_t* place = reinterpret_cast<uint32_t*>(ws + L.off_place);
  uint32_t* starts = reinterpret_cast<uint32_t*>(ws + L.off_starts);
  const uint32_t cap_mask = L.cap - 1;
  volatile int* box = nullptr;
  int ticket = 0;
  rc = host_mailbox(&box, &ticket);
  if (rc != SPC_OK) return rc;
  vox_clear_kernel<<<static_cast<unsigned>(std::min<int64_t>(ceil_div(L.cap, kVoxThreads), 16ll * sm_count())), kVoxThreads, 0, st>>>(
      reinterpret_cast<uint4*>(status), reinterpret_cast<uint4*>(slots), L.cap);
  SPC_LAUNCH_OK();
  quantize_insert_kernel<<<vox_blocks(a.n), kVoxThreads, 0, st>>>(a.g, points, a.n, point_stride, slots, cap_mask, slot_of, place, status);
  SPC_LAUNCH_OK();
  const unsigned blocks = static_cast<unsigned>(ceil_div(a.n, kVoxBlock));
  count_first_kernel<<<blocks, kVoxThreads, 0, st>>>(slot_of, a.n, slots, first_bits, starts, status, box, ticket);
  SPC_LAUNCH_OK();
  number_voxels_kernel<<<blocks, kVoxThreads, 0, st>>>(a.g, slot_of, a.n, slots, first_bits, starts, max_voxels, max_points, status, indices,
                                                       num_per_voxel);
  SPC_LAUNCH_OK();
  place_kernel<<<vox_blocks(a.n), kVoxThreads, 0, st>>>(slot_of, place, a.n, slots, reinterpret_cast<int*>(ws + L.off_list),
                                                     reinterpret_cast<long long*>(pc_voxel_id));
  SPC_LAUNCH_OK();
  rc = wait_for_ticket(box, ticket, st);
  if (rc != SPC_OK) return rc;
  if (box[1] != 0) return fail(box[1], "voxelize: hash table full (status %d)", box[1]);
  *num_voxels_host = std::min<int64_t>(box[2], max_voxels);
  *sorted_host = box[3] > kVoxMostRanked;
  return SPC_OK;
}

extern "C" int spc_voxelize_store(const float* points, int64_t n_points, int point_stride, int ndim, int num_features, int64_t max_voxels,
                                  int max_points, int clear_voxels, int empty_mean, void* workspace, size_t workspace_bytes,
                                  int64_t num_voxels, int sorted, const int32_t* indices, const int32_t* num_per_voxel,
                                  const int64_t* pc_voxel_id, float* voxels, float* voxels_out, int32_t* indices_out, int32_t* num_out,
                                  void* stream) {
  if (!workspace || !indices || !num_per_voxel || !voxels || n_points < 0 || num_voxels < 0 || num_voxels > max_voxels || num_features < 1 ||
      max_points <= 0 || ndim < 1 || (n_points > 0 && (!points || !pc_voxel_id)) || (voxels_out && (!indices_out || !num_out)))
    return fail(SPC_ERR_INVALID_ARGUMENT, "voxelize: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const VoxLayout L = vox_layout(n_points, max_voxels, max_points);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "voxelize: workspace %zu < %zu bytes", workspace_bytes, L.total);
  char* ws = static_cast<char*>(workspace);
  int* chosen = reinterpret_cast<int*>(ws + L.off_chosen);
  if (num_voxels > 0 && !sorted) {
    rank_kernel<<<vox_blocks(n_points), kVoxThreads, 0, st>>>(
        reinterpret_cast<uint32_t*>(ws + L.off_slot_of), n_points, reinterpret_cast<VoxSlot*>(ws + L.off_slots),
        reinterpret_cast<int*>(ws + L.off_list),
        max_points, chosen);
    SPC_LAUNCH_OK();
  } else if (num_voxels > 0) {
    uint32_t* sk_a = reinterpret_cast<uint32_t*>(ws + L.off_sk_a);
    uint32_t* sk_b = reinterpret_cast<uint32_t*>(ws + L.off_sk_b);
    int* sv_a = reinterpret_cast<int*>(ws + L.off_sv_a);
    int* sv_b = reinterpret_cast<int*>(ws + L.off_sv_b);
    const uint32_t behind = static_cast<uint32_t>(num_voxels);  // dropped points sort behind every voxel
    sort_keys_kernel<<<vox_blocks(n_points), kVoxThreads, 0, st>>>(reinterpret_cast<const long long*>(pc_voxel_id), n_points, behind, sk_a, sv_a);
    SPC_LAUNCH_OK();
    int bits = 1;
    while (bits < 32 && (1ll << bits) <= num_voxels) ++bits;
    size_t cub_bytes = L.cub_bytes;
    SPC_CUDA_OK(cub::DeviceRadixSort::SortPairs(ws + L.off_cub, cub_bytes, sk_a, sk_b, sv_a, sv_b, static_cast<int>(n_points), 0, bits, st));
    choose_sorted_kernel<<<vox_blocks(n_points), kVoxThreads, 0, st>>>(sk_b, sv_b, n_points, behind, max_points, chosen);
    SPC_LAUNCH_OK();
  }
  const int64_t rows = clear_voxels ? max_voxels : num_voxels;
  const bool wide = num_features % 4 == 0 && point_stride % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(points) | reinterpret_cast<uintptr_t>(voxels) | reinterpret_cast<uintptr_t>(voxels_out)) & 15u) == 0;
  if (rows > 0) {
    const int64_t work = rows * max_points * (wide ? num_features / 4 : num_features);
    const bool small = work < (1ll << 31);
    const auto emit = [&](auto kernel, auto index, int each) {
      using Index = decltype(index);
      kernel<<<vox_blocks(ceil_div(work, each)), kVoxThreads, 0, st>>>(points, point_stride, num_features, chosen, num_per_voxel, indices, ndim,
                                                      static_cast<Index>(num_voxels), static_cast<Index>(rows), max_points, clear_voxels, voxels,
                                                      voxels_out, indices_out, num_out);
    };
    // Up to three times the threads that the chip holds, one element a thread: four leave it partly empty.  A call, us, four / one:
    // 0.02 of the chip's threads 47.2 / 43.1, 0.8 49.6 / 46.5, 1.3 51.9 / 50.2 and 53.4 / 52.6, 3.3 65.6 / 65.6, 13
    // 152.6 / 155.0.
    const bool few = work <= 3 * 2048 * static_cast<int64_t>(sm_count());
    if (wide && few) emit(emit_voxels_kernel<4, 1, uint32_t>, uint32_t{}, 1);
    else if (few) emit(emit_voxels_kernel<1, 1, uint32_t>, uint32_t{}, 1);
    else if (wide && small) emit(emit_voxels_kernel<4, kEmitEach, uint32_t>, uint32_t{}, kEmitEach);
    else if (wide) emit(emit_voxels_kernel<4, kEmitEach, long long>, 0ll, kEmitEach);
    else if (small) emit(emit_voxels_kernel<1, kEmitEach, uint32_t>, uint32_t{}, kEmitEach);
    else emit(emit_voxels_kernel<1, kEmitEach, long long>, 0ll, kEmitEach);
    SPC_LAUNCH_OK();
  }
  if (num_voxels == 0) return SPC_OK;
  if (empty_mean) {
    for (float* v : {voxels, voxels_out}) {
      if (v == nullptr) continue;
      fill_mean_kernel<<<vox_blocks(num_voxels * num_features), kVoxThreads, 0, st>>>(v, num_per_voxel, num_voxels, max_points, num_features);
      SPC_LAUNCH_OK();
    }
  }
  return SPC_OK;
}

extern "C" int spc_voxelize(const float* points, int64_t n_points, int point_stride, int ndim, int num_features,
                            const float* cmin, const float* vsize, const int32_t* grid_xyz, int64_t max_voxels,
                            int max_points, int clear_voxels, int empty_mean, void* workspace,
                            size_t workspace_bytes, float* voxels, int32_t* indices, int32_t* num_per_voxel,
                            int64_t* pc_voxel_id, int64_t* num_voxels_host, void* stream) {
  if (!voxels) return fail(SPC_ERR_INVALID_ARGUMENT, "voxelize: bad arguments");
  int sorted = 0;
  const int rc = spc_voxelize_number(points, n_points, point_stride, ndim, num_features, cmin, vsize, grid_xyz, max_voxels, max_points,
                                     workspace, workspace_bytes, indices, num_per_voxel, pc_voxel_id, num_voxels_host, &sorted, stream);
  if (rc != SPC_OK) return rc;
  return spc_voxelize_store(points, n_points, point_stride, ndim, num_features, max_voxels, max_points, clear_voxels, empty_mean, workspace,
                            workspace_bytes, *num_voxels_host, sorted, indices, num_per_voxel, pc_voxel_id, voxels, nullptr, nullptr, nullptr,
                            stream);
}
