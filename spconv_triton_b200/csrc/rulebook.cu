// Rulebook (indice-pair) generation for sparse convolution on B200.
//
// Design (differs from the reference on purpose): the reference materialises
// the kv*N candidate grid (out_lin, valid, out_row) in HBM, sorts the input
// coordinates, runs kv*N binary searches and scatters into -1 pre-filled
// tables (spconv_triton/pytorch/_impl/pairs.py:126-426).  Here an occupancy bitmap of the
// input grid and a hash table keyed by the batch-major linear coordinate replace
// the sorts and searches (grids too large for a bitmap: hash tables alone).  A
// thread owns a row: of a submanifold layer it looks the neighbours up, one
// bitmap window per line of offsets, the present ones in the hash table; of a
// strided or transposed layer it walks the one to eight outputs of an INPUT row
// and scatters the pair into both tables.  Output rows are numbered by the rank
// of their bit, which is the ascending order torch.unique gives the reference,
// without a sort (grids too large for a bitmap: a hash table and a library radix
// sort of its keys).  No candidate grid.  A submanifold layer's entries are plain
// stores; a strided layer's output side is cleared and scattered to with atomicMin
// (the lowest input row of equal coordinates wins) and atomicOr (mask words).  The
// tables are L2-resident (126 MB) up to a few hundred thousand rows.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <atomic>
#include <climits>
#include <type_traits>

#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "gemm_internal.cuh"
#include "rulebook_internal.cuh"
#include "tile_order.cuh"

namespace spc {
namespace {

constexpr int kThreads = 256;

struct Geo {
  int ndim, batch, subm, transpose, kv;
  int in_shape[SPC_MAX_NDIM], out_shape[SPC_MAX_NDIM];
  int ksize[SPC_MAX_NDIM], stride[SPC_MAX_NDIM], pad[SPC_MAX_NDIM], dil[SPC_MAX_NDIM];
  int shift[SPC_MAX_NDIM];    // log2 of a stride that is a power of two, else -1
  int axes_fit;               // every axis has at most 32 offsets: the valid ones are a bitmask
  int window;                 // the cells of a line of offsets lie in one 64-bit window of the occupancy bitmap
  unsigned char key_pos[32];  // bit k of the mask word goes to bit key_pos[k] of the tile-order word (kv <= 32)
};

// ------------------------------------------------------------------------
// Hash tables.  K64 = false: key < 2^31, slot = (key << 32) | value in one
// 64-bit word, so a probe is one 8-byte access and an insert one atomicCAS.
// K64 = true: 64-bit keys with a separate value array.
// Probing is linear and bounded by the capacity; a full table raises a status
// flag instead of spinning.
// ------------------------------------------------------------------------
__device__ __forceinline__ uint32_t mix32(uint32_t h) {
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}

template <bool K64>
struct Table;

template <>
struct Table<false> {
  using key_t = uint32_t;
  unsigned long long* slots;
  uint32_t cap_mask;
  // Dense numbering (output side of strided layers on a grid small enough for a bitmap): one bit per
  // cell and, per 32-bit word, the number of set bits before it.  The value of a key is then its
  // rank among the set bits = its row in ascending key order, with no hash table and no sort.
  uint32_t* obits = nullptr;
  const uint32_t* oprefix = nullptr;
  // Input side: rows equal ranks only when the rows came in ascending key order (the outputs of an
  // earlier layer do); where `unsorted` points at a device flag that says they did not, row = perm[rank].
  const int* unsorted = nullptr;
  const int32_t* perm = nullptr;
  __device__ __forceinline__ bool permuted() const { return unsorted != nullptr && *unsorted != 0; }
  __device__ __forceinline__ int rank_of(key_t key) const {
    const uint32_t w = __ldg(&obits[key >> 5]);
    if (!((w >> (key & 31u)) & 1u)) return -1;
    return static_cast<int>(__ldg(&oprefix[key >> 5]) + __popc(w & ((1u << (key & 31u)) - 1u)));
  }
  static constexpr unsigned long long kEmpty = ~0ull;

  // Four consecutive keys (neighbours along the fastest coordinate) share one
  // 32-byte sector: the block is chosen by hashing key >> 2, the lane inside it
  // by key & 3, and probing moves a whole block at a time.  The three x
  // neighbours of a voxel then cost one or two sectors instead of three.
  static constexpr uint32_t kStep = 4;
  __device__ __forceinline__ uint32_t home(key_t k) const { return ((mix32(k >> 2) << 2) | (k & 3u)) & cap_mask; }

  // Keeps the smallest value among equal keys (duplicate coordinates resolve
  // to the lowest row, as a stable sort + lower bound does in the reference).
  __device__ bool insert_min(key_t key, uint32_t val) const {
    const unsigned long long packed = (static_cast<unsigned long long>(key) << 32) | val;
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      unsigned long long old = atomicCAS(&slots[s], kEmpty, packed);
      if (old == kEmpty) return true;
      if (static_cast<key_t>(old >> 32) == key) {
        atomicMin(&slots[s], packed);
        return true;
      }
      s = (s + kStep) & cap_mask;
    }
    return false;
  }
  // 1: this call inserted the key, 0: already present, -1: table full.
  __device__ int insert_unique(key_t key) const {
    const unsigned long long packed = (static_cast<unsigned long long>(key) << 32) | 0x7fffffffu;
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      unsigned long long old = atomicCAS(&slots[s], kEmpty, packed);
      if (old == kEmpty) return 1;
      if (static_cast<key_t>(old >> 32) == key) return 0;
      s = (s + kStep) & cap_mask;
    }
    return -1;
  }
  __device__ int find(key_t key) const {
    if (obits != nullptr) {
      const int rank = rank_of(key);
      return rank >= 0 && permuted() ? __ldg(&perm[rank]) : rank;
    }
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      const unsigned long long v = __ldg(&slots[s]);
      if (v == kEmpty) return -1;
      if (static_cast<key_t>(v >> 32) == key) return static_cast<int>(v & 0xffffffffu);
      s = (s + kStep) & cap_mask;
    }
    return -1;
  }
  // A look-up split in two so that several keys' first probes can be in flight at once:
  // first_probe() returns the home slot's word, finish() resolves it (almost always at once).
  __device__ __forceinline__ unsigned long long first_probe(key_t key) const { return __ldg(&slots[home(key)]); }
  // Whether a home slot's word that is not empty is the key's; *row = its row then.
  __device__ __forceinline__ bool settled(key_t key, unsigned long long v, int* row) const {
    *row = static_cast<int>(v & 0xffffffffu);
    return static_cast<key_t>(v >> 32) == key;
  }
  __device__ __forceinline__ int finish(key_t key, unsigned long long v) const {
    if (v == kEmpty) return -1;
    if (static_cast<key_t>(v >> 32) == key) return static_cast<int>(v & 0xffffffffu);
    uint32_t s = (home(key) + kStep) & cap_mask;
    for (uint32_t probe = 1; probe <= (cap_mask >> 2); ++probe) {
      const unsigned long long w = __ldg(&slots[s]);
      if (w == kEmpty) return -1;
      if (static_cast<key_t>(w >> 32) == key) return static_cast<int>(w & 0xffffffffu);
      s = (s + kStep) & cap_mask;
    }
    return -1;
  }
  __device__ void set_value(key_t key, uint32_t val) const {
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      const unsigned long long v = slots[s];
      if (v == kEmpty) return;
      if (static_cast<key_t>(v >> 32) == key) {
        slots[s] = (static_cast<unsigned long long>(key) << 32) | val;
        return;
      }
      s = (s + kStep) & cap_mask;
    }
  }
};

template <>
struct Table<true> {
  using key_t = unsigned long long;
  unsigned long long* slots;  // keys
  int* vals;
  uint32_t cap_mask;
  static constexpr unsigned long long kEmpty = ~0ull;

  static constexpr uint32_t kStep = 4;
  __device__ __forceinline__ uint32_t home(key_t k) const {
    const key_t b = k >> 2;
    return ((mix32(static_cast<uint32_t>(b) ^ mix32(static_cast<uint32_t>(b >> 32))) << 2) |
            (static_cast<uint32_t>(k) & 3u)) & cap_mask;
  }
  __device__ bool insert_min(key_t key, uint32_t val) const {
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      unsigned long long old = atomicCAS(&slots[s], kEmpty, key);
      if (old == kEmpty || old == key) {
        atomicMin(&vals[s], static_cast<int>(val));
        return true;
      }
      s = (s + kStep) & cap_mask;
    }
    return false;
  }
  __device__ int insert_unique(key_t key) const {
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      unsigned long long old = atomicCAS(&slots[s], kEmpty, key);
      if (old == kEmpty) return 1;
      if (old == key) return 0;
      s = (s + kStep) & cap_mask;
    }
    return -1;
  }
  __device__ int find(key_t key) const {
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      const unsigned long long v = __ldg(&slots[s]);
      if (v == kEmpty) return -1;
      if (v == key) return __ldg(&vals[s]);
      s = (s + kStep) & cap_mask;
    }
    return -1;
  }
  __device__ __forceinline__ unsigned long long first_probe(key_t) const { return 0; }
  __device__ __forceinline__ bool settled(key_t, unsigned long long, int*) const { return false; }
  __device__ __forceinline__ int finish(key_t key, unsigned long long) const { return find(key); }
  __device__ void set_value(key_t key, uint32_t val) const {
    uint32_t s = home(key);
    for (uint32_t probe = 0; probe <= (cap_mask >> 2); ++probe) {
      const unsigned long long v = slots[s];
      if (v == kEmpty) return;
      if (v == key) {
        vals[s] = static_cast<int>(val);
        return;
      }
      s = (s + kStep) & cap_mask;
    }
  }
};

// ------------------------------------------------------------------------
// Coordinate arithmetic (follows spconv_triton/pytorch/_impl/pair_kernels.py:66-91).
// Kernel offsets are enumerated row-major, last dimension fastest, never
// flipped (spconv_triton/pytorch/_impl/pairs.py:43-48).
// ------------------------------------------------------------------------
template <int ND>
struct Odometer {
  int pos[ND];
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int d = 0; d < ND; ++d) pos[d] = 0;
  }
  __device__ __forceinline__ void set(const Geo& g, int k) {
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      pos[d] = k % g.ksize[d];
      k /= g.ksize[d];
    }
  }
  __device__ __forceinline__ void next(const Geo& g) {
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      if (++pos[d] < g.ksize[d]) return;
      pos[d] = 0;
    }
  }
};

// Output linear coordinate reached from input coordinate `c` through kernel
// offset `kp`, or -1 if that offset does not produce an output.
template <int ND>
__device__ __forceinline__ long long out_key_from_input(const Geo& g, const int* c, const int* kp) {
  long long lin = c[0];
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    int o;
    if (g.transpose) {
      o = c[d + 1] * g.stride[d] + kp[d] * g.dil[d] - g.pad[d];
    } else {
      const int num = c[d + 1] + g.pad[d] - kp[d] * g.dil[d];
      if (num < 0) return -1;
      o = num / g.stride[d];
      if (o * g.stride[d] != num) return -1;
    }
    if (o < 0 || o >= g.out_shape[d]) return -1;
    lin = lin * g.out_shape[d] + o;
  }
  return lin;
}

template <int ND>
__device__ __forceinline__ void load_coord(const int32_t* __restrict__ idx, long long row, int* c) {
#pragma unroll
  for (int d = 0; d <= ND; ++d) c[d] = __ldg(&idx[row * (ND + 1) + d]);
}

// A row whose batch index or coordinates lie outside [0, batch) x [0, in_shape) must not be
// turned into a bitmap or table index.  Kernels skip such rows (they get no pairs); the phase-1
// kernels also record SPC_ERR_INVALID_ARGUMENT so that the host raises.
template <int ND>
__device__ __forceinline__ bool coord_in_grid(const Geo& g, const int* c) {
  bool ok = c[0] >= 0 && c[0] < g.batch;
#pragma unroll
  for (int d = 0; d < ND; ++d) ok = ok && c[d + 1] >= 0 && c[d + 1] < g.in_shape[d];
  return ok;
}
__device__ __forceinline__ void flag_bad_row(int* counters, int* dev_status) {
  atomicExch(&counters[1], SPC_ERR_INVALID_ARGUMENT);  // counters[kStatus]
  if (dev_status != nullptr) atomicExch(dev_status, SPC_ERR_INVALID_ARGUMENT);
}

template <int ND>
__device__ __forceinline__ long long in_key_of(const Geo& g, const int* c) {
  long long lin = c[0];
#pragma unroll
  for (int d = 0; d < ND; ++d) lin = lin * g.in_shape[d] + c[d + 1];
  return lin;
}

template <int ND>
__device__ __forceinline__ void delinearize_out(const Geo& g, long long lin, int* c) {
#pragma unroll
  for (int d = ND - 1; d >= 0; --d) {
    c[d + 1] = static_cast<int>(lin % g.out_shape[d]);
    lin /= g.out_shape[d];
  }
  c[0] = static_cast<int>(lin);
}

enum Counter { kUniqueCount = 0, kStatus = 1, kUnsorted = 2, kTicket = 3 };

// ------------------------------------------------------------------------
// Phase 1 kernels
// ------------------------------------------------------------------------
// Scratch regions are cleared by a kernel rather than by cudaMemsetAsync, and all of them by one launch: a
// kernel can neither be routed to a copy engine (where it would queue behind a large transfer of the
// application) nor cost a driver memset's set-up.  Regions are whole words and may start and end anywhere: the
// caller's tables do.
struct Clear {
  static constexpr int kMost = 8;
  uint4* at[kMost];         // the 16-byte vectors of a region,
  long long n16[kMost];
  int head[kMost], tail[kMost];  // and up to three words before and behind them
  uint32_t word[kMost];
  int n = 0;
  long long total = 0;
  void add(void* p, int byte, size_t bytes) {
    if (bytes == 0) return;
    const size_t words = bytes / 4;
    const size_t before = std::min<size_t>((16 - (reinterpret_cast<uintptr_t>(p) & 15u)) % 16 / 4, words);
    at[n] = reinterpret_cast<uint4*>(static_cast<uint32_t*>(p) + before);
    n16[n] = static_cast<long long>((words - before) / 4);
    head[n] = static_cast<int>(before);
    tail[n] = static_cast<int>((words - before) % 4);
    word[n] = 0x01010101u * (static_cast<uint32_t>(byte) & 0xffu);
    total += n16[n++] + 1;
  }
};
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ Clear c) {
  const long long stride = static_cast<long long>(gridDim.x) * 256;
  for (int s = 0; s < c.n; ++s) {
    const uint4 v = make_uint4(c.word[s], c.word[s], c.word[s], c.word[s]);
    uint4* __restrict__ dst = c.at[s];
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < c.n16[s]; i += stride) dst[i] = v;
    if (blockIdx.x == 0 && threadIdx.x < 8) {
      const int t = threadIdx.x & 3;
      if (threadIdx.x < 4 && t < c.head[s]) (reinterpret_cast<uint32_t*>(dst) - c.head[s])[t] = v.x;
      if (threadIdx.x >= 4 && t < c.tail[s]) reinterpret_cast<uint32_t*>(dst + c.n16[s])[t] = v.x;
    }
  }
}

__device__ __forceinline__ uint32_t* dense_bits(const Table<false>& t) { return t.obits; }
__device__ __forceinline__ uint32_t* dense_bits(const Table<true>&) { return nullptr; }
__device__ __forceinline__ const uint32_t* dense_prefix(const Table<false>& t) { return t.oprefix; }
__device__ __forceinline__ const uint32_t* dense_prefix(const Table<true>&) { return nullptr; }
__device__ __forceinline__ const int32_t* row_permutation(const Table<false>& t) { return t.permuted() ? t.perm : nullptr; }
__device__ __forceinline__ const int32_t* row_permutation(const Table<true>&) { return nullptr; }

__device__ __forceinline__ void set_bit(uint32_t* bits, long long cell) {
  uint32_t* word = bits + (cell >> 5);
  const uint32_t bit = 1u << (cell & 31);
  if (!(*word & bit)) atomicOr(word, bit);
}

// The cells an own coordinate meets along axis d: `div` = the cell is what this coordinate was reached from
// ((own + pad - k * dil) / stride, if that divides), else own * stride - pad + k * dil.
// Returns -1 where there is none.
__device__ __forceinline__ int axis_cell(const Geo& g, bool div, int d, int own, int k, int limit) {
  int x;
  if (div) {
    x = own + g.pad[d] - k * g.dil[d];
    if (x < 0) return -1;
    if (g.shift[d] >= 0) {
      if (x & ((1 << g.shift[d]) - 1)) return -1;
      x >>= g.shift[d];
    } else {
      const int q = x / g.stride[d];
      if (q * g.stride[d] != x) return -1;
      x = q;
    }
  } else {
    x = own * g.stride[d] - g.pad[d] + k * g.dil[d];
  }
  return x >= 0 && x < limit ? x : -1;
}

// The bits of every output cell an input row reaches.  Per axis only the kernel offsets that land on an
// output coordinate are kept (a bitmask over the offsets of that axis: with stride 2 and a 3-wide kernel
// one or two of three), and the cells are the product of the axes, so a k3 s2 layer visits at most 8
// candidates per input instead of testing all 27.
template <int D, int ND>
__device__ __forceinline__ void mark_cells(const Geo& g, const int* c, const uint32_t* mask, long long lin,
                                           uint32_t* __restrict__ bits) {
  if constexpr (D == ND) {
    set_bit(bits, lin);
  } else {
    for (uint32_t m = mask[D]; m != 0; m &= m - 1)
      mark_cells<D + 1, ND>(g, c, mask,
                            lin * g.out_shape[D] + axis_cell(g, !g.transpose, D, c[D + 1], __ffs(m) - 1, g.out_shape[D]), bits);
  }
}

// First pass over the input rows: checks them, enters them into the input table (`in_bits`: the bit of the
// cell, noting whether the rows are in strictly ascending key order; else the hash table, if `insert`) and,
// with `out_bits`, marks the output cells.  `cells`: the rows' cells, where an earlier layer has listed them
// (its coordinates need not have been written yet).  One pass instead of one each: the coordinates are read once and
// a small rulebook is three launches shorter.
template <int ND, bool K64>
__global__ void __launch_bounds__(kThreads)
ingest_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ idx, const uint32_t* __restrict__ cells,
              long long n, Table<K64> tin, int insert, uint32_t* __restrict__ in_bits, uint32_t* __restrict__ out_bits, int* counters, int* dev_status) {
  const long long j = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (j >= n) return;
  int c[ND + 1];
  if (cells != nullptr) {
    uint32_t lin = cells[j];
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      const uint32_t q = lin / static_cast<uint32_t>(g.in_shape[d]);
      c[d + 1] = static_cast<int>(lin - q * static_cast<uint32_t>(g.in_shape[d]));
      lin = q;
    }
    c[0] = static_cast<int>(lin);
  } else {
    load_coord<ND>(idx, j, c);
  }
  if (!coord_in_grid<ND>(g, c)) {
    flag_bad_row(counters, dev_status);
    counters[kUnsorted] = 1;  // a skipped row breaks "row number = rank of its bit"
    return;
  }
  const long long key = in_key_of<ND>(g, c);
  if (in_bits != nullptr) {
    set_bit(in_bits, key);
    if (j > 0) {
      int p[ND + 1];
      load_coord<ND>(idx, j - 1, p);
      if (in_key_of<ND>(g, p) >= key) counters[kUnsorted] = 1;
    }
  } else if (insert) {
    using key_t = typename Table<K64>::key_t;
    if (!tin.insert_min(static_cast<key_t>(key), static_cast<uint32_t>(j)))
      atomicExch(&counters[kStatus], SPC_ERR_HASH_TABLE_FULL);
  }
  if (out_bits == nullptr) return;
  uint32_t mask[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    uint32_t m = 0;
    for (int k = 0; k < g.ksize[d]; ++k)
      m |= static_cast<uint32_t>(axis_cell(g, !g.transpose, d, c[d + 1], k, g.out_shape[d]) >= 0) << k;
    if (m == 0) return;
    mask[d] = m;
  }
  mark_cells<0, ND>(g, c, mask, c[0], out_bits);
}

// ------------------------------------------------------------------------
// Numbering the set bits of the input and the output bitmap in ascending cell order.  A block owns 2048
// words.  count_cells_kernel adds up every block's bits; its last block to finish turns the sums into
// starts and hands the output count to the host, which can then allocate while number_cells_kernel gives
// every word the number of bits before it and lists the output cells.  (A library scan over the words plus
// separate counting, listing and publishing kernels was five launches more per bitmap.)
// ------------------------------------------------------------------------
constexpr int kCellBlock = 2048;
constexpr int kWordsPerThread = kCellBlock / kThreads;

struct Cells {
  const uint32_t* bits[2];  // input, output (null: not there)
  uint32_t* prefix[2];
  uint32_t* starts[2];      // per block: its bits, then the bits before it; one more entry for the total
  long long words[2];
  int blocks[2];
};

// counters[kUniqueCount], counters[kStatus] and the device status word -> page-locked host memory; the
// ticket last, so that a host that sees it sees the rest.
__device__ void publish(const int* counters, const int* dev_status, volatile int* host_box, int ticket) {
  host_box[1] = counters[kUniqueCount];
  host_box[2] = counters[kStatus];
  host_box[3] = dev_status != nullptr ? *dev_status : 0;
  __threadfence_system();
  host_box[0] = ticket;
}
__global__ void publish_counters_kernel(const int* counters, const int* dev_status, int* host_box, int ticket) {
  if (threadIdx.x == 0) publish(counters, dev_status, host_box, ticket);
}

__device__ __forceinline__ uint32_t block_exclusive_sum(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  __syncthreads();  // warp_sums may still be read from a previous call
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    if (w < warp) before += warp_sums[w];
    all += warp_sums[w];
  }
  *total = all;
  return before + incl - v;
}

__global__ void __launch_bounds__(kThreads)
count_cells_kernel(const __grid_constant__ Cells c, int* counters, const int* dev_status, int* host_box, int ticket) {
  __shared__ uint32_t warp_sums[kThreads / 32];
  __shared__ int last;
  const int side = blockIdx.x < static_cast<unsigned>(c.blocks[0]) ? 0 : 1;
  const int block = blockIdx.x - (side ? c.blocks[0] : 0);
  const uint32_t* bits = c.bits[side];
  const long long first = static_cast<long long>(block) * kCellBlock;
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kWordsPerThread; ++i) {
    const long long w = first + i * kThreads + threadIdx.x;
    if (w < c.words[side]) sum += __popc(bits[w]);
  }
  uint32_t total;
  block_exclusive_sum(sum, warp_sums, &total);
  if (threadIdx.x == 0) {
    c.starts[side][block] = total;
    __threadfence();
    last = atomicAdd(&counters[kTicket], 1) == static_cast<int>(gridDim.x) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int s = 0; s < 2; ++s) {
    volatile uint32_t* starts = c.starts[s];
    uint32_t carry = 0;
    constexpr int kEach = 4;
    for (int b0 = 0; b0 < c.blocks[s]; b0 += kEach * kThreads) {
      uint32_t v[kEach], sum4 = 0, all;
#pragma unroll
      for (int q = 0; q < kEach; ++q) {
        const int b = b0 + threadIdx.x * kEach + q;
        v[q] = b < c.blocks[s] ? starts[b] : 0u;
        sum4 += v[q];
      }
      uint32_t before = carry + block_exclusive_sum(sum4, warp_sums, &all);
#pragma unroll
      for (int q = 0; q < kEach; ++q) {
        const int b = b0 + threadIdx.x * kEach + q;
        if (b < c.blocks[s]) starts[b] = before;
        before += v[q];
      }
      carry += all;
    }
    if (threadIdx.x == 0 && c.blocks[s] != 0) {
      starts[c.blocks[s]] = carry;
      if (s == 1) counters[kUniqueCount] = static_cast<int>(carry);
    }
  }
  if (threadIdx.x == 0 && host_box != nullptr) {
    __threadfence();
    publish(counters, dev_status, host_box, ticket);
  }
}

__global__ void __launch_bounds__(kThreads)
number_cells_kernel(const __grid_constant__ Cells c, long long limit, uint32_t* __restrict__ sorted) {
  __shared__ uint32_t warp_sums[kThreads / 32];
  const int side = blockIdx.x < static_cast<unsigned>(c.blocks[0]) ? 0 : 1;
  const int block = blockIdx.x - (side ? c.blocks[0] : 0);
  const uint32_t start = c.starts[side][block];
  if (c.starts[side][block + 1] == start) return;  // an empty block: nobody asks for the prefix of a zero word
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t* bits = c.bits[side];
  uint32_t* prefix = c.prefix[side];
  const long long first = static_cast<long long>(block) * kCellBlock + warp * (kCellBlock / (kThreads / 32)) + lane;
  uint32_t word[kWordsPerThread], sum = 0;
#pragma unroll
  for (int i = 0; i < kWordsPerThread; ++i) {
    const long long w = first + i * 32;
    word[i] = w < c.words[side] ? bits[w] : 0u;
    sum += __popc(word[i]);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if (lane == 0) warp_sums[warp] = sum;
  __syncthreads();
  uint32_t at = start;
  for (int w = 0; w < warp; ++w) at += warp_sums[w];
#pragma unroll
  for (int i = 0; i < kWordsPerThread; ++i) {
    const uint32_t mine = __popc(word[i]);
    uint32_t incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    const uint32_t before = at + incl - mine;
    at += __shfl_sync(0xffffffffu, incl, 31);
    if (word[i] != 0) prefix[first + i * 32] = before;
    if (side == 0) continue;
    const uint32_t in_warp = __shfl_sync(0xffffffffu, incl, 31);
    if (in_warp <= 8 * 32) {
      // few cells a word: every lane lists those of its own
      uint32_t to = before;
      for (uint32_t w = word[i]; w != 0 && to < limit; w &= w - 1)
        sorted[to++] = static_cast<uint32_t>((first + i * 32) * 32 + __ffs(w) - 1);
      continue;
    }
    // many: the warp lists one word's cells at a time, consecutive lanes to consecutive entries
    unsigned some = __ballot_sync(0xffffffffu, word[i] != 0);
    while (some != 0) {
      const int src = __ffs(some) - 1;
      some &= some - 1;
      const uint32_t w = __shfl_sync(0xffffffffu, word[i], src);
      const uint32_t to = __shfl_sync(0xffffffffu, before, src) + __popc(w & ((1u << lane) - 1u));
      if (((w >> lane) & 1u) && to < limit)
        sorted[to] = static_cast<uint32_t>((first - lane + i * 32 + src) * 32 + lane);
    }
  }
}

// perm[rank of a row's cell] = the row (the lowest one of equal coordinates, as a stable sort and a lower
// bound give in the reference), where the rows did not come in ascending order.
template <int ND>
__global__ void __launch_bounds__(kThreads)
permute_rows_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ idx, long long n, Table<false> tin,
                    int32_t* __restrict__ perm) {
  if (!tin.permuted()) return;
  const long long j = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (j >= n) return;
  int c[ND + 1];
  load_coord<ND>(idx, j, c);
  if (!coord_in_grid<ND>(g, c)) return;
  atomicMin(&perm[tin.rank_of(static_cast<uint32_t>(in_key_of<ND>(g, c)))], static_cast<int32_t>(j));
}

// One thread per input row walks the kv offsets and inserts each candidate
// output coordinate into the output table (grids too large for a bitmap).  Offsets are handled in groups of
// 32: a thread remembers in a bitmask which of its candidates were first-time
// inserts, the warp reserves room for all of them in `uniq` with ONE atomicAdd
// per group (a per-insert counter serialises on a single address), and a
// second walk over the group writes the keys.
template <int ND, bool K64>
__global__ void __launch_bounds__(kThreads)
enumerate_outputs_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ idx, long long n,
                         Table<K64> tout, typename Table<K64>::key_t* __restrict__ uniq,
                         int* counters) {
  using key_t = typename Table<K64>::key_t;
  const long long j = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  bool live = j < n;
  int c[ND + 1];
  if (live) {
    load_coord<ND>(idx, j, c);
    live = coord_in_grid<ND>(g, c);  // a row outside the grid (recorded by the input pass) reaches no output
  }
  const unsigned lane = threadIdx.x & 31u;
  for (int k0 = 0; k0 < g.kv; k0 += 32) {
    const int gcount = min(32, g.kv - k0);
    Odometer<ND> od;
    od.set(g, k0);
    uint32_t fresh = 0;
    if (live) {
      for (int kk = 0; kk < gcount; ++kk) {
        const long long key = out_key_from_input<ND>(g, c, od.pos);
        if (key >= 0) {
          if (dense_bits(tout) != nullptr) {
            set_bit(dense_bits(tout), key);
          } else {
            const int r = tout.insert_unique(static_cast<key_t>(key));
            if (r < 0) atomicExch(&counters[kStatus], SPC_ERR_HASH_TABLE_FULL);
            fresh |= static_cast<uint32_t>(r > 0) << kk;
          }
        }
        od.next(g);
      }
    }
    // warp-inclusive prefix of the per-thread counts
    const int mine = __popc(fresh);
    int incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= static_cast<unsigned>(off)) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (total == 0) continue;
    int base = 0;
    if (lane == 31) base = atomicAdd(&counters[kUniqueCount], total);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - mine;
    if (fresh) {
      od.set(g, k0);
      for (int kk = 0; kk < gcount; ++kk) {
        if ((fresh >> kk) & 1u) uniq[base++] = static_cast<key_t>(out_key_from_input<ND>(g, c, od.pos));
        od.next(g);
      }
    }
  }
}

template <bool K64>
__global__ void __launch_bounds__(kThreads)
assign_ranks_kernel(Table<K64> tout, const typename Table<K64>::key_t* __restrict__ sorted,
                    long long n_out) {
  const long long r = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (r < n_out) tout.set_value(sorted[r], static_cast<uint32_t>(r));
}

// ------------------------------------------------------------------------
// Phase 2 kernels (implicit-gemm tables)
// ------------------------------------------------------------------------
// What a fill kernel writes for its rows; every pointer may be null.
struct FillOut {
  int32_t* cm;           // [kv, n]: the neighbour table, column-major
  int32_t* rm;           // [n, kvp]: the same, row-major, padded with -1
  int32_t* cm_rev;       // both with the offset axis reversed: the input side of a submanifold layer, whose
  int32_t* rm_rev;       //   offset k seen from the input is offset kv - 1 - k seen from the output
  uint32_t* words;       // [n, mic]: bit k = offset k has a neighbour
  int32_t* iota;         // 0..n-1 (values of the exact mask sort)
  uint32_t* keys;        // [n]: key of the tile order (kv <= 32)
  uint32_t* counts;      // rows per bucket of that order (kTileBuckets, zeroed), or null
  // Input side only: the output side's tables, pre-filled with -1 (words: 0), to which every pair found is
  // scattered.  The lowest input row wins an entry, as equal coordinates resolve elsewhere (-1 is the
  // largest unsigned number).
  int32_t* out_cm;       // [kv, n_limit]
  int32_t* out_rm;       // [n_limit, kvp]
  uint32_t* out_words;   // [n_limit, mic]: mask words, or tile-order words with `order_bits`
  int order_bits;
};

// A thread owns one row and looks its neighbours up; a warp's 32 rows are collected in shared memory (up to
// 32 offsets at a time), where absent entries are pre-filled, so that only neighbours that exist cost an
// entry, and leave it as full 16-byte-per-lane stores (row-major) and coalesced columns.
// BWD = false: the rows of a submanifold layer, and `table` holds the same cells.
// BWD = true: the input rows of a strided or transposed layer, and `table` holds the output cells (rows from
// n_limit on are cut).  The output side's tables are made by the same pass, by scattering: an input reaches at
// most 8 of 27 offsets' outputs of a k3 s2 layer, and they are bits of the output bitmap that also numbers
// them, so the input cells need no table at all.  Gathering (every output row looks its 27 input cells up)
// took 350 us for 480 k -> 1.36 M rows and an input hash table; clearing 152 MB and scattering 1.6 M pairs
// takes 73.
//
// The row's kl offsets along the last axis meet cells that lie close together in the occupancy bitmap: one
// (at a word boundary two) loads test all of them, and one prefix load numbers all of them, since the prefix
// of the next word is this word's prefix plus its population count.  Three such lines are requested together:
// the kernel waits on L2 latency otherwise.  A submanifold or strided k3 layer so has 9 + 9 loads in flight in
// three rounds instead of 27 probes of a hash table.
constexpr int kLines = 3;
constexpr int kBucketSlots = 512;  // of the CTA's own bucket counts: at most 256 distinct buckets

__host__ __device__ __forceinline__ int fill_pitch(int kvp) {
  // row pitch of the shared tile in entries: 4 mod 8, so that a warp's rows start in eight different bank groups
  const int w = kvp < 32 ? kvp : 32;
  return (w & 7) == 4 ? w : w + 4;
}

__device__ __forceinline__ void clear_buckets(int* slot_bucket, uint32_t* slot_count) {
  for (int i = threadIdx.x; i < kBucketSlots; i += kThreads) {
    slot_bucket[i] = -1;
    slot_count[i] = 0;
  }
  __syncthreads();
}
// Rows per bucket (-1: no row), by all threads of a CTA: first inside the warp, then inside the CTA, so that a
// bucket most rows fall into is one global addition per CTA.
__device__ __forceinline__ void count_buckets(int bucket, int* slot_bucket, uint32_t* slot_count, uint32_t* counts) {
  const unsigned same = __match_any_sync(0xffffffffu, bucket);
  if (bucket >= 0 && __ffs(same) - 1 == static_cast<int>(threadIdx.x & 31)) {
    uint32_t s = (static_cast<uint32_t>(bucket) * 2654435761u) >> 23;
    for (int probe = 0; probe < kBucketSlots; ++probe) {
      const int old = atomicCAS(&slot_bucket[s], -1, bucket);
      if (old == -1 || old == bucket) {
        atomicAdd(&slot_count[s], static_cast<uint32_t>(__popc(same)));
        break;
      }
      s = (s + 1) & (kBucketSlots - 1);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kBucketSlots; i += kThreads)
    if (slot_bucket[i] >= 0) atomicAdd(&counts[slot_bucket[i]], slot_count[i]);
}

// Looks a row's K^ND neighbours up.  The offsets of the last two axes are known at compile time, so that
// the loads of K lines (bitmap) or of their K * K cells (hash table) are requested together: the kernel waits
// on L2 latency otherwise (32 us for 2 000 rows with one line at a time).  The first of three axes stays a
// loop, and a hash chain is followed in a loop of its own: unrolled completely the code no longer fits the
// instruction cache, and on few rows fetching it is what takes the time (20 us for the same rows).
//
// A plane is the K * K offsets of the last two axes; one call looks a slab of planes up, at most 32 offsets,
// which is what the shared tile holds: all of a 3x3x3 kernel, a plane of a 5x5x5 one, 27 of 81 in four dimensions.
template <int ND, int K>
struct Cube {
  static constexpr int plane = ND == 1 ? K : K * K;
  static constexpr int planes = ND <= 2 ? 1 : ND == 3 ? K : K * K;
  static constexpr int together = plane * planes <= 32 ? planes : plane * K <= 32 ? K : 1;  // planes of a slab
  static constexpr int slab = plane * together;
};
template <int ND, bool K64, int K, typename Emit>
__device__ __forceinline__ void look_up_cube(const Geo& g, bool div, const int* own, const int* limit,
                                             const Table<K64>& table, int first_plane, const Emit& emit) {
  using key_t = typename Table<K64>::key_t;
  constexpr int kLast = ND - 1, kMid = ND >= 2 ? ND - 2 : 0;
  constexpr int kLinesHere = ND == 1 ? 1 : K;
  int xm[K], xl[K];
  int lo = INT_MAX, hi = -1;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    xm[k] = ND >= 2 ? axis_cell(g, div, kMid, own[kMid + 1], k, limit[kMid]) : 0;
    xl[k] = axis_cell(g, div, kLast, own[kLast + 1], k, limit[kLast]);
    if (xl[k] >= 0) {
      lo = min(lo, xl[k]);
      hi = max(hi, xl[k]);
    }
  }
  if (hi < 0) return;
  const uint32_t* bits = dense_bits(table);
  const uint32_t* prefix = dense_prefix(table);
  const int32_t* perm = row_permutation(table);
#pragma unroll 1
  for (int p = first_plane; p < first_plane + Cube<ND, K>::together; ++p) {
    key_t lead = static_cast<key_t>(own[0]);
    if (ND == 4) {
      const int x0 = axis_cell(g, div, 0, own[1], p / K, limit[0]);
      if (x0 < 0) continue;
      lead = lead * static_cast<key_t>(limit[0]) + static_cast<key_t>(x0);
    }
    if (ND >= 3) {
      constexpr int kAxis = ND >= 3 ? ND - 3 : 0;
      const int x0 = axis_cell(g, div, kAxis, own[kAxis + 1], p % K, limit[kAxis]);
      if (x0 < 0) continue;
      lead = lead * static_cast<key_t>(limit[kAxis]) + static_cast<key_t>(x0);
    }
    const int k0 = p * Cube<ND, K>::plane;
    key_t base[kLinesHere];
#pragma unroll
    for (int l = 0; l < kLinesHere; ++l)
      base[l] = (ND >= 2 ? lead * static_cast<key_t>(limit[kMid]) + static_cast<key_t>(xm[l]) : lead) * static_cast<key_t>(limit[kLast]);
    if (bits != nullptr) {
      uint32_t w0[kLinesHere], w1[kLinesHere], before[kLinesHere], hits[kLinesHere];
#pragma unroll
      for (int l = 0; l < kLinesHere; ++l) {
        const key_t at = base[l] + static_cast<key_t>(lo);
        w0[l] = xm[l] >= 0 ? __ldg(&bits[at >> 5]) : 0u;
        w1[l] = xm[l] >= 0 && static_cast<int>(at & 31) + hi - lo >= 32 ? __ldg(&bits[(at >> 5) + 1]) : 0u;
      }
#pragma unroll
      for (int l = 0; l < kLinesHere; ++l) {
        const key_t at = base[l] + static_cast<key_t>(lo);
        const unsigned long long win = ((static_cast<unsigned long long>(w1[l]) << 32) | w0[l]) >> (at & 31);
        hits[l] = 0;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (xl[k] >= 0) hits[l] |= static_cast<uint32_t>((win >> (xl[k] - lo)) & 1ull) << k;
        // (a word without bits has no prefix: the second word's rows then come first)
        before[l] = hits[l] != 0 ? __ldg(&prefix[(at >> 5) + (w0[l] == 0 ? 1 : 0)]) : 0u;
      }
      int row[kLinesHere * K];
#pragma unroll
      for (int l = 0; l < kLinesHere; ++l) {
        const int sh = static_cast<int>((base[l] + static_cast<key_t>(lo)) & 31);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          int j = -1;
          if ((hits[l] >> k) & 1u) {
            const int bit = sh + xl[k] - lo;
            j = static_cast<int>(before[l]) + (bit < 32 ? __popc(w0[l] & ((1u << bit) - 1u))
                                                        : __popc(w0[l]) + __popc(w1[l] & ((1u << (bit - 32)) - 1u)));
            if (perm != nullptr) j = __ldg(&perm[j]);
          }
          row[l * K + k] = j;
        }
      }
#pragma unroll
      for (int q = 0; q < kLinesHere * K; ++q) emit(k0 + q, row[q]);
    } else {
      unsigned long long probe[kLinesHere * K];
      uint32_t far = 0;  // cells whose home slot holds another key
#pragma unroll
      for (int l = 0; l < kLinesHere; ++l)
#pragma unroll
        for (int k = 0; k < K; ++k)
          probe[l * K + k] = xm[l] >= 0 && xl[k] >= 0 ? table.first_probe(base[l] + static_cast<key_t>(xl[k])) : Table<K64>::kEmpty;
#pragma unroll
      for (int l = 0; l < kLinesHere; ++l)
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int q = l * K + k;
          int j;
          const bool taken = probe[q] != Table<K64>::kEmpty;
          const bool own_key = table.settled(base[l] + static_cast<key_t>(xl[k]), probe[q], &j) && taken;
          emit(k0 + q, own_key ? j : -1);
          far |= static_cast<uint32_t>(taken && !own_key) << q;
        }
#pragma unroll 1
      for (; far != 0; far &= far - 1) {
        const int q = __ffs(far) - 1, l = q / K, k = q % K;
        const key_t line = ND >= 2 ? lead * static_cast<key_t>(limit[kMid]) + static_cast<key_t>(axis_cell(g, div, kMid, own[kMid + 1], l, limit[kMid])) : lead;
        emit(k0 + q, table.find(line * static_cast<key_t>(limit[kLast]) +
                                static_cast<key_t>(axis_cell(g, div, kLast, own[kLast + 1], k, limit[kLast]))));
      }
    }
  }
}

template <int ND, bool K64, bool BWD, int K>
__global__ void __launch_bounds__(kThreads)
fill_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ idx, long long n, long long n_limit, Table<K64> table,
            const __grid_constant__ FillOut out, int mic, int kvp) {
  using key_t = typename Table<K64>::key_t;
  extern __shared__ __align__(16) int32_t fill_s[];
  __shared__ int slot_bucket[kBucketSlots];
  __shared__ uint32_t slot_count[kBucketSlots];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pitch = fill_pitch(kvp);
  int32_t* tile = fill_s + warp * 32 * pitch;
  int32_t* mine = tile + lane * pitch;
  if (out.counts != nullptr) clear_buckets(slot_bucket, slot_count);
  const long long r = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  const long long row0 = r - lane;
  const bool live = r < n;
  const bool div = BWD && !g.transpose;
  const int* __restrict__ limit = BWD ? g.out_shape : g.in_shape;

  int own[ND + 1];
  bool ok = live;  // a row outside the grid gets no neighbours
  if (live) {
    load_coord<ND>(idx, r, own);
    ok = coord_in_grid<ND>(g, own);
    if (out.iota != nullptr) out.iota[r] = static_cast<int32_t>(r);
  }
  uint32_t valid[ND];  // per axis: the offsets that meet a cell of the grid
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    uint32_t m = 0;
    if (K == 0 && ok && g.axes_fit)
      for (int k = 0; k < g.ksize[d]; ++k)
        m |= static_cast<uint32_t>(axis_cell(g, div, d, own[d + 1], k, limit[d]) >= 0) << k;
    valid[d] = m;
  }
  const uint32_t* bits = dense_bits(table);
  const uint32_t* prefix = dense_prefix(table);
  const int32_t* perm = row_permutation(table);
  const int kl = g.ksize[ND - 1];
  const int q_lo = valid[ND - 1] ? __ffs(valid[ND - 1]) - 1 : 0;
  const int q_hi = valid[ND - 1] ? 31 - __clz(valid[ND - 1]) : -1;
  // lowest and highest cell of a line of offsets along the last axis
  int x_lo = 0, x_span = 0;
  if (q_hi >= 0) {
    const int xa = axis_cell(g, div, ND - 1, own[ND], q_lo, limit[ND - 1]);
    const int xb = axis_cell(g, div, ND - 1, own[ND], q_hi, limit[ND - 1]);
    x_lo = xa < xb ? xa : xb;
    x_span = (xa < xb ? xb : xa) - x_lo;
  }
  uint32_t order_word = 0;
  constexpr int kPiece = K == 0 ? 32 : Cube<ND, K == 0 ? 1 : K>::slab;  // offsets looked up and written at a time
  // (the pieces of a large kernel are dealt over grid.y: a few thousand rows fill the chip only together with them)
  for (int c0 = static_cast<int>(blockIdx.y) * kPiece; c0 < g.kv; c0 += kPiece * static_cast<int>(gridDim.y)) {
    const int width = min(32, kvp - c0);           // entries of a row in this piece, a multiple of four
    const int c1 = min(g.kv, c0 + kPiece);
    __syncwarp();  // the previous piece has been copied out
    {
      const int4 none = make_int4(-1, -1, -1, -1);
      for (int i = lane; i < 8 * pitch; i += 32) reinterpret_cast<int4*>(tile)[i] = none;
    }
    __syncwarp();
    uint32_t word = 0;
    auto emit = [&](int k, int j) {
      if constexpr (K != 0 && !BWD) {
        // every entry is stored, absent ones too: no branch, so the lanes of a warp stay together
        mine[k - c0] = j;
        word |= static_cast<uint32_t>(j >= 0) << (k - c0);
      } else {
        if ((K == 0 && (k < c0 || k >= c1)) || j < 0 || (BWD && j >= n_limit)) return;
        mine[k - c0] = j;
        word |= 1u << (k - c0);
        if (BWD && out.out_rm != nullptr)
          atomicMin(reinterpret_cast<unsigned*>(&out.out_rm[static_cast<long long>(j) * kvp + k]), static_cast<unsigned>(r));
        if (BWD && out.out_cm != nullptr)
          atomicMin(reinterpret_cast<unsigned*>(&out.out_cm[k * n_limit + j]), static_cast<unsigned>(r));
        if (BWD && out.out_words != nullptr)
          atomicOr(&out.out_words[static_cast<long long>(j) * mic + (k >> 5)], 1u << (out.order_bits ? g.key_pos[k] : (k & 31)));
      }
    };
    if constexpr (K != 0) {
      if (ok) look_up_cube<ND, K64, K>(g, div, own, limit, table, c0 / Cube<ND, K>::plane, emit);
    } else if (ok && g.axes_fit && q_hi >= 0) {
      int pos[ND];  // offsets of the leading axes
      const int l0 = c0 / kl, l1 = (c1 - 1) / kl;
      {
        int rest = l0;
#pragma unroll
        for (int d = ND - 2; d >= 0; --d) {
          pos[d] = rest % g.ksize[d];
          rest /= g.ksize[d];
        }
      }
      for (int l = l0; l <= l1; l += kLines) {
        bool on[kLines];
        key_t base[kLines];
#pragma unroll
        for (int b = 0; b < kLines; ++b) {
          on[b] = l + b <= l1;
          key_t key = static_cast<key_t>(own[0]);
#pragma unroll
          for (int d = 0; d < ND - 1; ++d) {
            on[b] = on[b] && ((valid[d] >> pos[d]) & 1u);
            const int x = on[b] ? axis_cell(g, div, d, own[d + 1], pos[d], limit[d]) : 0;
            key = key * static_cast<key_t>(limit[d]) + static_cast<key_t>(x);
          }
          base[b] = key * static_cast<key_t>(limit[ND - 1]);
          // next line
          bool carry = true;
#pragma unroll
          for (int d = ND - 2; d >= 0; --d) {
            if (carry) {
              carry = ++pos[d] == g.ksize[d];
              if (carry) pos[d] = 0;
            }
          }
        }
        if (bits != nullptr && g.window) {
          uint32_t w0[kLines], w1[kLines], hits[kLines], before[kLines];
#pragma unroll
          for (int b = 0; b < kLines; ++b) {
            w0[b] = w1[b] = 0;
            if (on[b]) {
              const key_t at = base[b] + static_cast<key_t>(x_lo);
              w0[b] = __ldg(&bits[at >> 5]);
              if (static_cast<int>(at & 31) + x_span >= 32) w1[b] = __ldg(&bits[(at >> 5) + 1]);
            }
          }
#pragma unroll
          for (int b = 0; b < kLines; ++b) {
            hits[b] = before[b] = 0;
            const key_t at = base[b] + static_cast<key_t>(x_lo);
            if ((w0[b] | w1[b]) != 0) {
              const unsigned long long win = ((static_cast<unsigned long long>(w1[b]) << 32) | w0[b]) >> (at & 31);
              for (uint32_t m = valid[ND - 1]; m != 0; m &= m - 1) {
                const int q = __ffs(m) - 1;
                const int x = axis_cell(g, div, ND - 1, own[ND], q, limit[ND - 1]) - x_lo;
                hits[b] |= static_cast<uint32_t>((win >> x) & 1ull) << q;
              }
              // (a word without bits has no prefix: the second word's rows then come first)
              if (hits[b] != 0) before[b] = __ldg(&prefix[(at >> 5) + (w0[b] == 0 ? 1 : 0)]);
            }
          }
#pragma unroll
          for (int b = 0; b < kLines; ++b) {
            const int sh = static_cast<int>((base[b] + static_cast<key_t>(x_lo)) & 31);
            for (uint32_t m = hits[b]; m != 0; m &= m - 1) {
              const int q = __ffs(m) - 1;
              const int bit = sh + axis_cell(g, div, ND - 1, own[ND], q, limit[ND - 1]) - x_lo;
              int j = static_cast<int>(before[b]) +
                      (bit < 32 ? __popc(w0[b] & ((1u << bit) - 1u)) : __popc(w0[b]) + __popc(w1[b] & ((1u << (bit - 32)) - 1u)));
              if (perm != nullptr) j = __ldg(&perm[j]);
              emit((l + b) * kl + q, j);
            }
          }
        } else {
          // hash table (or cells too far apart for a window): up to three probes in flight
#pragma unroll
          for (int b = 0; b < kLines; ++b) {
            if (!on[b]) continue;
            uint32_t m = valid[ND - 1];
            while (m != 0) {
              key_t key[3];
              int q[3];
              unsigned long long probe[3];
#pragma unroll
              for (int u = 0; u < 3; ++u) {
                q[u] = m != 0 ? __ffs(m) - 1 : -1;
                m &= m - 1;
                probe[u] = 0;
                if (q[u] >= 0) {
                  key[u] = base[b] + static_cast<key_t>(axis_cell(g, div, ND - 1, own[ND], q[u], limit[ND - 1]));
                  if (bits == nullptr) probe[u] = table.first_probe(key[u]);
                }
              }
#pragma unroll
              for (int u = 0; u < 3; ++u)
                if (q[u] >= 0) emit((l + b) * kl + q[u], bits == nullptr ? table.finish(key[u], probe[u]) : table.find(key[u]));
            }
          }
        }
      }
    } else if (ok && !g.axes_fit) {
      // an axis of more than 32 offsets: one offset after the other
      Odometer<ND> od;
      od.set(g, c0);
      for (int k = c0; k < c1; ++k) {
        long long key = own[0];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const int x = axis_cell(g, div, d, own[d + 1], od.pos[d], limit[d]);
          key = key < 0 || x < 0 ? -1 : key * limit[d] + x;
        }
        if (key >= 0) emit(k, table.find(static_cast<key_t>(key)));
        od.next(g);
      }
    }
    if (live && out.words != nullptr) out.words[r * mic + (c0 >> 5)] = word;
    if (out.keys != nullptr)  // (one piece)
      for (uint32_t m = word; m != 0; m &= m - 1) order_word |= 1u << g.key_pos[__ffs(m) - 1];
    __syncwarp();
    const int rows = static_cast<int>(n - row0 < 32 ? (n - row0 > 0 ? n - row0 : 0) : 32);
    if (out.rm != nullptr) {
      const int quads = width / 4;
      if (kPiece != 32 && g.kv > kPiece) {
        // pieces that do not start at multiples of four entries: a row's are written by consecutive lanes
        for (int row = 0; row < rows; ++row)
          if (lane < c1 - c0) out.rm[(row0 + row) * kvp + c0 + lane] = tile[row * pitch + lane];
        if (c1 == g.kv && live)
          for (int k = g.kv; k < kvp; ++k) out.rm[r * kvp + k] = -1;
      } else if (pitch == kvp) {
        int4* dst = reinterpret_cast<int4*>(out.rm + row0 * kvp);
        for (int i = lane; i < rows * quads; i += 32) dst[i] = reinterpret_cast<const int4*>(tile)[i];
      } else {
        for (int i = lane; i < rows * quads; i += 32) {
          const int row = i / quads, q = i - row * quads;
          *reinterpret_cast<int4*>(out.rm + (row0 + row) * kvp + c0 + 4 * q) =
              *reinterpret_cast<const int4*>(tile + row * pitch + 4 * q);
        }
      }
    }
    if (out.rm_rev != nullptr) {
      for (int row = 0; row < rows; ++row)
        if (lane < c1 - c0) out.rm_rev[(row0 + row) * kvp + g.kv - 1 - (c0 + lane)] = tile[row * pitch + lane];
      if (c1 == g.kv && live)
        for (int k = g.kv; k < kvp; ++k) out.rm_rev[r * kvp + k] = -1;
    }
    if (live) {
      if (out.cm != nullptr)
        for (int k = c0; k < c1; ++k) out.cm[static_cast<long long>(k) * n + r] = mine[k - c0];
      if (out.cm_rev != nullptr)
        for (int k = c0; k < c1; ++k) out.cm_rev[static_cast<long long>(g.kv - 1 - k) * n + r] = mine[k - c0];
    }
  }
  if (out.keys == nullptr) return;
  if (live) out.keys[r] = gray_decode(order_word);
  if (out.counts != nullptr) count_buckets(live ? bucket_of(order_word) : -1, slot_bucket, slot_count, out.counts);
}

// The output rows of a strided or transposed layer, after the scatter: their coordinates and, from the
// scattered tile-order words, the keys and bucket counts of their order.
template <int ND, bool K64>
__global__ void __launch_bounds__(kThreads)
finish_outputs_kernel(const __grid_constant__ Geo g, const typename Table<K64>::key_t* __restrict__ sorted, long long n,
                      int32_t* __restrict__ out_indices, int32_t* __restrict__ iota, const uint32_t* __restrict__ order_words,
                      uint32_t* __restrict__ keys, uint32_t* __restrict__ counts) {
  using key_t = typename Table<K64>::key_t;
  __shared__ int slot_bucket[kBucketSlots];
  __shared__ uint32_t slot_count[kBucketSlots];
  if (counts != nullptr) clear_buckets(slot_bucket, slot_count);
  const long long r = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  const bool live = r < n;
  if (live && out_indices != nullptr) {
    int o[ND + 1];
    key_t lin = sorted[r];
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      const key_t q = lin / static_cast<key_t>(g.out_shape[d]);
      o[d + 1] = static_cast<int>(lin - q * static_cast<key_t>(g.out_shape[d]));
      lin = q;
    }
    o[0] = static_cast<int>(lin);
    if (ND == 3 && (reinterpret_cast<uintptr_t>(out_indices) & 15u) == 0) {
      reinterpret_cast<int4*>(out_indices)[r] = make_int4(o[0], o[1], o[ND > 1 ? 2 : 0], o[ND > 2 ? 3 : 0]);
    } else {
#pragma unroll
      for (int d = 0; d <= ND; ++d) out_indices[r * (ND + 1) + d] = o[d];
    }
  }
  if (live && iota != nullptr) iota[r] = static_cast<int32_t>(r);
  if (order_words == nullptr) return;
  const uint32_t word = live ? order_words[r] : 0u;
  if (live) keys[r] = gray_decode(word);
  if (counts != nullptr) count_buckets(live ? bucket_of(word) : -1, slot_bucket, slot_count, counts);
}

// The keys of the order from a finished row-major table, as the fill makes them on its way.
__global__ void __launch_bounds__(kThreads)
rowmajor_keys_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ rm, int kvp, long long n, uint32_t* __restrict__ keys) {
  const long long r = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (r >= n) return;
  uint32_t word = 0;
  for (int k = 0; k < g.kv; ++k) word |= (__ldg(&rm[r * kvp + k]) >= 0 ? 1u : 0u) << g.key_pos[k];
  keys[r] = gray_decode(word);
}

// keys[i] = words[rows[i], w] & and_mask ; rows == nullptr means identity.
__global__ void __launch_bounds__(kThreads)
gather_mask_word_kernel(const uint32_t* __restrict__ words, const int32_t* __restrict__ rows,
                        long long n, int mic, int w, uint32_t and_mask, uint32_t* __restrict__ keys,
                        int32_t* __restrict__ iota) {
  const long long i = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (i >= n) return;
  const long long row = rows ? rows[i] : i;
  keys[i] = words[row * mic + w] & and_mask;
  if (iota) iota[i] = static_cast<int32_t>(i);
}

// mask_out[i, w] = words[rows[i], w] (word 0 ANDed with and_mask); argsort_out[i] = rows[i].
__global__ void __launch_bounds__(kThreads)
emit_sorted_masks_kernel(const uint32_t* __restrict__ words, const int32_t* __restrict__ rows,
                         long long n, int mic, uint32_t and_mask, int32_t* __restrict__ mask_out,
                         int32_t* __restrict__ argsort_out) {
  const long long i = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (i >= n) return;
  const long long row = rows ? rows[i] : i;
  for (int w = 0; w < mic; ++w) {
    uint32_t v = words[row * mic + w];
    if (w == 0) v &= and_mask;
    mask_out[i * mic + w] = static_cast<int32_t>(v);
  }
  argsort_out[i] = static_cast<int32_t>(row);
}

// ------------------------------------------------------------------------
// Phase 2 kernels (Native format): per offset, a stable compaction of the
// contributing input rows.  Grid = (row blocks, kv).
// ------------------------------------------------------------------------
template <int ND, bool K64>
__device__ __forceinline__ int native_out_row(const Geo& g, const int32_t* __restrict__ idx,
                                              long long j, int k, long long n_out,
                                              const Table<K64>& lookup) {
  using key_t = typename Table<K64>::key_t;
  int c[ND + 1];
  load_coord<ND>(idx, j, c);
  if (!coord_in_grid<ND>(g, c)) return -1;
  Odometer<ND> od;
  od.set(g, k);
  const long long key = out_key_from_input<ND>(g, c, od.pos);
  if (key < 0) return -1;
  const int r = lookup.find(static_cast<key_t>(key));
  return (r >= n_out) ? -1 : r;
}

template <int ND, bool K64>
__global__ void __launch_bounds__(kThreads)
native_count_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ idx, long long n_in,
                    long long n_out, Table<K64> lookup, int* __restrict__ block_counts) {
  const long long j = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  const int k = blockIdx.y;
  const int ok = (j < n_in) && native_out_row<ND, K64>(g, idx, j, k, n_out, lookup) >= 0;
  const int total = __syncthreads_count(ok);
  if (threadIdx.x == 0) block_counts[static_cast<long long>(k) * gridDim.x + blockIdx.x] = total;
}

// One block per offset: exclusive scan of that offset's block counts (in place)
// and the per-offset total.
__global__ void __launch_bounds__(kThreads)
native_scan_kernel(int* __restrict__ block_counts, int n_blocks, int32_t* __restrict__ npl, int kv,
                   int subm) {
  __shared__ int warp_sums[kThreads / 32];
  __shared__ int carry;
  const int k = blockIdx.x;
  int* row = block_counts + static_cast<long long>(k) * n_blocks;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n_blocks; base += kThreads) {
    const int i = base + threadIdx.x;
    const int v = i < n_blocks ? row[i] : 0;
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, off);
      if ((threadIdx.x & 31) >= off) incl += t;
    }
    if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = incl;
    __syncthreads();
    int warp_off = 0;
    for (int w = 0; w < (threadIdx.x >> 5); ++w) warp_off += warp_sums[w];
    const int excl = carry + warp_off + incl - v;
    if (i < n_blocks) row[i] = excl;
    __syncthreads();
    if (threadIdx.x == kThreads - 1) carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    // subm: counts are reported only for offsets before the centre
    // (spconv_triton/pytorch/_impl/pairs.py:269-277); the pair content is still complete.
    npl[k] = (subm && k >= kv / 2) ? 0 : carry;
  }
}

template <int ND, bool K64>
__global__ void __launch_bounds__(kThreads)
native_write_kernel(const __grid_constant__ Geo g, const int32_t* __restrict__ idx, long long n_in,
                    long long n_out, Table<K64> lookup, const int* __restrict__ block_offsets,
                    int32_t* __restrict__ pair) {
  __shared__ int warp_sums[kThreads / 32];
  const long long j = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  const int k = blockIdx.y;
  const int r = (j < n_in) ? native_out_row<ND, K64>(g, idx, j, k, n_out, lookup) : -1;
  const unsigned ballot = __ballot_sync(0xffffffffu, r >= 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) warp_sums[warp] = __popc(ballot);
  __syncthreads();
  if (r >= 0) {
    int pos = block_offsets[static_cast<long long>(k) * gridDim.x + blockIdx.x];
    for (int w = 0; w < warp; ++w) pos += warp_sums[w];
    pos += __popc(ballot & ((1u << lane) - 1u));
    pair[static_cast<long long>(k) * n_in + pos] = static_cast<int32_t>(j);
    pair[(static_cast<long long>(g.kv) + k) * n_in + pos] = r;
  }
}

// out[row, 4q..4q+3] = pairs[4q..4q+3, row]; one thread per (row, q), q fastest, so
// that the 16-byte stores of a row are contiguous.
__global__ void __launch_bounds__(kThreads)
pairs_to_rowmajor_kernel(const int32_t* __restrict__ pairs, int kv, int kvp, long long n,
                         int32_t* __restrict__ out) {
  const long long e = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  const int quads = kvp / 4;
  const long long row = e / quads;
  if (row >= n) return;
  const int k0 = static_cast<int>(e % quads) * 4;
  int v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = (k0 + u < kv) ? __ldg(&pairs[static_cast<long long>(k0 + u) * n + row]) : -1;
  *reinterpret_cast<int4*>(&out[row * kvp + k0]) = make_int4(v[0], v[1], v[2], v[3]);
}

// 32 x 32 entries through shared memory: both sides are read and written in full rows.
__global__ void __launch_bounds__(kThreads)
rowmajor_to_pairs_kernel(const int32_t* __restrict__ rowmajor, int kv, int kvp, long long n, int32_t* __restrict__ pairs) {
  __shared__ int32_t tile[32][33];
  const long long row0 = blockIdx.x * 32ll;
  const int k0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (row0 + r < n && k0 + threadIdx.x < kv) tile[r][threadIdx.x] = rowmajor[(row0 + r) * kvp + k0 + threadIdx.x];
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8)
    if (row0 + threadIdx.x < n && k0 + k < kv) pairs[static_cast<long long>(k0 + k) * n + row0 + threadIdx.x] = tile[threadIdx.x][k];
}

__global__ void __launch_bounds__(kThreads)
native_to_tables_kernel(const int32_t* __restrict__ pair_in, const int32_t* __restrict__ pair_out,
                        int kv, long long n_pair, int32_t* __restrict__ pair_fwd, long long n_out,
                        int32_t* __restrict__ pair_bwd, long long n_in) {
  const long long p = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  const int k = blockIdx.y;
  if (p >= n_pair) return;
  const int i = pair_in[static_cast<long long>(k) * n_pair + p];
  const int o = pair_out[static_cast<long long>(k) * n_pair + p];
  if (i < 0 || o < 0) return;
  if (o < n_out) pair_fwd[static_cast<long long>(k) * n_out + o] = i;
  if (pair_bwd != nullptr && i < n_in) pair_bwd[static_cast<long long>(k) * n_in + i] = o;
}

// ------------------------------------------------------------------------
// Host side: workspace layout
// ------------------------------------------------------------------------
struct Layout {
  bool k64;
  int key_bits;
  int mic;
  int64_t bound;  // upper bound on n_out
  // Occupancy bitmaps (words; 0 = that side uses a hash table): the output side of a strided layer is
  // numbered and looked up through its bitmap, the input side looked up.
  int64_t ibits_words = 0, obits_words = 0;
  size_t off_ibits = 0, off_iprefix = 0, off_istarts = 0, off_perm = 0;
  size_t off_obits = 0, off_oprefix = 0, off_ostarts = 0;
  uint32_t cap_in, cap_out;
  int64_t n_blocks_native;
  size_t off_counters, off_tin, off_tin_vals, off_tout, off_tout_vals, off_uniq, off_sorted;
  size_t off_words, off_keys_a, off_keys_b, off_vals_a, off_vals_b, off_cub, off_native;
  size_t off_order_pairs, off_order_counts;
  size_t cub_bytes, total;
  // Chained rulebooks: the input rows are exactly the output rows of an earlier strided layer whose
  // output bitmap and prefix (in ITS workspace) then serve as this layer's input bitmap; rows are
  // ranks by construction, and no input hash table is built.
  const uint32_t* shared_bits = nullptr;
  const uint32_t* shared_prefix = nullptr;
  const uint32_t* shared_cells = nullptr;  // the cells of those rows
};
// bucket counts of the tile order (one set for each side of a layer)
constexpr size_t kOrderCountBytes = kTileOrderWords * 4;

inline int cell_blocks(int64_t words) { return static_cast<int>(ceil_div(words, kCellBlock)); }

// Scratch of the library's radix sort for n (key, row) pairs: asked for once per power of two.
size_t radix_sort_bytes(int64_t n, bool keys64) {
  static std::atomic<size_t> known[2][64];
  int e = 0;
  while ((1ll << e) < n) ++e;
  size_t have = known[keys64][e].load(std::memory_order_relaxed);
  if (have != 0) return have;
  const int64_t most = std::min<int64_t>(1ll << e, INT32_MAX);
  size_t keys = 0, pairs = 0;
  if (keys64)
    cub::DeviceRadixSort::SortKeys(nullptr, keys, static_cast<unsigned long long*>(nullptr),
                                   static_cast<unsigned long long*>(nullptr), most);
  else
    cub::DeviceRadixSort::SortKeys(nullptr, keys, static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr), most);
  cub::DeviceRadixSort::SortPairs(nullptr, pairs, static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  static_cast<int32_t*>(nullptr), static_cast<int32_t*>(nullptr), most);
  have = std::max<size_t>(std::max(keys, pairs), 16);
  known[keys64][e].store(have, std::memory_order_relaxed);
  return have;
}

uint32_t pow2_at_least(int64_t v) {
  uint64_t c = 64;
  while (c < static_cast<uint64_t>(v)) c <<= 1;
  return static_cast<uint32_t>(std::min<uint64_t>(c, 1ull << 31));
}

int gcd_int(int a, int b) { return b == 0 ? a : gcd_int(b, a % b); }

bool make_geo(const spc_geometry* s, Geo* g) {
  if (s == nullptr || s->ndim < 1 || s->ndim > SPC_MAX_NDIM || s->batch_size <= 0) return false;
  g->ndim = s->ndim;
  g->batch = s->batch_size;
  g->subm = s->subm != 0;
  g->transpose = (!g->subm) && s->transpose != 0;
  g->kv = 1;
  for (int d = 0; d < SPC_MAX_NDIM; ++d) {
    const bool live = d < s->ndim;
    g->in_shape[d] = live ? s->in_shape[d] : 1;
    g->ksize[d] = live ? s->ksize[d] : 1;
    g->dil[d] = live ? s->dilation[d] : 1;
    if (live && (g->ksize[d] <= 0 || g->in_shape[d] <= 0 || g->dil[d] <= 0)) return false;
    if (g->subm) {
      g->out_shape[d] = g->in_shape[d];
      g->stride[d] = 1;
      g->pad[d] = (g->ksize[d] / 2) * g->dil[d];
    } else {
      g->out_shape[d] = live ? s->out_shape[d] : 1;
      g->stride[d] = live ? s->stride[d] : 1;
      g->pad[d] = live ? s->padding[d] : 0;
      if (live && (g->out_shape[d] <= 0 || g->stride[d] <= 0)) return false;
    }
    g->kv *= g->ksize[d];
  }
  g->axes_fit = 1;
  for (int d = 0; d < SPC_MAX_NDIM; ++d) {
    g->axes_fit = g->axes_fit && g->ksize[d] <= 32;
    g->shift[d] = -1;
    for (int b = 0; b < 31; ++b)
      if (g->stride[d] == (1 << b)) g->shift[d] = b;
  }
  g->window = static_cast<int64_t>(g->ksize[s->ndim - 1] - 1) * g->dil[s->ndim - 1] <= 32;
  for (int k = 0; k < 32; ++k) g->key_pos[k] = static_cast<unsigned char>(k);
  if (g->kv <= 32) {
    // distance of every offset from the kernel's centre (sum over the axes), then positions in
    // ascending distance, ties in offset order
    int dist[32];
    for (int k = 0; k < g->kv; ++k) {
      int rest = k, sum = 0;
      for (int d = g->ndim - 1; d >= 0; --d) {
        const int pos = rest % g->ksize[d];
        rest /= g->ksize[d];
        sum += std::abs(2 * pos - (g->ksize[d] - 1));
      }
      dist[k] = sum;
    }
    for (int k = 0; k < g->kv; ++k) {
      int rank = 0;
      for (int q = 0; q < g->kv; ++q) rank += dist[q] < dist[k] || (dist[q] == dist[k] && q < k);
      g->key_pos[k] = static_cast<unsigned char>(rank);
    }
  }
  return true;
}

Layout make_layout(const Geo& g, int64_t n_in) {
  Layout L{};
  double vol_in = g.batch, vol_out = g.batch;
  for (int d = 0; d < g.ndim; ++d) {
    vol_in *= g.in_shape[d];
    vol_out *= g.out_shape[d];
  }
  const double max_lin = std::max(vol_in, vol_out);
  L.k64 = max_lin >= 2147483648.0;
  L.key_bits = 1;
  while (L.key_bits < 63 && static_cast<double>(1ull << L.key_bits) < max_lin) ++L.key_bits;
  L.mic = (g.kv + 31) / 32;
  double per_input = 1;
  for (int d = 0; d < g.ndim; ++d) {
    int m = g.ksize[d];
    if (!g.transpose && !g.subm && gcd_int(g.dil[d], g.stride[d]) == 1)
      m = (g.ksize[d] + g.stride[d] - 1) / g.stride[d];
    per_input *= m;
  }
  if (g.subm) {
    L.bound = n_in;
  } else {
    const double b = std::min(static_cast<double>(n_in) * per_input, vol_out);
    L.bound = static_cast<int64_t>(std::max(b, 1.0));
  }
  // The rows of a submanifold layer through a bitmap of the grid (most neighbour cells of a voxel are empty, a bit test
  // answers for a whole line of them, and a row is its rank) where the bitmap is no dearer to clear and
  // count than a hash table (512 cells or 64 bytes a voxel), small enough to stay in L2 beside the tables
  // (24 MB), and there are enough rows for the looks-up to outweigh three more launches.
  const double max_bits = 24.0 * 1024 * 1024 * 8;
  if (g.subm && !L.k64 && vol_in <= max_bits && vol_in <= 512.0 * n_in && n_in >= 16384)
    L.ibits_words = static_cast<int64_t>(vol_in / 32.0) + 1;
  // the output bitmap also numbers the outputs, which a hash table needs a sort for
  if (!g.subm && !L.k64 && vol_out <= max_bits) L.obits_words = static_cast<int64_t>(vol_out / 32.0) + 1;
  // Most look-ups miss, so a loaded table costs probe chains, which a warp follows one after the other: a sixteenth
  // full while that is a few MB to clear (2 000 rows: the look-up 17 -> 11 us), a quarter beyond.
  L.cap_in = !g.subm || L.ibits_words ? 0 : pow2_at_least((n_in <= 32768 ? 16 : 4) * n_in);
  L.cap_out = g.subm || L.obits_words ? 0 : pow2_at_least(2 * L.bound);
  const int64_t n_max = std::max<int64_t>(n_in, L.bound);
  L.n_blocks_native = ceil_div(std::max<int64_t>(n_in, 1), kThreads);
  const size_t key_sz = L.k64 ? 8 : 4;
  L.cub_bytes = radix_sort_bytes(n_max, L.k64);

  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  L.off_counters = take(256);
  L.off_tin = take(static_cast<size_t>(L.cap_in) * 8);
  L.off_tin_vals = take(L.k64 ? static_cast<size_t>(L.cap_in) * 4 : 0);
  L.off_tout = take(static_cast<size_t>(L.cap_out) * 8);
  L.off_tout_vals = take(L.k64 ? static_cast<size_t>(L.cap_out) * 4 : 0);
  L.off_uniq = take(g.subm ? 0 : static_cast<size_t>(L.bound) * key_sz);
  L.off_sorted = take(g.subm ? 0 : static_cast<size_t>(L.bound) * key_sz);
  L.off_words = take(static_cast<size_t>(n_max) * L.mic * 4);
  L.off_keys_a = take(static_cast<size_t>(n_max) * 4);
  L.off_keys_b = take(static_cast<size_t>(n_max) * 4);
  L.off_vals_a = take(static_cast<size_t>(n_max) * 4);
  L.off_vals_b = take(static_cast<size_t>(n_max) * 4);
  L.off_cub = take(L.cub_bytes);
  L.off_native = take(static_cast<size_t>(L.n_blocks_native) * g.kv * 4);
  L.off_order_pairs = take(g.kv <= 32 ? static_cast<size_t>(n_max) * 8 : 0);
  L.off_order_counts = take(2 * kOrderCountBytes);
  L.off_ibits = take(static_cast<size_t>(L.ibits_words) * 4);
  L.off_iprefix = take(static_cast<size_t>(L.ibits_words) * 4);
  L.off_istarts = take(L.ibits_words ? static_cast<size_t>(cell_blocks(L.ibits_words) + 1) * 4 : 0);
  L.off_perm = take(L.ibits_words ? static_cast<size_t>(n_in) * 4 : 0);
  L.off_obits = take(static_cast<size_t>(L.obits_words) * 4);
  L.off_oprefix = take(static_cast<size_t>(L.obits_words) * 4);
  L.off_ostarts = take(L.obits_words ? static_cast<size_t>(cell_blocks(L.obits_words) + 1) * 4 : 0);
  L.total = off;
  return L;
}

template <bool K64>
Table<K64> table_at(char* ws, size_t off_slots, size_t off_vals, uint32_t cap);
template <>
Table<false> table_at<false>(char* ws, size_t off_slots, size_t, uint32_t cap) {
  Table<false> t;
  t.slots = reinterpret_cast<unsigned long long*>(ws + off_slots);
  t.cap_mask = cap ? cap - 1 : 0;
  return t;
}
template <>
Table<true> table_at<true>(char* ws, size_t off_slots, size_t off_vals, uint32_t cap) {
  Table<true> t;
  t.slots = reinterpret_cast<unsigned long long*>(ws + off_slots);
  t.vals = reinterpret_cast<int*>(ws + off_vals);
  t.cap_mask = cap ? cap - 1 : 0;
  return t;
}

template <bool K64>
Table<K64> tin_at(char* ws, const Layout& L);
template <>
Table<false> tin_at<false>(char* ws, const Layout& L) {
  Table<false> t = table_at<false>(ws, L.off_tin, L.off_tin_vals, L.cap_in);
  if (L.shared_bits != nullptr) {
    t.obits = const_cast<uint32_t*>(L.shared_bits);
    t.oprefix = L.shared_prefix;
    return t;  // `unsorted` stays null: the rows are the ranks
  }
  if (L.ibits_words) {
    t.obits = reinterpret_cast<uint32_t*>(ws + L.off_ibits);
    t.oprefix = reinterpret_cast<const uint32_t*>(ws + L.off_iprefix);
    t.unsorted = reinterpret_cast<const int*>(ws + L.off_counters) + kUnsorted;
    t.perm = reinterpret_cast<const int32_t*>(ws + L.off_perm);
  }
  return t;
}
template <>
Table<true> tin_at<true>(char* ws, const Layout& L) {
  return table_at<true>(ws, L.off_tin, L.off_tin_vals, L.cap_in);
}

template <bool K64>
Table<K64> tout_at(char* ws, const Layout& L);
template <>
Table<false> tout_at<false>(char* ws, const Layout& L) {
  Table<false> t = table_at<false>(ws, L.off_tout, L.off_tout_vals, L.cap_out);
  if (L.obits_words) {
    t.obits = reinterpret_cast<uint32_t*>(ws + L.off_obits);
    t.oprefix = reinterpret_cast<const uint32_t*>(ws + L.off_oprefix);
  }
  return t;
}
template <>
Table<true> tout_at<true>(char* ws, const Layout& L) {
  return table_at<true>(ws, L.off_tout, L.off_tout_vals, L.cap_out);
}

int launch_clear(const Clear& c, cudaStream_t st) {
  const unsigned blocks = static_cast<unsigned>(std::max<long long>(1, std::min<long long>(ceil_div(c.total, 256), 16ll * sm_count())));
  clear_kernel<<<blocks, 256, 0, st>>>(c);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

inline unsigned blocks_for(int64_t n) { return static_cast<unsigned>(ceil_div(std::max<int64_t>(n, 1), kThreads)); }

// ------------------------------------------------------------------------
// Phase 1
// ------------------------------------------------------------------------
template <int ND, bool K64>
int prepare_impl(const Geo& g, const Layout& L, const int32_t* idx, int64_t n_in, char* ws,
                 int64_t* n_out_host, cudaStream_t st) {
  using key_t = typename Table<K64>::key_t;
  int* counters = reinterpret_cast<int*>(ws + L.off_counters);
  // Submanifold layers return without a host read, so a row outside the grid is also recorded in the
  // device status word, which the host reads at its next synchronisation point.
  int* dev_status = device_status_ptr();
  const bool chained = L.shared_bits != nullptr;  // input bitmap and prefix exist already, no input table
  const bool dense_in = !chained && L.ibits_words != 0, dense_out = L.obits_words != 0;
  Clear clear;
  clear.add(counters, 0, 256);
  if (dense_in) {
    clear.add(ws + L.off_ibits, 0, static_cast<size_t>(L.ibits_words) * 4);
    clear.add(ws + L.off_perm, 0x7F, static_cast<size_t>(n_in) * 4);
  } else if (g.subm && !chained) {
    clear.add(ws + L.off_tin, 0xFF, static_cast<size_t>(L.cap_in) * 8);
    if (K64) clear.add(ws + L.off_tin_vals, 0x7F, static_cast<size_t>(L.cap_in) * 4);
  }
  if (dense_out) {
    clear.add(ws + L.off_obits, 0, static_cast<size_t>(L.obits_words) * 4);
  } else if (!g.subm) {
    clear.add(ws + L.off_tout, 0xFF, static_cast<size_t>(L.cap_out) * 8);
    if (K64) clear.add(ws + L.off_tout_vals, 0x7F, static_cast<size_t>(L.cap_out) * 4);
  }
  clear.add(ws + L.off_order_counts, 0, 2 * kOrderCountBytes);
  int rc = launch_clear(clear, st);
  if (rc != SPC_OK) return rc;
  Table<K64> tin = tin_at<K64>(ws, L);
  Table<K64> tout = tout_at<K64>(ws, L);
  uint32_t* ibits = dense_in ? reinterpret_cast<uint32_t*>(ws + L.off_ibits) : nullptr;
  uint32_t* obits = dense_out ? reinterpret_cast<uint32_t*>(ws + L.off_obits) : nullptr;
  key_t* uniq = reinterpret_cast<key_t*>(ws + L.off_uniq);
  key_t* sorted = reinterpret_cast<key_t*>(ws + L.off_sorted);
  if (!chained || (dense_out && g.axes_fit)) {
    ingest_kernel<ND, K64><<<blocks_for(n_in), kThreads, 0, st>>>(g, idx, L.shared_cells, n_in, tin, g.subm && !chained, ibits,
                                                                  g.axes_fit ? obits : nullptr, counters, dev_status);
    SPC_LAUNCH_OK();
  }
  if (!g.subm && !(dense_out && g.axes_fit)) {
    enumerate_outputs_kernel<ND, K64><<<blocks_for(n_in), kThreads, 0, st>>>(g, idx, n_in, tout, uniq, counters);
    SPC_LAUNCH_OK();
  }
  // The output count reaches the host through a page-locked word that a kernel writes, not through a
  // device-to-host copy: a copy would queue on the copy engine behind whatever transfer the
  // application has in flight (a previous result going back to the host, say) and stall the whole
  // rulebook chain for its duration.
  volatile int* box = nullptr;
  int ticket = 0;
  if (!g.subm) {
    rc = host_mailbox(&box, &ticket);
    if (rc != SPC_OK) return rc;
  }
  if (dense_in || dense_out) {
    Cells c{};
    if (dense_in) {
      c.bits[0] = ibits;
      c.prefix[0] = reinterpret_cast<uint32_t*>(ws + L.off_iprefix);
      c.starts[0] = reinterpret_cast<uint32_t*>(ws + L.off_istarts);
      c.words[0] = L.ibits_words;
      c.blocks[0] = cell_blocks(L.ibits_words);
    }
    if (dense_out) {
      c.bits[1] = obits;
      c.prefix[1] = reinterpret_cast<uint32_t*>(ws + L.off_oprefix);
      c.starts[1] = reinterpret_cast<uint32_t*>(ws + L.off_ostarts);
      c.words[1] = L.obits_words;
      c.blocks[1] = cell_blocks(L.obits_words);
    }
    const unsigned blocks = static_cast<unsigned>(c.blocks[0] + c.blocks[1]);
    count_cells_kernel<<<blocks, kThreads, 0, st>>>(c, counters, dev_status, dense_out ? const_cast<int*>(box) : nullptr, ticket);
    SPC_LAUNCH_OK();
    number_cells_kernel<<<blocks, kThreads, 0, st>>>(c, L.bound, reinterpret_cast<uint32_t*>(sorted));
    SPC_LAUNCH_OK();
    if constexpr (!K64) {
      if (dense_in) {
        permute_rows_kernel<ND><<<blocks_for(n_in), kThreads, 0, st>>>(g, idx, n_in, tin,
                                                                       reinterpret_cast<int32_t*>(ws + L.off_perm));
        SPC_LAUNCH_OK();
      }
    }
  }
  if (g.subm) {
    *n_out_host = n_in;
    return SPC_OK;
  }
  if (!dense_out) {
    publish_counters_kernel<<<1, 32, 0, st>>>(counters, dev_status, const_cast<int*>(box), ticket);
    SPC_LAUNCH_OK();
  }
  rc = wait_for_ticket(box, ticket, st);
  if (rc != SPC_OK) return rc;
  int host[2] = {box[1], box[2]};
  const int sticky = box[3];  // the device status word: a bounded wait of an earlier kernel, or a bad row of an earlier layer
  if (host[kStatus] != 0 || sticky != 0) {
    if (dev_status != nullptr && sticky != 0) SPC_CUDA_OK(cudaMemsetAsync(dev_status, 0, sizeof(int), st));
    const int code = host[kStatus] != 0 ? host[kStatus] : sticky;
    if (code == SPC_ERR_INVALID_ARGUMENT)
      return fail(code, "rulebook: an index row lies outside batch_size / spatial_shape");
    if (code == SPC_ERR_DEVICE_WAIT_EXPIRED)
      return fail(code, "a bounded device-side wait of an earlier kernel expired; its output is incomplete");
    return fail(code, "rulebook: hash table full (status %d)", code);
  }
  const int64_t n_out = host[kUniqueCount];
  *n_out_host = n_out;
  if (n_out == 0) return SPC_OK;
  if (n_out > L.bound) return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "rulebook: %lld outputs exceed bound %lld",
                                   static_cast<long long>(n_out), static_cast<long long>(L.bound));
  if (dense_out) return SPC_OK;  // numbered and listed in ascending order already
  size_t cub_bytes = L.cub_bytes;
  SPC_CUDA_OK(cub::DeviceRadixSort::SortKeys(ws + L.off_cub, cub_bytes, uniq, sorted, n_out, 0,
                                              std::min<int>(L.key_bits, sizeof(key_t) * 8), st));
  assign_ranks_kernel<K64><<<blocks_for(n_out), kThreads, 0, st>>>(tout, sorted, n_out);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

// Sorts the per-row bitmasks (stable, ascending as unsigned, highest word most
// significant) and emits pair_mask / mask_argsort for every split.
// One mask word per row, one split that keeps every bit, sorted: the words are the sort keys as
// they stand and the sort can write pair_mask / mask_argsort itself, if the kernel that produced the
// words also left 0..n-1 in the value scratch (mask_iota()).
bool masks_sort_in_place(const Layout& L, const uint32_t* split_masks, int n_split, int do_sort) {
  return L.mic == 1 && n_split == 1 && do_sort != 0 && split_masks[0] == 0xffffffffu;
}
int32_t* mask_iota(const Layout& L, char* ws, const uint32_t* split_masks, int n_split, int do_sort) {
  return masks_sort_in_place(L, split_masks, n_split, do_sort) ? reinterpret_cast<int32_t*>(ws + L.off_vals_a)
                                                                 : nullptr;
}

int emit_masks(const Layout& L, char* ws, int64_t n, int kv, const uint32_t* split_masks, int n_split,
               int do_sort, int32_t* mask_out, int32_t* argsort_out, cudaStream_t st) {
  const uint32_t* words = reinterpret_cast<const uint32_t*>(ws + L.off_words);
  if (masks_sort_in_place(L, split_masks, n_split, do_sort)) {
    size_t cub_bytes = L.cub_bytes;
    SPC_CUDA_OK(cub::DeviceRadixSort::SortPairs(ws + L.off_cub, cub_bytes, words, reinterpret_cast<uint32_t*>(mask_out),
                                                 reinterpret_cast<const int32_t*>(ws + L.off_vals_a), argsort_out, n, 0,
                                                 std::min(32, kv), st));
    return SPC_OK;
  }
  uint32_t* keys_a = reinterpret_cast<uint32_t*>(ws + L.off_keys_a);
  uint32_t* keys_b = reinterpret_cast<uint32_t*>(ws + L.off_keys_b);
  int32_t* vals_a = reinterpret_cast<int32_t*>(ws + L.off_vals_a);
  int32_t* vals_b = reinterpret_cast<int32_t*>(ws + L.off_vals_b);
  const int mic = L.mic;
  for (int s = 0; s < n_split; ++s) {
    const uint32_t and0 = split_masks[s];
    int32_t* m_out = mask_out + static_cast<int64_t>(s) * n * mic;
    int32_t* a_out = argsort_out + static_cast<int64_t>(s) * n;
    const int32_t* rows = nullptr;
    if (do_sort) {
      int32_t* cur = vals_a;
      int32_t* nxt = vals_b;
      for (int w = 0; w < mic; ++w) {
        const uint32_t andw = (w == 0) ? and0 : 0xffffffffu;
        gather_mask_word_kernel<<<blocks_for(n), kThreads, 0, st>>>(
            words, w == 0 ? nullptr : cur, n, mic, w, andw, keys_a, w == 0 ? cur : nullptr);
        SPC_LAUNCH_OK();
        const int bits = std::min(32, kv - 32 * w);
        size_t cub_bytes = L.cub_bytes;
        SPC_CUDA_OK(cub::DeviceRadixSort::SortPairs(ws + L.off_cub, cub_bytes, keys_a, keys_b, cur, nxt,
                                                     n, 0, bits, st));
        std::swap(cur, nxt);
      }
      rows = cur;
    }
    emit_sorted_masks_kernel<<<blocks_for(n), kThreads, 0, st>>>(words, rows, n, mic, and0, m_out, a_out);
    SPC_LAUNCH_OK();
  }
  return SPC_OK;
}

// Kernel width of a cube-shaped kernel with a fill kernel of its own, else 0.  (The mask words of several
// pieces start at multiples of 32 offsets, which the pieces of these kernels do not.)
int cube_width(const Geo& g, bool words) {
  for (int d = 0; d < g.ndim; ++d)
    if (g.ksize[d] != g.ksize[0] || g.dil[d] != 1) return 0;
  const int k = g.ksize[0];
  if (words && g.kv > 32) return 0;
  return k == 2 || k == 3 || (k == 5 && g.ndim <= 3) ? k : 0;
}
size_t fill_smem_bytes(int kvp) { return static_cast<size_t>(kThreads / 32) * 32 * fill_pitch(kvp) * 4; }

template <int ND, bool K64, bool BWD>
int launch_fill(const Geo& g, const int32_t* idx, int64_t n, int64_t n_limit, const Table<K64>& table, const FillOut& out,
                int mic, cudaStream_t st) {
  const int kvp = (g.kv + 3) & ~3;
  const unsigned blocks = blocks_for(n);
  const size_t smem = fill_smem_bytes(kvp);
  const auto launch = [&](auto width) {
    constexpr int K = decltype(width)::value;
    const int pieces = K == 0 ? 1 : g.kv / Cube<ND, K == 0 ? 1 : K>::slab;
    fill_kernel<ND, K64, BWD, K><<<dim3(blocks, static_cast<unsigned>(pieces)), kThreads, smem, st>>>(g, idx, n, n_limit, table, out, mic, kvp);
  };
  const int width = cube_width(g, out.words != nullptr || out.out_words != nullptr);
  if (width == 3) launch(std::integral_constant<int, 3>{});
  else if (width == 2 && BWD) launch(std::integral_constant<int, BWD ? 2 : 0>{});  // (submanifold kernels are odd)
  else if (ND <= 3 && width == 5) launch(std::integral_constant<int, ND <= 3 ? 5 : 0>{});
  else launch(std::integral_constant<int, 0>{});
  SPC_LAUNCH_OK();
  return SPC_OK;
}

// One side's tables, as the callers ask for them.
struct SideTables {
  int32_t* cm = nullptr;
  int32_t* rm = nullptr;
  int32_t* order = nullptr;        // the tile order, or
  int32_t* mask = nullptr;         // the exactly sorted masks
  int32_t* argsort = nullptr;
  bool wanted() const { return cm || rm || order || mask; }
};
struct MaskSplits {
  const uint32_t* words = nullptr;
  int n = 1, do_sort = 0;
};

// Scratch of the tile order; the input side of a strided layer has keys and counts of its own, so that both
// sides come out of one pass.  The counts are zero after phase 1 and after every order.
uint32_t* order_keys(const Layout& L, char* ws, bool input) {
  return reinterpret_cast<uint32_t*>(ws + (input ? L.off_keys_b : L.off_keys_a));
}
uint32_t* bucket_counts(const Layout& L, char* ws, int64_t n, bool input) {
  return tile_order_needs_buckets(n) ? reinterpret_cast<uint32_t*>(ws + L.off_order_counts + (input ? kOrderCountBytes : 0)) : nullptr;
}
int emit_order(const Layout& L, char* ws, int64_t n, int kv, int32_t* order, bool input, cudaStream_t st) {
  uint32_t* counts = reinterpret_cast<uint32_t*>(ws + L.off_order_counts + (input ? kOrderCountBytes : 0));
  return tile_order(order_keys(L, ws, input), n, kv, counts, reinterpret_cast<uint2*>(ws + L.off_order_pairs), order, st);
}
// Keys or words of the rows that a fill kernel owns.
void ask_fill(const Layout& L, char* ws, int64_t n, const SideTables& t, const MaskSplits& m, bool input, FillOut* out) {
  out->cm = t.cm;
  out->rm = t.rm;
  if (t.order != nullptr) {
    out->keys = order_keys(L, ws, input);
    out->counts = bucket_counts(L, ws, n, input);
  }
  if (t.mask != nullptr) {
    out->words = reinterpret_cast<uint32_t*>(ws + L.off_words);
    out->iota = mask_iota(L, ws, m.words, m.n, m.do_sort);
  }
}
int emit_side(const Geo& g, const Layout& L, char* ws, int64_t n, const SideTables& t, const MaskSplits& m, bool input,
              cudaStream_t st) {
  if (t.order != nullptr) {
    const int rc = emit_order(L, ws, n, g.kv, t.order, input, st);
    if (rc != SPC_OK) return rc;
  }
  return t.mask != nullptr ? emit_masks(L, ws, n, g.kv, m.words, m.n, m.do_sort, t.mask, t.argsort, st) : SPC_OK;
}

// Input side of a strided / transposed layer on its own (its output side was made by an earlier call).
template <int ND, bool K64>
int backward_impl(const Geo& g, const Layout& L, const int32_t* idx, int64_t n_in, int64_t n_out, char* ws,
                  const SideTables& bwd, const MaskSplits& m, cudaStream_t st) {
  FillOut out{};
  ask_fill(L, ws, n_in, bwd, m, true, &out);
  const int rc = launch_fill<ND, K64, true>(g, idx, n_in, n_out, tout_at<K64>(ws, L), out, L.mic, st);
  return rc != SPC_OK ? rc : emit_side(g, L, ws, n_in, bwd, m, true, st);
}

// Both sides of a strided / transposed layer: clear the output side's tables, one pass over the input rows,
// one over the output rows.  The exactly sorted masks of both sides share their scratch, so an input side with
// masks is a pass of its own.
template <int ND, bool K64>
int strided_impl(const Geo& g, const Layout& L, const int32_t* idx, int64_t n_in, int64_t n_out, char* ws,
                 int32_t* out_indices, const SideTables& fwd, const SideTables& bwd, const MaskSplits& m, cudaStream_t st) {
  using key_t = typename Table<K64>::key_t;
  const int kvp = (g.kv + 3) & ~3;
  uint32_t* words = fwd.order || fwd.mask ? reinterpret_cast<uint32_t*>(ws + L.off_words) : nullptr;
  Clear c;
  c.add(fwd.rm, 0xFF, fwd.rm ? static_cast<size_t>(n_out) * kvp * 4 : 0);
  c.add(words, 0, words ? static_cast<size_t>(n_out) * L.mic * 4 : 0);
  c.add(fwd.cm, 0xFF, fwd.cm ? static_cast<size_t>(g.kv) * n_out * 4 : 0);
  int rc = c.total != 0 ? launch_clear(c, st) : SPC_OK;
  if (rc != SPC_OK) return rc;
  FillOut out{};
  const bool together = bwd.wanted() && bwd.mask == nullptr;
  if (together) ask_fill(L, ws, n_in, bwd, m, true, &out);
  out.out_cm = fwd.cm;
  out.out_rm = fwd.rm;
  out.out_words = words;
  out.order_bits = fwd.order != nullptr;
  rc = launch_fill<ND, K64, true>(g, idx, n_in, n_out, tout_at<K64>(ws, L), out, L.mic, st);
  if (rc != SPC_OK) return rc;
  finish_outputs_kernel<ND, K64><<<blocks_for(n_out), kThreads, 0, st>>>(
      g, reinterpret_cast<const key_t*>(ws + L.off_sorted), n_out, out_indices,
      fwd.mask ? mask_iota(L, ws, m.words, m.n, m.do_sort) : nullptr, fwd.order ? words : nullptr,
      order_keys(L, ws, false), bucket_counts(L, ws, n_out, false));
  SPC_LAUNCH_OK();
  rc = emit_side(g, L, ws, n_out, fwd, m, false, st);
  if (rc != SPC_OK || !bwd.wanted()) return rc;
  if (together) return emit_side(g, L, ws, n_in, bwd, m, true, st);
  return backward_impl<ND, K64>(g, L, idx, n_in, n_out, ws, bwd, m, st);
}

// A submanifold layer; rev_cm / rev_rm: its input side.
template <int ND, bool K64>
int subm_impl(const Geo& g, const Layout& L, const int32_t* idx, int64_t n, char* ws, const SideTables& fwd, int32_t* rev_cm,
              int32_t* rev_rm, const MaskSplits& m, cudaStream_t st) {
  FillOut out{};
  ask_fill(L, ws, n, fwd, m, false, &out);
  out.cm_rev = rev_cm;
  out.rm_rev = rev_rm;
  const int rc = launch_fill<ND, K64, false>(g, idx, n, n, tin_at<K64>(ws, L), out, L.mic, st);
  return rc != SPC_OK ? rc : emit_side(g, L, ws, n, fwd, m, false, st);
}

template <int ND, bool K64>
int native_impl(const Geo& g, const Layout& L, const int32_t* idx, int64_t n_in, int64_t n_out, char* ws,
                int32_t* out_indices, int32_t* pair, int32_t* npl, cudaStream_t st) {
  using key_t = typename Table<K64>::key_t;
  Table<K64> tin = tin_at<K64>(ws, L);
  Table<K64> tout = tout_at<K64>(ws, L);
  const Table<K64>& lookup = g.subm ? tin : tout;
  const key_t* sorted = reinterpret_cast<const key_t*>(ws + L.off_sorted);
  int* block_counts = reinterpret_cast<int*>(ws + L.off_native);
  const unsigned nb = static_cast<unsigned>(L.n_blocks_native);
  dim3 grid(nb, static_cast<unsigned>(g.kv));
  Clear c;
  c.add(pair, 0xFF, static_cast<size_t>(2) * g.kv * n_in * sizeof(int32_t));
  const int rc = launch_clear(c, st);
  if (rc != SPC_OK) return rc;
  native_count_kernel<ND, K64><<<grid, kThreads, 0, st>>>(g, idx, n_in, n_out, lookup, block_counts);
  SPC_LAUNCH_OK();
  native_scan_kernel<<<g.kv, kThreads, 0, st>>>(block_counts, static_cast<int>(nb), npl, g.kv, g.subm);
  SPC_LAUNCH_OK();
  native_write_kernel<ND, K64><<<grid, kThreads, 0, st>>>(g, idx, n_in, n_out, lookup, block_counts, pair);
  SPC_LAUNCH_OK();
  (void)sorted;
  (void)out_indices;
  return SPC_OK;
}

template <int ND, bool K64>
__global__ void __launch_bounds__(kThreads)
write_out_indices_kernel(const __grid_constant__ Geo g,
                         const typename Table<K64>::key_t* __restrict__ sorted, long long n_out,
                         int32_t* __restrict__ out_indices) {
  const long long r = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x;
  if (r >= n_out) return;
  int o[ND + 1];
  delinearize_out<ND>(g, static_cast<long long>(sorted[r]), o);
#pragma unroll
  for (int d = 0; d <= ND; ++d) out_indices[r * (ND + 1) + d] = o[d];
}

template <typename F>
int dispatch(int ndim, bool k64, F&& f) {
  switch (ndim * 2 + (k64 ? 1 : 0)) {
    case 2: return f(std::integral_constant<int, 1>{}, std::false_type{});
    case 3: return f(std::integral_constant<int, 1>{}, std::true_type{});
    case 4: return f(std::integral_constant<int, 2>{}, std::false_type{});
    case 5: return f(std::integral_constant<int, 2>{}, std::true_type{});
    case 6: return f(std::integral_constant<int, 3>{}, std::false_type{});
    case 7: return f(std::integral_constant<int, 3>{}, std::true_type{});
    case 8: return f(std::integral_constant<int, 4>{}, std::false_type{});
    case 9: return f(std::integral_constant<int, 4>{}, std::true_type{});
    default: return fail(SPC_ERR_INVALID_ARGUMENT, "ndim %d not in 1..4", ndim);
  }
}

// Points `L` at the output bitmap of `producer` if that strided layer numbered its outputs through
// one and its output grid is this layer's input grid.
void adopt_producer_bits(const Geo& g, Layout* L, const RulebookProducer* producer) {
  if (producer == nullptr || producer->geom == nullptr || producer->workspace == nullptr || L->k64) return;
  Geo gp;
  if (!make_geo(producer->geom, &gp) || gp.subm || gp.ndim != g.ndim || gp.batch != g.batch) return;
  for (int d = 0; d < g.ndim; ++d)
    if (gp.out_shape[d] != g.in_shape[d]) return;
  const Layout Lp = make_layout(gp, producer->n_in);
  if (Lp.obits_words == 0) return;
  const char* wp = static_cast<const char*>(producer->workspace);
  L->shared_bits = reinterpret_cast<const uint32_t*>(wp + Lp.off_obits);
  L->shared_prefix = reinterpret_cast<const uint32_t*>(wp + Lp.off_oprefix);
  L->shared_cells = reinterpret_cast<const uint32_t*>(wp + Lp.off_sorted);
}

}  // namespace

// A few page-locked words per host thread and device that kernels write and the host reads after
// synchronising (host memory: the library still allocates no device memory).
// One per host thread and device, with the ticket of the next message.
int host_mailbox(volatile int** out, int* ticket) {
  static thread_local int* boxes[kMaxDevices] = {nullptr};
  static thread_local int tickets[kMaxDevices] = {0};
  const int dev = current_device_slot();
  if (dev < 0) return fail(SPC_ERR_CUDA, "rulebook: no current device");
  if (boxes[dev] == nullptr) {
    void* p = nullptr;
    SPC_CUDA_OK(cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped));
    boxes[dev] = static_cast<int*>(p);
    boxes[dev][0] = 0;
  }
  *out = boxes[dev];
  tickets[dev] = (tickets[dev] + 1) & 0x7fffffff;
  if (tickets[dev] == 0) tickets[dev] = 1;
  *ticket = tickets[dev];
  return SPC_OK;
}

// How the host waits for a count: it spins on the page-locked ticket that the publishing kernel writes last,
// which is the fastest wake-up (the count is there before the stream has drained and without the driver's
// completion signal) but needs an idle core per pass in flight; with SPC_HOST_WAIT=block in the
// environment (read once) the thread sleeps on a blocking event instead, for processes that keep several
// passes in flight on few cores (one process per GPU, eight GPUs, three host threads each).  A stream that
// has drained, or failed, without the ticket ends the spin.  One event per host thread and device.
int wait_for_ticket(volatile int* box, int ticket, cudaStream_t st) {
  static const bool block = [] {
    const char* v = std::getenv("SPC_HOST_WAIT");
    return v != nullptr && std::strcmp(v, "block") == 0;
  }();
  if (!block) {
    for (unsigned spin = 1; box[0] != ticket; ++spin) {
      __builtin_ia32_pause();
      if ((spin & 0xfffu) != 0) continue;
      const cudaError_t e = cudaStreamQuery(st);
      if (e == cudaErrorNotReady) continue;
      SPC_CUDA_OK(e);
      if (box[0] != ticket) return fail(SPC_ERR_CUDA, "rulebook: the output count did not arrive");
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return SPC_OK;
  }
  static thread_local cudaEvent_t events[kMaxDevices] = {nullptr};
  const int dev = current_device_slot();
  if (dev < 0) return fail(SPC_ERR_CUDA, "rulebook: no current device");
  if (events[dev] == nullptr)
    SPC_CUDA_OK(cudaEventCreateWithFlags(&events[dev], cudaEventBlockingSync | cudaEventDisableTiming));
  SPC_CUDA_OK(cudaEventRecord(events[dev], st));
  SPC_CUDA_OK(cudaEventSynchronize(events[dev]));
  if (box[0] != ticket) return fail(SPC_ERR_CUDA, "rulebook: the output count did not arrive");
  return SPC_OK;
}

int rulebook_prepare_chained(const spc_geometry* sg, const int32_t* indices, int64_t n_in, void* workspace,
                             size_t workspace_bytes, int64_t* n_out_host, const RulebookProducer* producer,
                             cudaStream_t st) {
  Geo g;
  if (!make_geo(sg, &g)) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook: bad geometry");
  if (n_in <= 0 || indices == nullptr || n_out_host == nullptr || workspace == nullptr)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook: n_in must be > 0 and pointers non-null");
  if (n_in >= (1ll << 30)) return fail(SPC_ERR_SIZE_LIMIT, "rulebook: n_in %lld too large", (long long)n_in);
  Layout L = make_layout(g, n_in);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "rulebook: workspace %zu < %zu bytes", workspace_bytes, L.total);
  adopt_producer_bits(g, &L, producer);
  char* ws = static_cast<char*>(workspace);
  return dispatch(g.ndim, L.k64, [&](auto nd, auto k64) {
    return prepare_impl<decltype(nd)::value, decltype(k64)::value>(g, L, indices, n_in, ws, n_out_host, st);
  });
}

bool rulebook_adopts(const spc_geometry* sg, int64_t n_in, const RulebookProducer* producer) {
  Geo g;
  if (!make_geo(sg, &g)) return false;
  Layout L = make_layout(g, n_in);
  adopt_producer_bits(g, &L, producer);
  // (outputs that are not marked in a bitmap are enumerated from the coordinates)
  return L.shared_bits != nullptr && (g.subm || (L.obits_words != 0 && g.axes_fit));
}

int rulebook_tables_chained(const spc_geometry* sg, const int32_t* indices, int64_t n_in, int64_t n_out,
                            void* workspace, size_t workspace_bytes, const RulebookTables& t,
                            const RulebookProducer* producer, cudaStream_t st) {
  Geo g;
  if (!make_geo(sg, &g)) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook: bad geometry");
  const bool input_side = t.bwd_colmajor || t.bwd_rowmajor || t.bwd_order;
  if (n_in <= 0 || n_out <= 0 || !indices || !workspace)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook tables: bad arguments");
  if (g.subm && (n_out != n_in || input_side))
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook tables: a submanifold layer has one side");
  if ((t.fwd_order || t.bwd_order) && g.kv > 32)
    return fail(SPC_ERR_UNSUPPORTED, "rulebook tables: tile order of %d offsets (32 at most)", g.kv);
  if ((reinterpret_cast<uintptr_t>(t.fwd_rowmajor) | reinterpret_cast<uintptr_t>(t.bwd_rowmajor)) & 15u)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook tables: row-major tables must be 16-byte aligned");
  Layout L = make_layout(g, n_in);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "rulebook: workspace %zu < %zu bytes", workspace_bytes, L.total);
  if (n_out > L.bound) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook tables: n_out exceeds prepared bound");
  adopt_producer_bits(g, &L, producer);
  char* ws = static_cast<char*>(workspace);
  return dispatch(g.ndim, L.k64, [&](auto nd, auto k64) -> int {
    constexpr int ND = decltype(nd)::value;
    constexpr bool K64 = decltype(k64)::value;
    SideTables fwd, bwd;
    fwd.cm = t.fwd_colmajor;
    fwd.rm = t.fwd_rowmajor;
    fwd.order = t.fwd_order;
    bwd.cm = t.bwd_colmajor;
    bwd.rm = t.bwd_rowmajor;
    bwd.order = t.bwd_order;
    if (g.subm) return subm_impl<ND, K64>(g, L, indices, n_in, ws, fwd, nullptr, nullptr, MaskSplits{}, st);
    if (!fwd.wanted() && t.out_indices == nullptr)
      return backward_impl<ND, K64>(g, L, indices, n_in, n_out, ws, bwd, MaskSplits{}, st);
    return strided_impl<ND, K64>(g, L, indices, n_in, n_out, ws, t.out_indices, fwd, bwd, MaskSplits{}, st);
  });
}

}  // namespace spc

using namespace spc;

extern "C" size_t spc_rulebook_workspace_bytes(const spc_geometry* sg, int64_t n_in) {
  Geo g;
  if (!make_geo(sg, &g) || n_in <= 0) return 0;
  return make_layout(g, n_in).total;
}

extern "C" int spc_rulebook_prepare(const spc_geometry* sg, const int32_t* indices, int64_t n_in,
                                    void* workspace, size_t workspace_bytes, int64_t* n_out_host,
                                    void* stream) {
  return rulebook_prepare_chained(sg, indices, n_in, workspace, workspace_bytes, n_out_host, nullptr,
                                  static_cast<cudaStream_t>(stream));
}

extern "C" int spc_rulebook_tables(const spc_geometry* sg, const int32_t* indices, int64_t n_in, int64_t n_out,
                                   void* workspace, size_t workspace_bytes, int32_t* out_indices,
                                   int32_t* pair_fwd, int32_t* pair_fwd_rowmajor, int32_t* order_fwd,
                                   int32_t* pair_bwd, int32_t* pair_bwd_rowmajor, int32_t* order_bwd, void* stream) {
  const RulebookTables t{out_indices, pair_fwd, pair_fwd_rowmajor, order_fwd, pair_bwd, pair_bwd_rowmajor, order_bwd};
  return rulebook_tables_chained(sg, indices, n_in, n_out, workspace, workspace_bytes, t, nullptr,
                                 static_cast<cudaStream_t>(stream));
}

extern "C" int spc_rulebook_igemm(const spc_geometry* sg, const int32_t* indices, int64_t n_in,
                                  int64_t n_out, void* workspace, size_t workspace_bytes,
                                  int32_t* out_indices, int32_t* pair_fwd, int32_t* pair_bwd,
                                  int32_t* mask_fwd, int32_t* argsort_fwd, int32_t* mask_bwd,
                                  int32_t* argsort_bwd, const uint32_t* split_masks, int n_split,
                                  int do_sort, int32_t* pair_fwd_rowmajor, int32_t* pair_bwd_rowmajor,
                                  void* stream) {
  Geo g;
  if (!make_geo(sg, &g)) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook: bad geometry");
  if (n_in <= 0 || n_out <= 0 || !indices || !workspace || !pair_fwd || !mask_fwd || !argsort_fwd || !split_masks ||
      n_split < 1 || n_split > 2)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm: bad arguments");
  if (!g.subm && out_indices == nullptr)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm: out_indices required for non-subm layers");
  if (g.subm && n_out != n_in) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm: subm needs n_out == n_in");
  if ((mask_bwd == nullptr) != (argsort_bwd == nullptr))
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm: mask_bwd and argsort_bwd go together");
  const Layout L = make_layout(g, n_in);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "rulebook: workspace %zu < %zu bytes", workspace_bytes, L.total);
  if (n_out > L.bound) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm: n_out exceeds prepared bound");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  SideTables fwd, bwd;
  fwd.cm = pair_fwd;
  fwd.rm = pair_fwd_rowmajor;
  fwd.mask = mask_fwd;
  fwd.argsort = argsort_fwd;
  bwd.cm = pair_bwd;
  bwd.rm = pair_bwd_rowmajor;
  bwd.mask = mask_bwd;
  bwd.argsort = argsort_bwd;
  const MaskSplits m{split_masks, n_split, do_sort};
  return dispatch(g.ndim, L.k64, [&](auto nd, auto k64) {
    constexpr int ND = decltype(nd)::value;
    constexpr bool K64 = decltype(k64)::value;
    if (g.subm) return subm_impl<ND, K64>(g, L, indices, n_in, ws, fwd, pair_bwd, pair_bwd_rowmajor, m, st);
    return strided_impl<ND, K64>(g, L, indices, n_in, n_out, ws, out_indices, fwd, pair_bwd ? bwd : SideTables{}, m, st);
  });
}

extern "C" int spc_rulebook_igemm_backward(const spc_geometry* sg, const int32_t* indices, int64_t n_in,
                                           int64_t n_out, void* workspace, size_t workspace_bytes,
                                           int32_t* pair_bwd, int32_t* mask_bwd, int32_t* argsort_bwd,
                                           const uint32_t* split_masks, int n_split, int do_sort,
                                           int32_t* pair_bwd_rowmajor, void* stream) {
  Geo g;
  if (!make_geo(sg, &g)) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook: bad geometry");
  if (g.subm) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm backward: submanifold tables come from the forward call");
  if (n_in <= 0 || n_out <= 0 || !indices || !workspace || !pair_bwd || !split_masks || n_split < 1 || n_split > 2)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm backward: bad arguments");
  if ((mask_bwd == nullptr) != (argsort_bwd == nullptr))
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm backward: mask_bwd and argsort_bwd go together");
  const Layout L = make_layout(g, n_in);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "rulebook: workspace %zu < %zu bytes", workspace_bytes, L.total);
  if (n_out > L.bound) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook igemm backward: n_out exceeds prepared bound");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  SideTables bwd;
  bwd.cm = pair_bwd;
  bwd.rm = pair_bwd_rowmajor;
  bwd.mask = mask_bwd;
  bwd.argsort = argsort_bwd;
  const MaskSplits m{split_masks, n_split, do_sort};
  return dispatch(g.ndim, L.k64, [&](auto nd, auto k64) {
    return backward_impl<decltype(nd)::value, decltype(k64)::value>(g, L, indices, n_in, n_out, ws, bwd, m, st);
  });
}

extern "C" int spc_rulebook_native(const spc_geometry* sg, const int32_t* indices, int64_t n_in,
                                   int64_t n_out, void* workspace, size_t workspace_bytes,
                                   int32_t* out_indices, int32_t* pair, int32_t* indice_num_per_loc,
                                   void* stream) {
  Geo g;
  if (!make_geo(sg, &g)) return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook: bad geometry");
  if (n_in <= 0 || n_out <= 0 || !indices || !workspace || !pair || !indice_num_per_loc)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook native: bad arguments");
  if (!g.subm && out_indices == nullptr)
    return fail(SPC_ERR_INVALID_ARGUMENT, "rulebook native: out_indices required for non-subm layers");
  const Layout L = make_layout(g, n_in);
  if (workspace_bytes < L.total)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "rulebook: workspace %zu < %zu bytes", workspace_bytes, L.total);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(workspace);
  return dispatch(g.ndim, L.k64, [&](auto nd, auto k64) {
    constexpr int ND = decltype(nd)::value;
    constexpr bool K64 = decltype(k64)::value;
    if (!g.subm) {
      using key_t = typename Table<K64>::key_t;
      write_out_indices_kernel<ND, K64><<<blocks_for(n_out), kThreads, 0, st>>>(
          g, reinterpret_cast<const key_t*>(ws + L.off_sorted), n_out, out_indices);
      SPC_LAUNCH_OK();
    }
    return native_impl<ND, K64>(g, L, indices, n_in, n_out, ws, out_indices, pair, indice_num_per_loc, st);
  });
}

extern "C" int spc_pairs_to_rowmajor(const int32_t* pairs, int kv, int64_t n, int32_t* out, void* stream) {
  if (!pairs || !out || kv <= 0 || n < 0) return fail(SPC_ERR_INVALID_ARGUMENT, "pairs_to_rowmajor: bad arguments");
  if (n == 0) return SPC_OK;
  const int kvp = (kv + 3) & ~3;
  pairs_to_rowmajor_kernel<<<blocks_for(n * (kvp / 4)), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      pairs, kv, kvp, n, out);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

extern "C" int spc_rowmajor_to_pairs(const int32_t* rowmajor, int kv, int64_t n, int32_t* pairs, void* stream) {
  if (!rowmajor || !pairs || kv <= 0 || n < 0) return fail(SPC_ERR_INVALID_ARGUMENT, "rowmajor_to_pairs: bad arguments");
  if (n == 0) return SPC_OK;
  const int kvp = (kv + 3) & ~3;
  const dim3 grid(static_cast<unsigned>(ceil_div(n, 32)), static_cast<unsigned>(ceil_div(kv, 32)));
  rowmajor_to_pairs_kernel<<<grid, dim3(32, 8), 0, static_cast<cudaStream_t>(stream)>>>(rowmajor, kv, kvp, n, pairs);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

extern "C" int spc_rowmajor_order(const spc_geometry* sg, const int32_t* rowmajor, int64_t n, int32_t* order, uint32_t* keys, void* stream) {
  Geo g;
  if (!make_geo(sg, &g) || !rowmajor || !order || !keys || n < 0) return fail(SPC_ERR_INVALID_ARGUMENT, "rowmajor_order: bad arguments");
  if (g.kv > 32 || tile_order_needs_buckets(n)) return fail(SPC_ERR_UNSUPPORTED, "rowmajor_order: %d offsets, %lld rows", g.kv, static_cast<long long>(n));
  if (n == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rowmajor_keys_kernel<<<blocks_for(n), kThreads, 0, st>>>(g, rowmajor, (g.kv + 3) & ~3, n, keys);
  SPC_LAUNCH_OK();
  return tile_order(keys, n, g.kv, nullptr, nullptr, order, st);
}

extern "C" int spc_native_to_tables(const int32_t* pair, int kv, int64_t n_pair, int inverse,
                                    int32_t* pair_fwd, int64_t n_out, int32_t* pair_bwd, int64_t n_in,
                                    void* stream) {
  if (!pair || !pair_fwd || kv <= 0 || n_pair < 0 || n_out < 0 || n_in < 0)
    return fail(SPC_ERR_INVALID_ARGUMENT, "native_to_tables: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Clear c;
  c.add(pair_fwd, 0xFF, static_cast<size_t>(kv) * n_out * 4);
  if (pair_bwd) c.add(pair_bwd, 0xFF, static_cast<size_t>(kv) * n_in * 4);
  const int rc = c.total != 0 ? launch_clear(c, st) : SPC_OK;
  if (rc != SPC_OK || n_pair == 0) return rc;
  const int32_t* pair_in = pair + static_cast<int64_t>(inverse ? 1 : 0) * kv * n_pair;
  const int32_t* pair_out = pair + static_cast<int64_t>(inverse ? 0 : 1) * kv * n_pair;
  dim3 grid(blocks_for(n_pair), static_cast<unsigned>(kv));
  native_to_tables_kernel<<<grid, kThreads, 0, st>>>(pair_in, pair_out, kv, n_pair, pair_fwd, n_out, pair_bwd, n_in);
  SPC_LAUNCH_OK();
  return SPC_OK;
}
