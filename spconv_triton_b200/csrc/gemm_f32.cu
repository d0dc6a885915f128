// IEEE fp32 gather-GEMM and weight gradient on the CUDA cores, for channel counts that are multiples of four.
//
// Bound: the fp32 pipe, once the operands come out of shared memory wide enough and work for absent rows is
// left out.  Both kernels compute 64 x 64 outputs with 128 threads, 8 x 4 each: per reduction step a thread
// reads three 16-byte words for 32 multiply-adds (16 packed fma.rn.f32x2, the same IEEE results), a warp
// four shared-memory wavefronts.  The tile's rows come in an order that groups rows with common offsets, a
// warp skips the offsets that none of its 16 rows has, and the next stage's operands are in flight during the
// multiplications.  SubM 64 -> 64, 100 k rows, 6.2 of 27 neighbours: forward 104 us, input gradient 97, weight
// gradient 75 (49 - 51 % of the issue slots in the first two; 128 registers, four CTAs a multiprocessor).  With 4 x 4 outputs a
// thread, scalar shared-memory reads and a barrier twice every 16 channels: 425, 425 (240 with sorted rows), 727.
#include <algorithm>

#include "common.cuh"
#include "gemm_internal.cuh"

namespace spc {
namespace {

constexpr int kTile = 64;      // rows and output channels of a tile
constexpr int kStep = 32;      // reduction steps of a stage
constexpr int kThreads = 128;
constexpr int kGroupOffsets = 32;

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// One reduction step of a thread's 8 x 4 outputs: acc[q][j] holds rows 2q and 2q + 1 of column j.
__device__ __forceinline__ void multiply_add(unsigned long long (&acc)[4][4], const float4& a0, const float4& a1, const float4& b) {
  const unsigned long long a[4] = {pack2(a0.x, a0.y), pack2(a0.z, a0.w), pack2(a1.x, a1.y), pack2(a1.z, a1.w)};
  const unsigned long long bb[4] = {pack2(b.x, b.x), pack2(b.y, b.y), pack2(b.z, b.z), pack2(b.w, b.w)};
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) fma2(acc[q][j], a[q], bb[j]);
}

struct F32Params {
  const float* src;
  const float* w;
  Epilogue epi;
  const int32_t* pairs;     // column-major table, or
  const int32_t* pairs_rm;  // row-major
  const int32_t* order;
  float* out;
  long long m_rows;
  int n_dim, r_dim, kv, kvp, reversed;
};

// Tiles of shared memory are [step][64 rows or channels] with the 4-entry blocks of step s permuted by
// (s / 4) mod 8: the transposing stores of 4 rows x 8 blocks of a warp then fall into 32 different banks,
// and a thread's reads stay 16-byte words.
__device__ __forceinline__ int swizzled(int step, int index) { return step * kTile + ((((index >> 2) ^ ((step >> 2) & 7)) << 2) | (index & 3)); }

// out[row, n] = sum over offsets k and reduction r of src[table[k, row], r] * w; W_MN = false: w[n][k][r]
// (forward), true: w[r][k][n] (input gradient).
template <bool W_MN>
__global__ void __launch_bounds__(kThreads, 4)
gather_gemm_f32_kernel(const __grid_constant__ F32Params p) {
  __shared__ __align__(16) float a_s[2][kStep * kTile];
  __shared__ __align__(16) float b_s[2][kStep * kTile];
  __shared__ int idx_s[kGroupOffsets * kTile];
  __shared__ uint32_t vote[kThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = tid & 15, ty = tid >> 4;  // columns 4 tx .., rows 8 ty ..: a warp has 16 rows
  // tiles from the end of the order first: those rows have the most offsets
  const long long m0 = static_cast<long long>(gridDim.x - 1 - blockIdx.x) * kTile;
  const int n0 = blockIdx.y * kTile;
  // loader: eight lanes a row (128 bytes), this thread's rows lr, lr + 16, ..
  const int lr = tid >> 3, lc = (tid & 7) * 4;

  unsigned long long acc[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[q][j] = 0ull;

  long long own = -1;  // the row whose table entries this thread fetches (threads 0..63)
  if (tid < kTile && m0 + tid < p.m_rows) own = p.order != nullptr ? static_cast<long long>(__ldg(&p.order[m0 + tid])) : m0 + tid;
  const int chunks = (p.r_dim + kStep - 1) / kStep;

  for (int k0 = 0; k0 < p.kv; k0 += kGroupOffsets) {
    const int gcount = min(kGroupOffsets, p.kv - k0);
    __syncthreads();  // the table tile of the previous group is no longer read
    uint32_t mine = 0;
    if (tid < kTile) {
      if (p.pairs_rm != nullptr) {
        const int4* at = reinterpret_cast<const int4*>(p.pairs_rm + (own >= 0 ? own : 0) * p.kvp + k0);
#pragma unroll
        for (int q = 0; q < kGroupOffsets / 4; ++q) {
          int4 v = make_int4(-1, -1, -1, -1);
          if (4 * q < gcount && own >= 0) v = __ldg(at + q);
          const int e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            idx_s[(4 * q + u) * kTile + tid] = e[u];
            mine |= static_cast<uint32_t>(e[u] >= 0) << (4 * q + u);
          }
        }
      } else {
#pragma unroll 8
        for (int kk = 0; kk < gcount; ++kk) {
          const int e = own >= 0 ? __ldg(&p.pairs[static_cast<long long>(k0 + kk) * p.m_rows + own]) : -1;
          idx_s[kk * kTile + tid] = e;
          mine |= static_cast<uint32_t>(e >= 0) << kk;
        }
      }
      // vote of 16 rows each: half warps
      const unsigned half = 0xffffu << (lane & 16);
      mine = __reduce_or_sync(half, mine);
      if ((lane & 15) == 0) vote[warp * 2 + (lane >> 4)] = mine;
    }
    __syncthreads();
    const uint32_t active = vote[0] | vote[1] | vote[2] | vote[3], wanted = vote[warp];

    // stages: (offset, chunk of the reduction); the next one is loaded to registers during a stage
    float4 ra[4], rb[4];
    uint32_t rest = active;
    int chunk = 0;
    auto load = [&](int kk, int rc) {
      const int r0 = rc * kStep;
      const int kw = p.reversed ? p.kv - 1 - (k0 + kk) : k0 + kk;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = idx_s[kk * kTile + lr + 16 * u];
        ra[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j >= 0 && r0 + lc < p.r_dim) ra[u] = __ldg(reinterpret_cast<const float4*>(p.src + static_cast<long long>(j) * p.r_dim + r0 + lc));
        rb[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!W_MN) {
          const int n = n0 + lr + 16 * u;
          if (n < p.n_dim && r0 + lc < p.r_dim)
            rb[u] = __ldg(reinterpret_cast<const float4*>(p.w + (static_cast<long long>(n) * p.kv + kw) * p.r_dim + r0 + lc));
        } else {
          // 16 lanes cover the 64 output channels of a reduction row
          const int r = r0 + (tid >> 4) + 8 * u, n = n0 + (tid & 15) * 4;
          if (n < p.n_dim && r < p.r_dim)
            rb[u] = __ldg(reinterpret_cast<const float4*>(p.w + (static_cast<long long>(r) * p.kv + kw) * p.n_dim + n));
        }
      }
    };
    auto store = [&](int buf) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int row = lr + 16 * u;
        const float a[4] = {ra[u].x, ra[u].y, ra[u].z, ra[u].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) a_s[buf][swizzled(lc + q, row)] = a[q];
        if (!W_MN) {
          const float b[4] = {rb[u].x, rb[u].y, rb[u].z, rb[u].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) b_s[buf][swizzled(lc + q, row)] = b[q];
        } else {
          *reinterpret_cast<float4*>(&b_s[buf][swizzled((tid >> 4) + 8 * u, (tid & 15) * 4)]) = rb[u];
        }
      }
    };
    int buf = 0;
    if (rest != 0) {
      load(__ffs(rest) - 1, 0);
      store(0);
    }
    while (rest != 0) {
      const int kk = __ffs(rest) - 1;
      __syncthreads();  // this stage is stored; the other buffer is no longer read
      uint32_t next = rest;
      int next_chunk = chunk + 1;
      if (next_chunk == chunks) {
        next_chunk = 0;
        next &= next - 1;
      }
      if (next != 0) load(__ffs(next) - 1, next_chunk);
      if ((wanted >> kk) & 1u) {
        const float* as = a_s[buf];
        const float* bs = b_s[buf];
        const int steps = min(kStep, p.r_dim - chunk * kStep);  // a multiple of four
        for (int s0 = 0; s0 < steps; s0 += 4) {
          const int x = (s0 >> 2) & 7;
          const float* ap = as + s0 * kTile + (((2 * ty) ^ x) << 2);
          const float* aq = as + s0 * kTile + (((2 * ty + 1) ^ x) << 2);
          const float* bp = bs + s0 * kTile + ((tx ^ x) << 2);
#pragma unroll
          for (int s = 0; s < 4; ++s)
            multiply_add(acc, *reinterpret_cast<const float4*>(ap + s * kTile), *reinterpret_cast<const float4*>(aq + s * kTile),
                         *reinterpret_cast<const float4*>(bp + s * kTile));
        }
      }
      if (next != 0) store(buf ^ 1);
      buf ^= 1;
      rest = next;
      chunk = next_chunk;
    }
  }

  const int n = n0 + 4 * tx;
  if (n >= p.n_dim) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float v[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) unpack2(acc[q][j], v[0][j], v[1][j]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long slot = m0 + 8 * ty + 2 * q + h;
      if (slot >= p.m_rows) continue;
      const long long row = p.order != nullptr ? static_cast<long long>(__ldg(&p.order[slot])) : slot;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[h][j] = apply_epilogue<float>(v[h][j], p.epi, n + j);
      if (p.epi.residual != nullptr) {
        const float4 r = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p.epi.residual) + row * p.n_dim + n));
        v[h][0] += r.x; v[h][1] += r.y; v[h][2] += r.z; v[h][3] += r.w;
      }
      *reinterpret_cast<float4*>(p.out + row * p.n_dim + n) = make_float4(v[h][0], v[h][1], v[h][2], v[h][3]);
    }
  }
}

// ---- weight gradient ---------------------------------------------------------------------------------------------

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %2, 0;\n\tcp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(static_cast<int>(live))
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int kListRows = 512;  // table entries compacted at a time

// partial[split, n, k, c] = sum over the pairs (i, o) of offset k with o in the split's rows of gout[o, n] * feats[i, c].
// The reduction runs over pairs: a stage is 32 of them, 64 channels of both rows, copied as they lie.
__global__ void __launch_bounds__(kThreads, 4)
wgrad_f32_kernel(const float* __restrict__ feats, const float* __restrict__ gout, const int32_t* __restrict__ pair_fwd,
                 float* __restrict__ partial, long long n_out, int c_in, int c_out, int kv, int first_turn, int splits, long long rows_per_split) {
  __shared__ __align__(16) float g_s[2][kStep * kTile];
  __shared__ __align__(16) float f_s[2][kStep * kTile];
  __shared__ int list_i[kListRows], list_o[kListRows];
  __shared__ int warp_cnt[kListRows / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = tid & 15, ty = tid >> 4;
  // the middle offsets first, all channel blocks of one before the next: they have the most pairs
  const int turn = first_turn + blockIdx.z / splits, split = blockIdx.z % splits;
  const int k = (turn & 1) ? (kv - 1) / 2 + (turn + 1) / 2 : (kv - 1) / 2 - turn / 2;
  const int c0 = blockIdx.x * kTile, n0 = blockIdx.y * kTile;
  const long long lo = split * rows_per_split, hi = min(n_out, lo + rows_per_split);
  const int32_t* col = pair_fwd + static_cast<long long>(k) * n_out;
  const int lp = tid >> 4, lc = (tid & 15) * 4;  // loader: sixteen lanes a pair, pairs lp, lp + 8, ..

  unsigned long long acc[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[q][j] = 0ull;

  constexpr int kEach = kListRows / kThreads;
  int ahead[kEach];  // table entries of the next round
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const long long m = lo + e * kThreads + tid;
    ahead[e] = m < hi ? __ldg(&col[m]) : -1;
  }
  for (long long base = lo; base < hi; base += kListRows) {
    unsigned ballot[kEach];
#pragma unroll
    for (int e = 0; e < kEach; ++e) {
      ballot[e] = __ballot_sync(0xffffffffu, ahead[e] >= 0);
      if (lane == 0) warp_cnt[e * (kThreads / 32) + warp] = __popc(ballot[e]);
    }
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int e = 0; e < kEach; ++e) {
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) {
        if (w == warp && ahead[e] >= 0) {
          const int at = total + __popc(ballot[e] & ((1u << lane) - 1u));
          list_i[at] = ahead[e];
          list_o[at] = e * kThreads + tid;
        }
        total += warp_cnt[e * (kThreads / 32) + w];
      }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kEach; ++e) {
      const long long m = base + kListRows + e * kThreads + tid;
      ahead[e] = m < hi ? __ldg(&col[m]) : -1;
    }
    auto load = [&](int p0, int buf) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int pr = lp + 8 * u;
        const bool live = p0 + pr < total;
        const long long o = live ? base + list_o[p0 + pr] : 0, i = live ? list_i[p0 + pr] : 0;
        copy16(&g_s[buf][pr * kTile + lc], gout + o * c_out + (n0 + lc < c_out ? n0 + lc : 0), live && n0 + lc < c_out);
        copy16(&f_s[buf][pr * kTile + lc], feats + i * c_in + (c0 + lc < c_in ? c0 + lc : 0), live && c0 + lc < c_in);
      }
      copies_commit();
    };
    if (total > 0) load(0, 0);
    for (int p0 = 0, buf = 0; p0 < total; p0 += kStep, buf ^= 1) {
      if (p0 + kStep < total) {
        load(p0 + kStep, buf ^ 1);
        copies_wait<1>();
      } else {
        copies_wait<0>();
      }
      __syncthreads();
      const float* gp = g_s[buf] + 8 * ty;
      const float* fp = f_s[buf] + 4 * tx;
      const int steps = min(kStep, (total - p0 + 3) & ~3);
      for (int s0 = 0; s0 < steps; s0 += 4)
#pragma unroll
        for (int s = 0; s < 4; ++s)
          multiply_add(acc, *reinterpret_cast<const float4*>(gp + (s0 + s) * kTile), *reinterpret_cast<const float4*>(gp + (s0 + s) * kTile + 4),
                       *reinterpret_cast<const float4*>(fp + (s0 + s) * kTile));
      __syncthreads();
    }
  }
  const int c = c0 + 4 * tx;
  if (c >= c_in) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float v[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) unpack2(acc[q][j], v[0][j], v[1][j]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = n0 + 8 * ty + 2 * q + h;
      if (n < c_out)
        *reinterpret_cast<float4*>(&partial[((static_cast<long long>(split) * c_out + n) * kv + k) * c_in + c]) =
            make_float4(v[h][0], v[h][1], v[h][2], v[h][3]);
    }
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Few rows (the rule is at gather_gemm_small_takes): a tile of 64 or 128 rows is one chain of up to 27 offsets on a chip that
// is nearly empty.  Here a CTA has eight rows, 16 lanes a row, and passes over the offsets that any of them has, a batch of
// them at a time: the weights of each (read by neighbouring lanes, whichever way they are transposed) and the rows that have
// it come by cp.async while the batch before is multiplied, by a row's lanes, NC output channels each, for the offsets that
// the row has.
// Bound: latency, of the table entries, then of the copies, then of the multiplications of a row.  Measured beside the rule.
constexpr int kSmallRows = kThreads / 16;
// Floats between staged rows: whole 16-byte words, an odd number of them, so that lanes on neighbouring rows meet different banks.
__host__ __device__ constexpr int small_pitch(int floats) { return ((floats >> 2) | 1) << 2; }
constexpr int kSmallBatchBytes = 40 * 1024, kSmallMostBatch = 8;  // of the offsets of a batch (two such buffers)
static_assert((64 + kSmallRows) * small_pitch(64) * sizeof(float) <= kSmallBatchBytes, "an offset at least");

__device__ __forceinline__ void copy16(uint32_t to, const float* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}

template <bool W_MN, int NC>  // NC: output channels of a lane
__global__ void __launch_bounds__(kThreads)
gather_gemm_small_kernel(const __grid_constant__ F32Params p, int batch_most) {
  extern __shared__ __align__(16) float small_stages[];  // [2][batch_most] stages
  __shared__ __align__(16) int entries[kSmallRows][32];
  __shared__ uint32_t votes[kThreads / 32];
  const int group = threadIdx.x >> 4, lane = threadIdx.x & 15;
  const long long row = static_cast<long long>(blockIdx.x) * kSmallRows + group;
  uint32_t mine = 0;
  if (lane < 8) {
    int4 e = make_int4(-1, -1, -1, -1);
    if (row < p.m_rows && 4 * lane < p.kvp) e = __ldg(reinterpret_cast<const int4*>(p.pairs_rm + row * p.kvp) + lane);
    *reinterpret_cast<int4*>(&entries[group][4 * lane]) = e;
    mine = ((e.x >= 0 ? 1u : 0u) | (e.y >= 0 ? 2u : 0u) | (e.z >= 0 ? 4u : 0u) | (e.w >= 0 ? 8u : 0u)) << (4 * lane);
  }
#pragma unroll
  for (int s = 8; s > 0; s >>= 1) mine |= __shfl_xor_sync(0xffffffffu, mine, s);
  const uint32_t both = mine | __shfl_xor_sync(0xffffffffu, mine, 16);
  if ((threadIdx.x & 31) == 0) votes[threadIdx.x >> 5] = both;
  __syncthreads();
  uint32_t all = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) all |= votes[w];

  // A stage: the weights, [n_dim][r_dim] or, read transposed, [r_dim][n_dim] with the pitch of their rows, and the CTA's rows.
  const int w_rows = W_MN ? p.r_dim : p.n_dim, w_cols = W_MN ? p.n_dim : p.r_dim;
  const int w_pitch = small_pitch(w_cols), x_pitch = small_pitch(p.r_dim);
  const int stage_floats = w_rows * w_pitch + kSmallRows * x_pitch;
  const int x_at = w_rows * w_pitch + group * x_pitch;
  // this thread's piece of the weight rows `group`, `group` + kSmallRows, ... and of its own row
  const float* const w_from = p.w + group * p.kv * w_cols + 4 * lane;
  const float* const x_from = p.src + 4 * lane;
  const int w_step = kSmallRows * p.kv * w_cols;
  const uint32_t stages = static_cast<uint32_t>(__cvta_generic_to_shared(small_stages));
  const uint32_t w_to = 4 * (group * w_pitch + 4 * lane), x_to = 4 * (x_at + 4 * lane);
  const bool w_lane = 4 * lane < w_cols, x_lane = 4 * lane < p.r_dim;
  const uint32_t stage_bytes = 4 * stage_floats;
  uint32_t ahead = all;  // offsets that have not been asked for
  // The next offsets, into one half of the stages in ascending order.
  const auto fetch = [&](int half) {
    const uint32_t before = ahead;
    uint32_t to = stages + half * batch_most * stage_bytes;
#pragma unroll 2
    for (int j = 0; j < batch_most && ahead != 0; ++j, to += stage_bytes) {
      const int kk = __ffs(ahead) - 1, k = p.reversed ? p.kv - 1 - kk : kk;
      ahead &= ahead - 1;
      const int entry = entries[group][kk];
      if (w_lane) {
        const float* from = w_from + k * w_cols;
        uint32_t there = to + w_to;
#pragma unroll 4
        for (int i = group; i < w_rows; i += kSmallRows, from += w_step, there += 4 * kSmallRows * w_pitch) copy16(there, from);
      }
      if (x_lane && entry >= 0) copy16(to + x_to, x_from + static_cast<long long>(entry) * p.r_dim);
    }
    return before ^ ahead;
  };

  float acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = 0.f;
  uint32_t next = fetch(0);
#pragma unroll 1
  for (int half = 0; next != 0; half ^= 1) {
    const uint32_t batch = next;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // this batch is there for everyone, and everyone is done with the one before it
    next = fetch(half ^ 1);
#pragma unroll 1
    for (uint32_t rest = batch & mine; rest != 0; rest &= rest - 1) {
      const float* const stage = small_stages + (half * batch_most + __popc(batch & ((rest & -rest) - 1u))) * stage_floats;
      const float4* const x = reinterpret_cast<const float4*>(stage + x_at);
#pragma unroll 4
      for (int r = 0; r < p.r_dim; r += 4) {
        const float4 a = x[r >> 2];
        float b[4][NC];
        if (W_MN) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < NC; ++c) b[q][c] = stage[(r + q) * w_pitch + lane + 16 * c];
        } else {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(stage + (lane + 16 * c) * w_pitch + r);
            b[0][c] = v.x; b[1][c] = v.y; b[2][c] = v.z; b[3][c] = v.w;
          }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          acc[c] = fmaf(a.x, b[0][c], acc[c]);
          acc[c] = fmaf(a.y, b[1][c], acc[c]);
          acc[c] = fmaf(a.z, b[2][c], acc[c]);
          acc[c] = fmaf(a.w, b[3][c], acc[c]);
        }
      }
    }
  }
  if (row >= p.m_rows) return;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int n = lane + 16 * c;
    float v = apply_epilogue<float>(acc[c], p.epi, n);
    if (p.epi.residual != nullptr) v += static_cast<const float*>(p.epi.residual)[row * p.n_dim + n];
    p.out[row * p.n_dim + n] = v;
  }
}

template <bool W_MN, int NC>
int launch_small(const F32Params& p, cudaStream_t st) {
  const int w_rows = W_MN ? p.r_dim : p.n_dim, w_cols = W_MN ? p.n_dim : p.r_dim;
  const size_t stage_bytes = (static_cast<size_t>(w_rows) * small_pitch(w_cols) + kSmallRows * small_pitch(p.r_dim)) * sizeof(float);
  const int batch = std::min(kSmallMostBatch, static_cast<int>(kSmallBatchBytes / stage_bytes));
  static bool configured[kMaxDevices] = {false};  // per instantiation and device
  SPC_CUDA_OK(ensure_dynamic_smem(gather_gemm_small_kernel<W_MN, NC>, 2 * kSmallBatchBytes, configured));
  gather_gemm_small_kernel<W_MN, NC>
      <<<static_cast<unsigned>(ceil_div(p.m_rows, kSmallRows)), kThreads, 2 * batch * stage_bytes, st>>>(p, batch);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace

// 16, 32, 48 or 64 output channels, 12 to 64 reduction channels in steps of four, one table word of offsets, and at most 2 M
// row-channel-channel products an offset, where the tiles catch up.  Layer of 27 offsets, its rulebook there, forward / input
// gradient in us, the tensor cores (with their operands' copies and a row order) -> this kernel; and lanes that read rows and
// weights through the caches, each lane its own channel's weights (16 lines a load), which this kernel replaces:
//     channels, rows      1.2 neighbours a row                                20 - 26 neighbours a row
//     16 -> 16,  2 000   18.8 / 18.7 ->  4.7 /  4.5    4.1 /  9.0            24.0 / 23.8 -> 12.5 / 13.0    16 /  54
//     16 -> 16,  8 192   19.1 / 19.2 ->  5.2 /  5.1    5.3 /  9.2            24.4 / 24.4 -> 21.5 / 24.8    32 /  43
//     16 -> 64,  2 048   20.7 / 50.5 ->  5.5 /  6.8    6.7 / 26.9            26.9 / 84.5 -> 19.0 / 27.7    37 / 187
//     32 -> 32,  2 048   28.4 / 29.3 ->  5.4 /  5.7    7.7 /  9.8            40.0 / 40.8 -> 19.4 / 23.4    60 /  58
//     48 -> 48,    900   49.7 / 45.2 ->  6.8 /  7.0    9.4 / 18.3            77.8 / 70.6 -> 26.2 / 28.2    51 /  91
//     64 -> 64,    512   81.0 / 72.1 ->  8.7 / 10.0   18.1 / 27.6            93.5 / 84.1 -> 30.6 / 35.2   131 / 151
bool gather_gemm_small_takes(long long m_rows, int n_dim, int r_dim, int kv) {
  return kv <= 32 && n_dim % 16 == 0 && n_dim <= 64 && r_dim % 4 == 0 && r_dim > 8 && r_dim <= 64 && m_rows * n_dim * r_dim <= (2ll << 20);
}

int gather_gemm_small(const void* src, const void* w, const Epilogue& epi, const int32_t* pairs_rowmajor, void* out, long long m_rows,
                      int n_dim, int r_dim, int kv, bool transposed_weight, bool reversed, cudaStream_t st) {
  F32Params p{static_cast<const float*>(src), static_cast<const float*>(w), epi, nullptr, pairs_rowmajor, nullptr,
              static_cast<float*>(out), m_rows, n_dim, r_dim, kv, (kv + 3) & ~3, reversed ? 1 : 0};
  switch (n_dim / 16) {
    case 1: return transposed_weight ? launch_small<true, 1>(p, st) : launch_small<false, 1>(p, st);
    case 2: return transposed_weight ? launch_small<true, 2>(p, st) : launch_small<false, 2>(p, st);
    case 3: return transposed_weight ? launch_small<true, 3>(p, st) : launch_small<false, 3>(p, st);
    case 4: return transposed_weight ? launch_small<true, 4>(p, st) : launch_small<false, 4>(p, st);
  }
  return fail(SPC_ERR_UNSUPPORTED, "fp32 gather-GEMM of few rows: %d output channels", n_dim);
}

// Thin layers (at most 8 reduction channels) have kernels of their own.
bool gather_gemm_f32_supported(int n_dim, int r_dim, int dtype, int out_dtype) {
  return dtype == SPC_F32 && out_dtype == SPC_F32 && n_dim % 4 == 0 && r_dim % 4 == 0 && r_dim > 8;
}

int gather_gemm_f32(const void* src, const void* w, const Epilogue& epi, const int32_t* pairs, const int32_t* pairs_rowmajor,
                    const int32_t* order, void* out, long long m_rows, int n_dim, int r_dim, int kv, bool transposed_weight, bool reversed,
                    cudaStream_t st) {
  if (!aligned16(src) || !aligned16(w) || !aligned16(out) || !aligned16(pairs_rowmajor))
    return fail(SPC_ERR_UNSUPPORTED, "fp32 gather-GEMM: operands and the row-major table must be 16-byte aligned");
  F32Params p{static_cast<const float*>(src), static_cast<const float*>(w), epi, pairs, pairs_rowmajor, order, static_cast<float*>(out),
              m_rows, n_dim, r_dim, kv, (kv + 3) & ~3, reversed};
  const dim3 grid(static_cast<unsigned>(ceil_div(m_rows, kTile)), static_cast<unsigned>(ceil_div(n_dim, kTile)));
  if (transposed_weight) gather_gemm_f32_kernel<true><<<grid, kThreads, 0, st>>>(p);
  else gather_gemm_f32_kernel<false><<<grid, kThreads, 0, st>>>(p);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

bool wgrad_f32_supported(int c_in, int c_out, int dtype) { return dtype == SPC_F32 && c_in % 4 == 0 && c_out % 4 == 0 && c_in > 8; }

// Eight CTAs a multiprocessor (offsets differ in their pairs), no split below 2048 rows or beyond 64 of them.
WgradSplit wgrad_f32_split(int64_t n_out, int c_in, int c_out, int kv) {
  WgradSplit s;
  const int64_t tiles = static_cast<int64_t>(kv) * ceil_div(c_in, kTile) * ceil_div(c_out, kTile);
  // The centre offset of a submanifold layer has a pair a row and is the longest chain: splits short enough that one is not
  // longer than the rest of the work (SubM 64 -> 64, 100 k rows: 44 splits in offset order 136 us, 64 and the middle first 75).
  int64_t want = ceil_div(16 * static_cast<int64_t>(sm_count()), std::max<int64_t>(tiles, 1));
  want = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, n_out / 1024), 64));
  s.splits = static_cast<int>(want);
  s.rows_per_split = ceil_div(std::max<int64_t>(n_out, 1), s.splits);
  s.bytes = static_cast<size_t>(s.splits) * c_out * kv * c_in * sizeof(float);
  return s;
}

int wgrad_f32(const void* feats, const void* gout, const int32_t* pair_fwd, float* partial, int64_t n_out, int c_in, int c_out, int kv,
              const WgradSplit& s, cudaStream_t st) {
  if (!aligned16(feats) || !aligned16(gout)) return fail(SPC_ERR_UNSUPPORTED, "fp32 weight gradient: operands must be 16-byte aligned");
  const int most = 65535 / s.splits;  // offsets of a launch
  for (int turn = 0; turn < kv; turn += most) {
    const dim3 grid(static_cast<unsigned>(ceil_div(c_in, kTile)), static_cast<unsigned>(ceil_div(c_out, kTile)),
                    static_cast<unsigned>(std::min(most, kv - turn) * s.splits));
    wgrad_f32_kernel<<<grid, kThreads, 0, st>>>(static_cast<const float*>(feats), static_cast<const float*>(gout), pair_fwd, partial, n_out,
                                                c_in, c_out, kv, turn, s.splits, s.rows_per_split);
    SPC_LAUNCH_OK();
  }
  return SPC_OK;
}

}  // namespace spc
