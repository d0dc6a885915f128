// Sparse max / average pooling over implicit-gemm pair tables.
//
// HBM-bound gather-reduce.  pool_group_kernel: an output row is owned by a group
// of 4..32 lanes, each holding up to four 16-byte channel vectors; the group
// reads 32 table entries of the row with one round of loads, a ballot per load
// builds the presence mask and the lanes walk only the set bits (the entry is
// passed around by shuffle), with the gathers of two rows in flight and the
// table entries of the next row group fetched ahead.  pool_compact_kernel
// (entries compacted per CTA in shared memory, one thread per 16-byte vector)
// takes the channel counts the group shape cannot.
// Algorithmic bytes per output row: kv*4 (table) + pairs*C*e (gathered
// rows) + C*e (store).
//
// Semantics follow spconv_triton/pytorch/_impl/pool.py: the max accumulator starts at 0
// (pool.py:75-76), max backward credits every input equal to the output
// (pool.py:148-149), average divides by the number of inputs present
// (pool.py:200-201) and its backward MULTIPLIES by that count (pool.py:250-252).
// fp16/bf16/fp32 accumulate in fp32, fp64 in fp64 (pool.py:72-74).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace spc {
namespace {

template <typename T> struct PoolAcc { using type = float; };
template <> struct PoolAcc<double> { using type = double; };

template <typename T> __device__ __forceinline__ typename PoolAcc<T>::type up(T v) { return to_float(v); }
template <> __device__ __forceinline__ double up<double>(double v) { return v; }
template <typename T> __device__ __forceinline__ T down(typename PoolAcc<T>::type v) { return from_float<T>(v); }
template <> __device__ __forceinline__ double down<double>(double v) { return v; }

template <typename T, int VEC>
struct alignas(sizeof(T) * VEC) Pack { T v[VEC]; };

template <typename T, int VEC>
__device__ __forceinline__ Pack<T, VEC> load_pack(const T* p) {
  return *reinterpret_cast<const Pack<T, VEC>*>(p);
}
template <typename T, int VEC>
__device__ __forceinline__ void store_pack(T* p, const Pack<T, VEC>& v) {
  *reinterpret_cast<Pack<T, VEC>*>(p) = v;
}

// Whole-vector conversions.  The 16-bit types convert two lanes per instruction
// on the FMA pipe; one-lane conversions issue on the quarter-rate XU pipe, which
// made the gather-reduce instruction-bound.
template <typename T, int VEC>
__device__ __forceinline__ void unpack(const Pack<T, VEC>& p, typename PoolAcc<T>::type (&out)[VEC]) {
#pragma unroll
  for (int v = 0; v < VEC; ++v) out[v] = up<T>(p.v[v]);
}
template <>
__device__ __forceinline__ void unpack<__half, 8>(const Pack<__half, 8>& p, float (&out)[8]) {
  const __half2* h = reinterpret_cast<const __half2*>(p.v);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 f = __half22float2(h[q]);
    out[2 * q] = f.x;
    out[2 * q + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void unpack<__nv_bfloat16, 8>(const Pack<__nv_bfloat16, 8>& p, float (&out)[8]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p.v);
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // bf16 is the upper half of an fp32
    out[2 * q] = __uint_as_float(w[q] << 16);
    out[2 * q + 1] = __uint_as_float(w[q] & 0xffff0000u);
  }
}

template <typename T, int VEC>
__device__ __forceinline__ Pack<T, VEC> pack(const typename PoolAcc<T>::type (&in)[VEC]) {
  Pack<T, VEC> o;
#pragma unroll
  for (int v = 0; v < VEC; ++v) o.v[v] = down<T>(in[v]);
  return o;
}
template <>
__device__ __forceinline__ Pack<__half, 8> pack<__half, 8>(const float (&in)[8]) {
  Pack<__half, 8> o;
  __half2* h = reinterpret_cast<__half2*>(o.v);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2half2_rn(in[2 * q], in[2 * q + 1]);
  return o;
}
template <>
__device__ __forceinline__ Pack<__nv_bfloat16, 8> pack<__nv_bfloat16, 8>(const float (&in)[8]) {
  Pack<__nv_bfloat16, 8> o;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(o.v);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(in[2 * q], in[2 * q + 1]);
  return o;
}

// Sums of two neighbouring channels per instruction; the same IEEE results as one at a time.
__device__ __forceinline__ void add2(float& a0, float& a1, float x0, float x1) {
  asm("{\n\t.reg .b64 a, x;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 x, {%2, %3};\n\t"
      "add.rn.f32x2 a, a, x;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(a0), "+f"(a1) : "f"(x0), "f"(x1));
}
__device__ __forceinline__ void fma2(float& a0, float& a1, float x0, float x1, float w) {
  asm("{\n\t.reg .b64 a, x, w;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 x, {%2, %3};\n\tmov.b64 w, {%4, %4};\n\t"
      "fma.rn.f32x2 a, x, w, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(a0), "+f"(a1) : "f"(x0), "f"(x1), "f"(w));
}
// o = x * w + a
__device__ __forceinline__ void fma2(float x0, float x1, float w, float a0, float a1, float& o0, float& o1) {
  o0 = a0;
  o1 = a1;
  fma2(o0, o1, x0, x1, w);
}
__device__ __forceinline__ void mul2(float& o0, float& o1, float x0, float x1, float w) {
  asm("{\n\t.reg .b64 o, x, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 w, {%4, %4};\n\t"
      "mul.rn.f32x2 o, x, w;\n\tmov.b64 {%0, %1}, o;\n\t}"
      : "=f"(o0), "=f"(o1) : "f"(x0), "f"(x1), "f"(w));
}

// a + x in one instruction; x is exact in fp32.
__device__ __forceinline__ void add_mixed(float& a, __half x) { asm("add.rn.f32.f16 %0, %1, %0;" : "+f"(a) : "h"(__half_as_ushort(x))); }
__device__ __forceinline__ void add_mixed(float& a, __nv_bfloat16 x) { asm("add.rn.f32.bf16 %0, %1, %0;" : "+f"(a) : "h"(__bfloat16_as_ushort(x))); }

// a / d for a whole number d, correctly rounded by one correction of a * (1 / d) with the exact remainder
// (Markstein 1990), two channels an instruction, instead of a division's ten instructions a value: a window
// of few present rows spent a quarter of its time there.  Used where the quotient is then rounded to 16 bits;
// where the remainder is no number (an infinity), the quotient is a * (1 / d).
template <int VEC>
__device__ __forceinline__ void divide_by_count(float (&a)[VEC], float d) {
  const float inverse = 1.f / d;
  float q[VEC], check0 = 0.f, check1 = 0.f;
#pragma unroll
  for (int v = 0; v < VEC; v += 2) {
    float rest0 = a[v], rest1 = a[v + 1];
    mul2(q[v], q[v + 1], a[v], a[v + 1], inverse);
    fma2(rest0, rest1, q[v], q[v + 1], -d);
    add2(check0, check1, rest0, rest1);
    fma2(rest0, rest1, inverse, q[v], q[v + 1], a[v], a[v + 1]);
  }
  if (check0 + check1 == check0 + check1) return;
#pragma unroll
  for (int v = 0; v < VEC; ++v)
    if (!(a[v] == a[v])) a[v] = q[v];
}

enum PoolOp { kMaxFwd = 0, kAvgFwd = 1, kAvgBwd = 2, kMaxBwd = 3 };
// Independent 16-byte gathers one thread keeps in flight (rows in flight = in_flight / U), and
// 16-byte vectors of a row one thread owns, per operator; each pair is the measured best on B200
// for 512-byte rows (C = 256 fp16): max forward has few present entries per row and gains from
// four rows in flight with two vectors each (0.26 ms = 0.81 of the copy peak, against 0.31 with
// 4 x 2); average forward over a 3^3 window prefers two vectors and two rows; max backward
// reads two rows per entry and keeps its own row in registers: one vector and one row per thread
// (more resident threads) is best for it.  `ctas` per SM bounds the registers (0: the
// compiler's choice): the forward average issues
// instructions most of the time and gains by a fourth CTA (1.1 M rows of 512 bytes, 7.4 entries: 494 to 447 us,
// 565 before its sums and quotients were packed), its gradient, bound by L2, loses by it (439 to 547).
template <int OP> struct PoolTune;
template <> struct PoolTune<0> { static constexpr int in_flight = 8, max_u = 2, ctas = 3; };  // kMaxFwd
template <> struct PoolTune<1> { static constexpr int in_flight = 4, max_u = 2, ctas = 4; };  // kAvgFwd
template <> struct PoolTune<2> { static constexpr int in_flight = 8, max_u = 2, ctas = 3; };  // kAvgBwd
template <> struct PoolTune<3> { static constexpr int in_flight = 1, max_u = 1, ctas = 0; };  // kMaxBwd
constexpr int kChunk = 32;    // table entries of one row compacted per pass (one per lane)
constexpr int kMaxRows = 64;  // rows per CTA

// What the four operators do with the rows their table names:
//   kMaxFwd : dst[row] = max(0, src[j])                        table = pair_fwd
//   kAvgFwd : dst[row] = sum(src[j]) / max(1, #j), aux_out=#j  table = pair_fwd
//   kMaxBwd : dst[row] = sum(src[o] where own[row]==ref[o])    table = pair_bwd, src = grad_out, ref = pooled
//   kAvgBwd : dst[row] = sum(src[o] * aux_in[o])               table = pair_bwd, src = grad_out
//
// One thread owns U 16-byte channel vectors of one row, spaced so that the
// threads of a row read contiguous 16*nt bytes per load; a random 512-byte
// row needs several loads in flight per thread to cover HBM latency, and the
// table walk is paid once per U vectors.
template <typename T, int VEC, int U, int OP>
struct PoolRow {
  using A = typename PoolAcc<T>::type;
  A acc[U][VEC];
  Pack<T, VEC> f[U];
  int total = 0;

  __device__ __forceinline__ void begin(const T* own, long long row, int channels, int c0, int cstep) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[u][v] = A(0);
      if (OP == kMaxBwd) f[u] = load_pack<T, VEC>(own + row * channels + c0 + u * cstep);
    }
  }

  // B rows at once (entries < 0 are skipped); B * U loads are issued before the first use.
  template <int B>
  __device__ __forceinline__ void gather(const int (&j)[B], const T* src, const T* ref, const int32_t* aux_in,
                                         int channels, int c0, int cstep) {
    Pack<T, VEC> pk[B][U], rk[B][U];
    A w[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      if (j[b] < 0) continue;
      const long long off = static_cast<long long>(j[b]) * channels + c0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        pk[b][u] = load_pack<T, VEC>(src + off + u * cstep);
        if (OP == kMaxBwd) rk[b][u] = load_pack<T, VEC>(ref + off + u * cstep);
      }
      if (OP == kAvgBwd) w[b] = static_cast<A>(__ldg(&aux_in[j[b]]));
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      if (j[b] < 0) continue;
      ++total;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if constexpr (OP == kAvgFwd && sizeof(T) == 2) {
#pragma unroll
          for (int v = 0; v < VEC; ++v) add_mixed(acc[u][v], pk[b][u].v[v]);
          continue;
        }
        A x[VEC], r[VEC], o[VEC];
        unpack<T, VEC>(pk[b][u], x);
        if (OP == kMaxBwd) {
          unpack<T, VEC>(rk[b][u], r);
          unpack<T, VEC>(f[u], o);
        }
        if constexpr ((OP == kAvgFwd || OP == kAvgBwd) && VEC % 2 == 0 && std::is_same<A, float>::value) {
#pragma unroll
          for (int v = 0; v < VEC; v += 2) {
            if (OP == kAvgFwd) add2(acc[u][v], acc[u][v + 1], x[v], x[v + 1]);
            else fma2(acc[u][v], acc[u][v + 1], x[v], x[v + 1], w[b]);
          }
          continue;
        }
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          if (OP == kMaxFwd) acc[u][v] = x[v] > acc[u][v] ? x[v] : acc[u][v];
          else if (OP == kAvgFwd) acc[u][v] += x[v];
          else if (OP == kMaxBwd) { if (r[v] == o[v]) acc[u][v] += x[v]; }
          else acc[u][v] += x[v] * w[b];
        }
      }
    }
  }

  __device__ __forceinline__ void finish(T* dst, int32_t* aux_out, long long row, int channels, int c0,
                                         int cstep) {
    const A d = static_cast<A>(total > 1 ? total : 1);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if constexpr (OP == kAvgFwd && sizeof(T) == 2 && VEC % 2 == 0) {
        divide_by_count<VEC>(acc[u], d);
      } else if (OP == kAvgFwd) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[u][v] /= d;
      }
      store_pack<T, VEC>(dst + row * channels + c0 + u * cstep, pack<T, VEC>(acc[u]));
    }
    if (OP == kAvgFwd && aux_out != nullptr && c0 == 0) aux_out[row] = total;
  }
};

// Launch geometry of the shared-memory kernel: `nt` threads per row (U vectors
// each), of which a CTA holds `tpb` (grid.y covers the rest), `rpb` rows per CTA.
struct PoolGeom { int nt, tpb, rpb; };

// Rows whose nt threads are a power of two between 4 and 32 (every channel count
// from 128 bytes to 2 KiB that is a multiple of 64 bytes): the nt lanes of a row
// read up to 32 table entries of the row with ONE round of loads (lane l takes
// entries l, l+nt, ...), a ballot per load builds the row's 32-bit presence
// mask, and the lanes then walk only the set bits, fetching each index from its
// owner lane by shuffle.  No shared memory, no CTA barrier.
// Each warp takes kGroupIters consecutive row groups and loads the table entries
// of the next group before it gathers for the current one, so a table latency is
// exposed once per warp and gathers are in flight the rest of the time.
constexpr int kGroupIters = 8;  // row groups per warp

template <typename T, int VEC, int U, int OP, int LGNT>
__global__ void __launch_bounds__(256, PoolTune<OP>::ctas)
pool_group_kernel(const T* __restrict__ src, const T* __restrict__ own, const T* __restrict__ ref,
                  const int32_t* __restrict__ table, const int32_t* __restrict__ order, const int32_t* __restrict__ aux_in,
                  T* __restrict__ dst, int32_t* __restrict__ aux_out, long long n_rows, int channels, int kv, long long sk, int sr) {
  // the threads per row are a compile-time power of two: the entry loops below unroll to
  // exactly 32 / nt loads, ballots and selects
  constexpr int lg_nt = LGNT;
  constexpr int kE = 32 >> LGNT;  // table entries per lane per round == rows per warp
  constexpr int B = PoolTune<OP>::in_flight / U > 0 ? PoolTune<OP>::in_flight / U : 1;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int nt = 1 << lg_nt;
  const int lane = threadIdx.x & 31;
  const int kl = lane & (nt - 1), gbase = lane - kl;
  const unsigned gmask = nt == 32 ? kFull : ((1u << nt) - 1u);
  const int c0 = kl * VEC, cstep = nt * VEC;
  constexpr int per_lane = kE;
  const long long warp_id = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long row_first = warp_id * kGroupIters * per_lane + (lane >> lg_nt);
  // The average's kernels keep the rows of the warp's groups in registers, requested at once where there is an
  // order; the forward pass, which has none, still gains by the shorter row arithmetic (505 to 450 us), the
  // maximum loses (116 to 144 and 216 to 268 us).
  constexpr bool kOrdered = OP == kAvgBwd || OP == kAvgFwd;
  int rows_of[(kGroupIters * kE + 31) / 32];
#pragma unroll
  for (int i = 0; i < (kGroupIters * kE + 31) / 32; ++i) {
    const long long slot = warp_id * kGroupIters * per_lane + i * 32 + lane;
    rows_of[i] = !kOrdered || order == nullptr ? static_cast<int>(slot) : (i * 32 + lane < kGroupIters * kE && slot < n_rows ? __ldg(&order[slot]) : 0);
  }
  auto row_at = [&](int it) {
    if (!kOrdered) return row_first + static_cast<long long>(it) * per_lane;
    const int at = it * kE + (lane >> lg_nt);
    int r = __shfl_sync(kFull, rows_of[0], at & 31);
#pragma unroll
    for (int i = 1; i < (kGroupIters * kE + 31) / 32; ++i) {
      const int other = __shfl_sync(kFull, rows_of[i], at & 31);
      r = (at >> 5) == i ? other : r;
    }
    return static_cast<long long>(r);
  };

  auto load_entries = [&](long long row, bool there, int k0, int (&v)[kE]) {
#pragma unroll
    for (int e = 0; e < kE; ++e) {
      const int k = k0 + e * nt + kl;
      v[e] = (there && k < kv) ? __ldg(&table[k * sk + row * sr]) : -1;
    }
  };

  int vn[kE];
  long long next = row_at(0);
  load_entries(next, row_first < n_rows, 0, vn);
#pragma unroll 1
  for (int it = 0; it < kGroupIters; ++it) {
    const long long slot = row_first + static_cast<long long>(it) * per_lane;
    if (slot - (lane >> lg_nt) >= n_rows) break;  // warp-uniform: the whole group is past the end
    const bool live = slot < n_rows;
    const long long row = kOrdered ? next : slot;
    int v[kE];
#pragma unroll
    for (int e = 0; e < kE; ++e) v[e] = vn[e];
    if (it + 1 < kGroupIters) {
      if (kOrdered) next = row_at(it + 1);
      load_entries(kOrdered ? next : slot + per_lane, slot + per_lane < n_rows, 0, vn);
    }

    PoolRow<T, VEC, U, OP> pr;
    if (live) pr.begin(own, row, channels, c0, cstep);
    for (int k0 = 0; k0 < kv; k0 += 32) {
      if (k0 != 0) load_entries(row, live, k0, v);
      unsigned gm = 0;
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        if (e < per_lane) {  // warp-uniform
          const unsigned m = __ballot_sync(kFull, v[e] >= 0);
          gm |= ((m >> gbase) & gmask) << (e * nt);
        }
      }
      while (__any_sync(kFull, gm != 0)) {
        int j[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const int p = gm ? __ffs(gm) - 1 : 0;
          const int e = p >> lg_nt;
          int mine = v[0];
#pragma unroll
          for (int q = 1; q < kE; ++q) mine = e == q ? v[q] : mine;
          const int got = __shfl_sync(kFull, mine, gbase + (p & (nt - 1)));
          j[b] = gm ? got : -1;
          gm &= gm - 1;
        }
        pr.template gather<B>(j, src, ref, aux_in, channels, c0, cstep);
      }
    }
    if (live) pr.finish(dst, aux_out, row, channels, c0, cstep);
  }
}

// Every other channel count.  Tables are mostly -1 (a 3^3 stride-1 pool over a
// LiDAR scene has about 3 of 27 entries present), so walking them per thread costs
// far more instructions than the gathers.  The CTA stages the [kv, rpb] tile of the
// table with coalesced loads, one warp per row compacts the entries that are
// present with a ballot (order of k preserved, so sums are formed in the same
// order as a plain walk), and every thread then reads only the compacted list.
template <typename T, int VEC, int U, int OP>
__global__ void __launch_bounds__(256)
pool_compact_kernel(const T* __restrict__ src, const T* __restrict__ own, const T* __restrict__ ref,
                    const int32_t* __restrict__ table, const int32_t* __restrict__ order, const int32_t* __restrict__ aux_in, T* __restrict__ dst,
                    int32_t* __restrict__ aux_out, long long n_rows, int channels, int kv, long long sk, int sr,
                    PoolGeom g) {
  constexpr int B = PoolTune<OP>::in_flight / U > 0 ? PoolTune<OP>::in_flight / U : 1;
  __shared__ int32_t tab[kChunk][kMaxRows + 1];
  __shared__ int32_t lst[kMaxRows][kChunk];
  __shared__ int32_t cnt[kMaxRows];
  const int t = threadIdx.x, nthr = blockDim.x;
  const int lane = t & 31, warp = t >> 5, nwarps = nthr >> 5;
  const long long row0 = static_cast<long long>(blockIdx.x) * g.rpb;
  const int rl = t / g.tpb;
  const int ct = t - rl * g.tpb + static_cast<int>(blockIdx.y) * g.tpb;
  const bool live = rl < g.rpb && row0 + rl < n_rows && ct < g.nt;
  const long long row = OP == kAvgBwd && order != nullptr && live ? __ldg(&order[row0 + rl]) : row0 + rl;
  const int c0 = ct * VEC, cstep = g.nt * VEC;

  PoolRow<T, VEC, U, OP> pr;
  if (live) pr.begin(own, row, channels, c0, cstep);

  for (int k0 = 0; k0 < kv; k0 += kChunk) {
    const int kc = min(kChunk, kv - k0);
    if (k0 != 0) __syncthreads();
    for (int i = t; i < kc * g.rpb; i += nthr) {
      // consecutive threads read consecutive entries of the table
      const int k = sr == 1 ? i / g.rpb : i % kc, r = sr == 1 ? i - k * g.rpb : i / kc;
      const bool there = row0 + r < n_rows;
      const long long rr = OP == kAvgBwd && there && order != nullptr ? __ldg(&order[row0 + r]) : row0 + r;
      tab[k][r] = there ? __ldg(&table[(k0 + k) * sk + rr * sr]) : -1;
    }
    __syncthreads();
    for (int r = warp; r < g.rpb; r += nwarps) {
      const int v = lane < kc ? tab[lane][r] : -1;
      const unsigned m = __ballot_sync(0xffffffffu, v >= 0);
      if (v >= 0) lst[r][__popc(m & ((1u << lane) - 1u))] = v;
      if (lane == 0) cnt[r] = __popc(m);
    }
    __syncthreads();
    if (!live) continue;
    const int n = cnt[rl];
    for (int i = 0; i < n; i += B) {
      int j[B];
#pragma unroll
      for (int b = 0; b < B; ++b) j[b] = i + b < n ? lst[rl][i + b] : -1;
      pr.template gather<B>(j, src, ref, aux_in, channels, c0, cstep);
    }
  }
  if (live) pr.finish(dst, aux_out, row, channels, c0, cstep);
}

// Rows in the order of the rows they read: by the first present entry of their table row, in up to 8192
// buckets of neighbouring targets, any order inside a bucket.
constexpr int kOrderBuckets = 8192;

__global__ void __launch_bounds__(1024) clear_buckets_kernel(int* counts) { counts[blockIdx.x * 1024 + threadIdx.x] = 0; }

__global__ void __launch_bounds__(256)
count_buckets_kernel(const int4* __restrict__ table, int words, int n_rows, int shift, int* __restrict__ counts,
                     int2* __restrict__ placed) {
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= n_rows) return;
  int first = 0;  // a row that reads nothing goes anywhere
  for (int q = 0; q < words; ++q) {
    const int4 e = __ldg(&table[static_cast<long long>(r) * words + q]);
    const int hit = e.x >= 0 ? e.x : e.y >= 0 ? e.y : e.z >= 0 ? e.z : e.w;  // (beyond kv the table holds -1)
    if (hit >= 0) {
      first = hit;
      break;
    }
  }
  const int b = first >> shift;
  placed[r] = make_int2(b, atomicAdd(&counts[b], 1));
}

__global__ void __launch_bounds__(1024) scan_buckets_kernel(int* counts) {
  __shared__ int sums[32];
  constexpr int kEach = kOrderBuckets / 1024;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int c[kEach], own = 0;
#pragma unroll
  for (int i = 0; i < kEach; ++i) {
    c[i] = counts[t * kEach + i];
    own += c[i];
  }
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  int before = incl - own;
  for (int w = 0; w < warp; ++w) before += sums[w];
#pragma unroll
  for (int i = 0; i < kEach; ++i) {
    counts[t * kEach + i] = before;
    before += c[i];
  }
}

__global__ void __launch_bounds__(256)
deal_buckets_kernel(const int2* __restrict__ placed, const int* __restrict__ starts, int n_rows, int32_t* __restrict__ order) {
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= n_rows) return;
  const int2 p = placed[r];
  order[starts[p.x] + p.y] = r;
}

template <typename T>
int vec_for(int channels, const void* a, const void* b, const void* c = nullptr, const void* d = nullptr) {
  constexpr int full = 16 / sizeof(T);
  auto aligned = [](const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (channels % full == 0 && aligned(a) && aligned(b) && aligned(c) && aligned(d)) return full;
  return 1;
}

template <typename T, int VEC, int U, int OP>
void pool_launch_u(const T* src, const T* own, const T* ref, const int32_t* table, const int32_t* order, const int32_t* aux_in, T* dst,
                   int32_t* aux_out, int64_t n_rows, int channels, int kv, int pitch, cudaStream_t st) {
  const long long sk = pitch ? 1 : n_rows;
  const int sr = pitch ? pitch : 1;
  PoolGeom g;
  g.nt = channels / (VEC * U);
  g.tpb = std::min(g.nt, 256);
  g.rpb = std::min(kMaxRows, std::max(1, 256 / g.tpb));
  const int threads = static_cast<int>(ceil_div(static_cast<long long>(g.tpb) * g.rpb, 32) * 32);
  const dim3 grid(static_cast<unsigned>(ceil_div(static_cast<long long>(n_rows), g.rpb)),
                  static_cast<unsigned>(ceil_div(g.nt, g.tpb)));
  if (g.nt >= 4 && g.nt <= 32 && (g.nt & (g.nt - 1)) == 0) {
    int lg = 0;
    while ((1 << lg) < g.nt) ++lg;
    const long long warps = ceil_div(static_cast<long long>(n_rows), (32 >> lg) * kGroupIters);
    const unsigned blocks = static_cast<unsigned>(ceil_div(warps, 8));
    switch (lg) {
      case 2: pool_group_kernel<T, VEC, U, OP, 2><<<blocks, 256, 0, st>>>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, sk, sr); break;
      case 3: pool_group_kernel<T, VEC, U, OP, 3><<<blocks, 256, 0, st>>>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, sk, sr); break;
      case 4: pool_group_kernel<T, VEC, U, OP, 4><<<blocks, 256, 0, st>>>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, sk, sr); break;
      default: pool_group_kernel<T, VEC, U, OP, 5><<<blocks, 256, 0, st>>>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, sk, sr); break;
    }
  } else {
    pool_compact_kernel<T, VEC, U, OP><<<grid, threads, 0, st>>>(src, own, ref, table, order, aux_in, dst, aux_out,
                                                                n_rows, channels, kv, sk, sr, g);
  }
}

template <typename T, int OP>
int pool_launch(const void* src_, const void* own_, const void* ref_, const int32_t* table, const int32_t* order,
                const int32_t* aux_in, void* dst_, int32_t* aux_out, int64_t n_rows, int channels, int kv, int pitch,
                cudaStream_t st) {
  constexpr int full = 16 / sizeof(T);
  const T* src = static_cast<const T*>(src_);
  const T* own = static_cast<const T*>(own_);
  const T* ref = static_cast<const T*>(ref_);
  T* dst = static_cast<T*>(dst_);
  if (vec_for<T>(channels, src_, own_, ref_, dst_) != full) {
    pool_launch_u<T, 1, 1, OP>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, pitch, st);
  } else {
    // most vectors per thread that still leave a row at least 4 threads (the warp-group kernel)
    const int tpr = channels / full;
    int u = PoolTune<OP>::max_u;
    while (u > 1 && (tpr % u != 0 || tpr / u < 4)) u /= 2;
    if (u == 4)
      pool_launch_u<T, full, 4, OP>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, pitch, st);
    else if (u == 2)
      pool_launch_u<T, full, 2, OP>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, pitch, st);
    else
      pool_launch_u<T, full, 1, OP>(src, own, ref, table, order, aux_in, dst, aux_out, n_rows, channels, kv, pitch, st);
  }
  SPC_LAUNCH_OK();
  return SPC_OK;
}

#define SPC_POOL_DISPATCH(dtype, CALL)                                        \
  switch (dtype) {                                                            \
    case SPC_F16: { using T = __half; return CALL; }                          \
    case SPC_BF16: { using T = __nv_bfloat16; return CALL; }                  \
    case SPC_F32: { using T = float; return CALL; }                           \
    case SPC_F64: { using T = double; return CALL; }                          \
    default: return fail(SPC_ERR_UNSUPPORTED, "pool: dtype %d not supported", dtype); \
  }

bool pool_args_ok(const void* a, const void* b, const void* c, int64_t n, int channels, int kv) {
  return a && b && c && n >= 0 && channels > 0 && kv > 0;
}

}  // namespace
}  // namespace spc

using namespace spc;

extern "C" int spc_maxpool_forward(const void* features, const int32_t* pair_fwd, void* out, int64_t n_out,
                                   int channels, int kv, int dtype, void* stream) {
  if (!pool_args_ok(features, pair_fwd, out, n_out, channels, kv))
    return fail(SPC_ERR_INVALID_ARGUMENT, "maxpool_forward: bad arguments");
  if (n_out == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SPC_POOL_DISPATCH(dtype, (pool_launch<T, kMaxFwd>(features, nullptr, nullptr, pair_fwd, nullptr, nullptr, out, nullptr, n_out, channels, kv, 0, st)));
}

extern "C" int spc_avgpool_forward(const void* features, const int32_t* pair_fwd, void* out, int32_t* count,
                                   int64_t n_out, int channels, int kv, int dtype, void* stream) {
  if (!pool_args_ok(features, pair_fwd, out, n_out, channels, kv))
    return fail(SPC_ERR_INVALID_ARGUMENT, "avgpool_forward: bad arguments");
  if (n_out == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SPC_POOL_DISPATCH(dtype, (pool_launch<T, kAvgFwd>(features, nullptr, nullptr, pair_fwd, nullptr, nullptr, out, count, n_out, channels, kv, 0, st)));
}

extern "C" int spc_maxpool_backward(const void* features, const void* out_features, const void* grad_out,
                                    const int32_t* pair_bwd, void* din, int64_t n_in, int channels, int kv,
                                    int dtype, void* stream) {
  if (!pool_args_ok(features, pair_bwd, din, n_in, channels, kv) || !out_features || !grad_out)
    return fail(SPC_ERR_INVALID_ARGUMENT, "maxpool_backward: bad arguments");
  if (n_in == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SPC_POOL_DISPATCH(dtype, (pool_launch<T, kMaxBwd>(grad_out, features, out_features, pair_bwd, nullptr, nullptr, din, nullptr, n_in, channels, kv, 0, st)));
}

extern "C" int spc_avgpool_backward(const void* grad_out, const int32_t* pair_bwd, const int32_t* count,
                                    void* din, int64_t n_in, int channels, int kv, int dtype, void* stream) {
  if (!pool_args_ok(grad_out, pair_bwd, din, n_in, channels, kv) || !count)
    return fail(SPC_ERR_INVALID_ARGUMENT, "avgpool_backward: bad arguments");
  if (n_in == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SPC_POOL_DISPATCH(dtype, (pool_launch<T, kAvgBwd>(grad_out, nullptr, nullptr, pair_bwd, nullptr, count, din, nullptr, n_in, channels, kv, 0, st)));
}

extern "C" int spc_pool(int op, const void* src, const void* own, const void* ref, const int32_t* table, int pitch,
                        const int32_t* order, const int32_t* aux_in, void* dst, int32_t* aux_out, int64_t n_rows, int channels, int kv,
                        int dtype, void* stream) {
  if (!pool_args_ok(src, table, dst, n_rows, channels, kv) || (pitch != 0 && pitch < kv) || op < kMaxFwd || op > kMaxBwd ||
      (op == kMaxBwd && (!own || !ref)) || (op == kAvgBwd && !aux_in) || (order != nullptr && op != kAvgBwd))
    return fail(SPC_ERR_INVALID_ARGUMENT, "pool: bad arguments");
  if (n_rows == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (op) {
    case kMaxFwd: SPC_POOL_DISPATCH(dtype, (pool_launch<T, kMaxFwd>(src, nullptr, nullptr, table, order, nullptr, dst, nullptr, n_rows, channels, kv, pitch, st)));
    case kAvgFwd: SPC_POOL_DISPATCH(dtype, (pool_launch<T, kAvgFwd>(src, nullptr, nullptr, table, order, nullptr, dst, aux_out, n_rows, channels, kv, pitch, st)));
    case kAvgBwd: SPC_POOL_DISPATCH(dtype, (pool_launch<T, kAvgBwd>(src, nullptr, nullptr, table, order, aux_in, dst, nullptr, n_rows, channels, kv, pitch, st)));
    default: SPC_POOL_DISPATCH(dtype, (pool_launch<T, kMaxBwd>(src, own, ref, table, order, nullptr, dst, nullptr, n_rows, channels, kv, pitch, st)));
  }
}

extern "C" size_t spc_pool_row_order_workspace_bytes(int64_t n_rows) {
  return kOrderBuckets * sizeof(int) + static_cast<size_t>(std::max<int64_t>(n_rows, 0)) * sizeof(int2);
}

extern "C" int spc_pool_row_order(const int32_t* table, int pitch, int kv, int64_t n_rows, int64_t n_targets, int32_t* order,
                                  void* workspace, size_t workspace_bytes, void* stream) {
  if (!table || !order || !workspace || pitch < kv || pitch % 4 != 0 || kv <= 0 || n_rows < 0 || n_rows >= (1ll << 31) ||
      n_targets <= 0 || n_targets >= (1ll << 31) || workspace_bytes < spc_pool_row_order_workspace_bytes(n_rows) ||
      ((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(workspace)) & 15u))
    return fail(SPC_ERR_INVALID_ARGUMENT, "pool_row_order: bad arguments");
  if (n_rows == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* counts = static_cast<int*>(workspace);
  int2* placed = reinterpret_cast<int2*>(counts + kOrderBuckets);
  int shift = 0;
  while (((n_targets - 1) >> shift) >= kOrderBuckets) ++shift;
  const unsigned blocks = static_cast<unsigned>(ceil_div(n_rows, 256));
  clear_buckets_kernel<<<kOrderBuckets / 1024, 1024, 0, st>>>(counts);
  SPC_LAUNCH_OK();
  count_buckets_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<const int4*>(table), pitch / 4, static_cast<int>(n_rows), shift, counts, placed);
  SPC_LAUNCH_OK();
  scan_buckets_kernel<<<1, 1024, 0, st>>>(counts);
  SPC_LAUNCH_OK();
  deal_buckets_kernel<<<blocks, 256, 0, st>>>(placed, counts, static_cast<int>(n_rows), order);
  SPC_LAUNCH_OK();
  return SPC_OK;
}
