// Implicit gather-GEMM on tcgen05 for layers whose rows are one stage (at most 128 bytes: 64 channels of 16 bits):
//
//   out[rm, n] = sum_k sum_r src[pairs[k, rm], r] * B_k[r, n]  (+ epilogue)
//
// forward and, with the weight read transposed, for the input gradient, as gemm_tma.cu.
//
// Bound.  A tile of 128 rows has one stage per kernel offset that any of its rows has: 1.3 - 1.5 stages in a strided
// layer's output or a sparse scene, 13 - 18 in a dense one.  With few stages a tile is a chain of latencies (row order,
// table entries, gather, multiplication, epilogue), with many the shared-memory pipe (16 KB of rows and 8 KB of weights
// written and read again per stage at 64 -> 64) and the issue of the copies.  So a CTA stays on the chip and takes every
// grid-th tile, and each link of the chain has warps of its own, a tile or more ahead of the next:
//   * warps 0-3, epilogue: a thread reads a row of one of two accumulators; the other is multiplied into meanwhile.
//   * warps 4-7, tables: the row-major entries of the next tile's rows (eight or four lanes a row) are on their way while
//     those of this one are dealt to a buffer in the order in which the copies read them, with the vote on the offsets.
//   * warps 8-10, copies: a stage each in turn: 128 rows by 16-byte cp.async and the weight slab by TMA, both
//     completing on the stage's barrier.
//   * warp 11: tcgen05.mma and the commits.
// Two CTAs of 384 threads fit a multiprocessor with 80 registers a thread (three warps each on a sub-partition).  All waits
// are bounded; after one has run out a warp leaves its loop, the others' waits run out in turn, and everything in flight
// is awaited before tensor memory goes back.
//
// Measured (one B200, us, alone, L2 cold; the kernel of one tile a CTA in gemm_tma.cu -> this one): strided 64 -> 128, 1.36 M
// rows with 1.4 stages a tile 289 -> 213; 32 -> 64, 1.47 M rows 154 -> 139; other sizes beside the rule at the end.  Wider rows
// stay there: with several stages an offset the multiplications cover the chain, and two accumulators cost the third CTA or
// stage (128 -> 128 on 74 k rows 33 -> 52).
//
// Measured and dropped: tables and epilogue by the same warps (57 -> 84 us at 64 -> 64: one chain again, and 32 unrolled
// offsets a tile are more instructions than the fetch keeps up with); table entries copied row by row with cp.async and
// read from there, stores by warps of their own (178 -> 227: a copy thread then reads an entry a row instead of four at once);
// stores by cp.async.bulk (about 48 cycles per row and multiprocessor); fewer table warps and more copy warps (equal or
// slower); two waves of CTAs instead of one (+ 2 - 5 % of the kernel alone); test_wait or nanosleep instead of try_wait (+ 5 %).
// A tcgen05.ld waits for the global stores that its warp has under way (17 -> 250 cycles on an idle chip, over 1 000 on a
// busy one), which is what is left of the epilogue of rows wider than its 128-byte passes.
#include <algorithm>

#include "common.cuh"
#include "gemm_internal.cuh"
#include "gemm_tma_common.cuh"

namespace spc {
namespace {

using namespace tc;

struct StreamParams {
  const void* src;
  Epilogue epi;
  const int32_t* pairs;
  const int32_t* pairs_rm;  // optional row-major copy [m_rows, kvp]
  const int32_t* order;
  void* out;
  int m_rows, tiles;
  int kvp;
  int n_dim, kv;
  int reversed;  // offset k of the table meets weight kv - 1 - k
  int stages, a_stage_bytes, b_stage_bytes;
  int copiers;     // copy warps at work: no more than there are stages (a slot's last round but one must be over)
  int acc_cols, tmem_cols;  // columns of one accumulator and of both
  int epi_bytes;   // bytes of a row that the epilogue passes through shared memory at a time: 32, 64 or 128, and 16 channels at least
  int epi_pad;     // output channels rounded up to 16; sizes the epilogue scale / shift arrays
  int b_row_bytes;  // swizzle span of the MN-major B rows
  int* status;
};

constexpr int kEpiWarps = 4, kTableWarps = 4, kCopyWarps = 3;
constexpr int kFirstTable = kEpiWarps, kFirstCopy = kFirstTable + kTableWarps, kMmaWarp = kFirstCopy + kCopyWarps;
constexpr int kThreads = (kMmaWarp + 1) * 32;
constexpr int kPassBytes = 32 * 16;  // one copy per lane covers this much of a tile
constexpr int kTables = 2;           // table buffers
constexpr int kAccs = 2;             // accumulators

// Barriers of a CTA, as numbers from the first.
constexpr int kBarFull = 0, kBarEmpty = kMaxStages, kBarTabFull = 2 * kMaxStages, kBarTabEmpty = kBarTabFull + kTables,
              kBarAccFull = kBarTabEmpty + kTables, kBarAccEmpty = kBarAccFull + kAccs, kBarDrain = kBarAccEmpty + kAccs,
              kBars = kBarDrain + 1;

// Position in a ring of n entries and the parity of its present round.
struct Ring {
  int at = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next(int n) {
    if (++at == n) {
      at = 0;
      parity ^= 1;
    }
  }
};

// (read where it is used: hoisted, the sixteen factors and shifts of a chunk would spill)
__device__ __forceinline__ float4 lds4(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
  return v;
}

// Offsets whose table entries go through shared memory together: a whole 3 x 3 x 3 kernel where the stages are small, half of
// it where the room is a stage more (the strided 64 -> 128 above: 235 us with whole kernels, 213 with halves; 32 -> 64: 139 whole,
// 152 halves).
__host__ __device__ constexpr int table_group(int lanes_per_row) { return lanes_per_row == 8 ? 16 : 32; }

// LPR: lanes per row = 16-byte pieces of one A row in a stage (8, 4 or 2 for rows of 128, 64 or 32 bytes).
template <typename T, typename TO, bool B_MN, int LPR>
__global__ void __launch_bounds__(kThreads, 2)
gather_gemm_stream_kernel(const __grid_constant__ StreamParams p, const __grid_constant__ CUtensorMap map_b) {
  constexpr int ELEM = sizeof(T);
  constexpr int UMMA_K = 32 / ELEM;
  constexpr int A_ROW_BYTES = 16 * LPR;
  constexpr int EPR = A_ROW_BYTES / ELEM;    // reduction elements
  constexpr int kRowsPass = 32 / LPR;        // rows that one copy per lane covers: 4, 8, 16
  constexpr int CP = kTileM / kRowsPass;     // copies per thread and stage: 32, 16, 8
  constexpr int KSTEPS = A_ROW_BYTES / 32;   // tcgen05.mma instructions per stage
  constexpr int GROUP = table_group(LPR);

  extern __shared__ uint8_t smem_raw[];
  // (an offset, not a rounded pointer: the compiler keeps knowing that these are shared-memory addresses)
  uint8_t* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int stage_bytes = p.a_stage_bytes + p.b_stage_bytes;
  const int group_rows = min(p.kv, GROUP);
  int* const tables = reinterpret_cast<int*>(smem + static_cast<size_t>(p.stages) * stage_bytes);  // [kTables][group_rows][128]
  uint8_t* const slabs = reinterpret_cast<uint8_t*>(tables + kTables * group_rows * kTileM);       // [128][epi_bytes]
  float* const epi_scale = reinterpret_cast<float*>(slabs + kTileM * p.epi_bytes);                 // [epi_pad]
  float* const epi_shift = epi_scale + p.epi_pad;  // [epi_pad] per-channel shift (bias folded in)
  uint32_t* const votes = reinterpret_cast<uint32_t*>(epi_shift + p.epi_pad);  // [kTables][4] offsets that rows of a warp have
  uint64_t* const bars = reinterpret_cast<uint64_t*>(votes + 4 * kTables);
  int* const acc_any = reinterpret_cast<int*>(bars + kBars);                   // [kAccs] whether anything was multiplied
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(acc_any + kAccs);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  // (one thread's reading, acted on by the whole CTA below: threads that saw different values must not part)
  const int stopped = tid == 32 ? *reinterpret_cast<volatile int*>(p.status) : 0;
  const uint32_t bar0 = smem_u32(bars);
  const auto bar = [bar0](int i) { return bar0 + 8u * i; };

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(bar(kBarFull + s), 32 + 1);  // every lane of the stage's copy warp + the weight slab
      mbar_init(bar(kBarEmpty + s), 1);
    }
    for (int s = 0; s < kTables; ++s) {
      mbar_init(bar(kBarTabFull + s), kTableWarps);
      mbar_init(bar(kBarTabEmpty + s), p.copiers + 1);
    }
    for (int s = 0; s < kAccs; ++s) {
      mbar_init(bar(kBarAccFull + s), 2);  // the multiplications, and the thread that issued them
      mbar_init(bar(kBarAccEmpty + s), kEpiWarps);
    }
    mbar_init(bar(kBarDrain), 1);
    fence_mbar_init();
    prefetch_tensormap(&map_b);
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish();
  }
  const bool has_epilogue = p.epi.bias != nullptr || p.epi.shift != nullptr || p.epi.act != SPC_ACT_NONE;
  if (has_epilogue) stage_epilogue<T>(p.epi, p.n_dim, epi_scale, epi_shift, tid, kThreads);
  tc_fence_before();
  const int stop = __syncthreads_or(stopped);
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (stop != 0) {
    if (warp == kMmaWarp) tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
    return;
  }
  const uint32_t stage0 = smem_u32(smem);
  // tiles are taken from the END of the mask-sorted order first: those rows have the most kernel offsets, and starting
  // the long tiles first leaves the short ones to fill the tail
  const int first = p.tiles - 1 - static_cast<int>(blockIdx.x);
  const int step = static_cast<int>(gridDim.x);
  const int my_tiles = first / step + 1;
  bool ok = true;
  // the output row at place i of this CTA's tile u, -1 beyond the last
  const auto row_at = [&](int u, int i) {
    const long long place = static_cast<long long>(first - u * step) * kTileM + i;
    if (u >= my_tiles || place >= p.m_rows) return -1;
    return p.order ? __ldg(&p.order[place]) : static_cast<int>(place);
  };

  if (warp < kEpiWarps) {
    // ---------------- epilogue: a thread per row of a tile ----------------
    // A thread reads one row out of tensor memory; stored from there, a warp's 16 bytes a lane would touch 32
    // cache lines an instruction.  The rows of a warp pass through its slab, up to 128 bytes of each at a time,
    // and leave with neighbouring lanes on neighbouring pieces of a row.
    const int pieces = p.epi_bytes / 16, lg = 31 - __clz(pieces);  // 2, 4 or 8 a row
    const int spread = lane >> (3 - lg) & (pieces - 1);            // rows of one 128-byte line go to different banks
    uint8_t* const slab = slabs + warp * 32 * p.epi_bytes;
    uint8_t* const slab_row = slab + lane * p.epi_bytes;
    const int out_bytes = p.n_dim * static_cast<int>(sizeof(TO));
    const int piece = lane & (pieces - 1);
    const uint32_t scale_at = smem_u32(epi_scale);
    int row32 = row_at(0, tid);
    Ring acc;
    for (int u = 0; u < my_tiles; ++u) {
      const int row_next = row_at(u + 1, tid);
      ok = __all_sync(0xffffffffu, mbar_wait_timed(bar(kBarAccFull + acc.at), acc.parity));
      if (!ok) break;
      tc_fence_after();
      const bool any = acc_any[acc.at] != 0;
      const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + acc.at * p.acc_cols;
      for (int b0 = 0; b0 < out_bytes; b0 += p.epi_bytes) {
        const int width = min(p.epi_bytes, out_bytes - b0);
        for (int at = 0; at < width; at += 16 * static_cast<int>(sizeof(TO))) {
          const int c0 = (b0 + at) / static_cast<int>(sizeof(TO));
          uint32_t raw[16];
          tmem_ld16(lane_addr + c0, raw);
          tmem_ld_wait();
          float v[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = any ? __uint_as_float(raw[q]) : 0.f;
          if (row32 >= 0) {
            if (has_epilogue) {
#pragma unroll
              for (int q = 0; q < 16; q += 4) {
                const float4 sc = lds4(scale_at + 4 * (c0 + q)), sh = lds4(scale_at + 4 * (p.epi_pad + c0 + q));
                v[q] = fmaf(v[q], sc.x, sh.x);
                v[q + 1] = fmaf(v[q + 1], sc.y, sh.y);
                v[q + 2] = fmaf(v[q + 2], sc.z, sh.z);
                v[q + 3] = fmaf(v[q + 3], sc.w, sh.w);
              }
              if (p.epi.act == SPC_ACT_RELU) {
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = fmaxf(v[q], 0.f);
              } else if (p.epi.act != SPC_ACT_NONE) {
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = finish_epilogue(v[q], 1.f, 0.f, p.epi.act, p.epi.alpha);
              }
            }
            if (p.epi.residual != nullptr)
              add_residual16<TO>(v, static_cast<const TO*>(p.epi.residual) + static_cast<long long>(row32) * p.n_dim + c0);
          }
          alignas(16) TO line[16];
          store_row16<TO>(line, v);
#pragma unroll
          for (int q = 0; q < static_cast<int>(sizeof(TO)); ++q)
            *reinterpret_cast<uint4*>(slab_row + (((at / 16 + q) ^ spread) * 16)) = reinterpret_cast<const uint4*>(line)[q];
        }
        __syncwarp();
#pragma unroll 2
        for (int i = 0; i < pieces; ++i) {
          const int r = (i << (5 - lg)) + (lane >> lg);
          const int row = __shfl_sync(0xffffffffu, row32, r);
          const int from = (piece ^ (r >> (3 - lg) & (pieces - 1))) * 16;
          if (row >= 0 && piece * 16 < width)
            *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.out) + static_cast<long long>(row) * out_bytes + b0 + piece * 16) =
                *reinterpret_cast<const uint4*>(slab + r * p.epi_bytes + from);
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kBarAccEmpty + acc.at));
      acc.next(kAccs);
      row32 = row_next;
    }
  } else if (warp < kFirstCopy) {
    // ---------------- tables ----------------
    // A warp takes 32 rows of each tile.  PPR neighbouring lanes read a row's entries of a group of offsets, 16 bytes
    // each, one tile (or group) ahead of the copy warps.
    constexpr int PPR = GROUP / 4;  // lanes per row
    constexpr int RPL = 32 / PPR;   // rows per load
    constexpr int LOADS = 32 / RPL;
    const int tw = warp - kFirstTable;
    const int lr = lane / PPR, piece = lane % PPR;
    int4 held[LOADS];
    const auto load = [&](int own_row, int k0) {
      const int k = k0 + 4 * piece;
#pragma unroll
      for (int i = 0; i < LOADS; ++i) {
        const int row = __shfl_sync(0xffffffffu, own_row, i * RPL + lr);
        held[i] = make_int4(-1, -1, -1, -1);
        if (k < p.kv && row >= 0) {
          if (p.pairs_rm != nullptr) {
            held[i] = __ldg(reinterpret_cast<const int4*>(p.pairs_rm + static_cast<long long>(row) * p.kvp + k));
          } else {
            const int32_t* const col = p.pairs + static_cast<long long>(k) * p.m_rows + row;
            held[i].x = __ldg(col);
            if (k + 1 < p.kv) held[i].y = __ldg(col + p.m_rows);
            if (k + 2 < p.kv) held[i].z = __ldg(col + 2ll * p.m_rows);
            if (k + 3 < p.kv) held[i].w = __ldg(col + 3ll * p.m_rows);
          }
        }
      }
    };
    int row = row_at(0, tw * 32 + lane), row_next = row_at(1, tw * 32 + lane);
    load(row, 0);
    Ring tab;
    for (int u = 0; ok && u < my_tiles; ++u) {
      for (int k0 = 0; k0 < p.kv; k0 += GROUP) {
        ok = __all_sync(0xffffffffu, mbar_wait_timed(bar(kBarTabEmpty + tab.at), tab.parity ^ 1));
        if (!ok) break;
        // where the copy threads expect the entry of a tile row: their CP rows lie together, in quads that are
        // permuted so that the threads of a warp meet different banks
        int* const table = tables + (tab.at * group_rows + 4 * piece) * kTileM;
        uint32_t mine = 0;
        const int left = group_rows - 4 * piece;  // rows of the buffer from this lane's first on
#pragma unroll
        for (int i = 0; i < LOADS; ++i) {
          const int r = tw * 32 + i * RPL + lr;
          const int lo = r % kRowsPass, nth = r / kRowsPass;
          const int at = lo * CP + (((nth >> 2) ^ ((lo / (32 / CP)) & (CP / 4 - 1))) << 2) + (nth & 3);
          if (left > 0) table[at] = held[i].x;
          if (left > 1) table[at + kTileM] = held[i].y;
          if (left > 2) table[at + 2 * kTileM] = held[i].z;
          if (left > 3) table[at + 3 * kTileM] = held[i].w;
          mine |= (held[i].x >= 0 ? 1u : 0u) | (held[i].y >= 0 ? 2u : 0u) | (held[i].z >= 0 ? 4u : 0u) | (held[i].w >= 0 ? 8u : 0u);
        }
        mine = __reduce_or_sync(0xffffffffu, mine << (4 * piece));
        if (lane == 0) votes[tab.at * 4 + tw] = mine;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kBarTabFull + tab.at));
        tab.next(kTables);
        if (k0 + GROUP < p.kv) {
          load(row, k0 + GROUP);
        } else {
          row = row_next;
          row_next = row_at(u + 2, tw * 32 + lane);
          load(row, 0);
        }
      }
    }
  } else if (warp < kMmaWarp) {
    // ---------------- row copies and weight slabs ----------------
    const int me = warp - kFirstCopy;
    const int b_cols = p.b_row_bytes / ELEM;  // MN-major: output channels per column block
    const int ncb = B_MN ? (p.n_dim + b_cols - 1) / b_cols : 1;
    const uint32_t b_bytes = B_MN ? static_cast<uint32_t>(ncb * EPR * p.b_row_bytes)
                                  : static_cast<uint32_t>(p.n_dim * A_ROW_BYTES);
    const int chunk = lane & (LPR - 1), row_lo = lane / LPR;
    // this lane's piece of its first two rows; the i-th copy goes to the first or second of them plus a multiple of
    // 2 * kPassBytes (the swizzle term, row modulo 8, 4 or 2, repeats at every other copy at the latest)
    uint32_t lin[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      lin[i] = static_cast<uint32_t>((row_lo + i * kRowsPass) * A_ROW_BYTES + chunk * 16);
      lin[i] ^= ((lin[i] >> 7) & static_cast<uint32_t>(LPR - 1)) << 4;
    }
    const uint32_t odd = lin[1] - lin[0];
    const uint8_t* const src_chunk = static_cast<const uint8_t*>(p.src) + chunk * 16;
    const int quad_x = (row_lo / (32 / CP)) & (CP / 4 - 1);

    Ring slot, tab;
    int turn = 0;  // whose stage comes next
    uint32_t issued = 0, issued_parity = 0;  // slots that this warp has filled, and the rounds it filled last
    const int items = me < p.copiers ? my_tiles * ((p.kv + GROUP - 1) / GROUP) : 0;
    int k0 = 0;
    for (int it = 0; it < items; ++it) {
      ok = __all_sync(0xffffffffu, mbar_wait_timed(bar(kBarTabFull + tab.at), tab.parity));
      if (!ok) break;
      const uint4 v4 = *reinterpret_cast<const uint4*>(votes + tab.at * 4);
      const int* const table = tables + tab.at * group_rows * kTileM + row_lo * CP;
      for (uint32_t rest = v4.x | v4.y | v4.z | v4.w; rest != 0; rest &= rest - 1) {
        if (turn == me) {
          ok = __all_sync(0xffffffffu, mbar_wait_timed(bar(kBarEmpty + slot.at), slot.parity ^ 1));
          if (!ok) break;
          const int kk = __ffs(rest) - 1;
          const int k = p.reversed ? p.kv - 1 - (k0 + kk) : k0 + kk;  // of the weight
          const uint32_t full = bar(kBarFull + slot.at);
          const uint32_t stage = stage0 + static_cast<uint32_t>(slot.at * stage_bytes);
          if (lane == 0) {
            mbar_expect_tx(full, b_bytes);
            const uint32_t b_dst = stage + p.a_stage_bytes;
            if (!B_MN) {
              // weight viewed as [c_out][kv][c_in]: rows n = 0..n_dim-1 of offset k
              tma_load_3d(b_dst, &map_b, 0, k, 0, full);
            } else {
              // weight viewed as [c_out = reduction][kv][c_in]: one load per column block
              for (int cb = 0; cb < ncb; ++cb)
                tma_load_3d(b_dst + cb * EPR * p.b_row_bytes, &map_b, cb * b_cols, k, 0, full);
            }
          }
          const int* const from = table + kk * kTileM;
          const uint32_t dst = stage + lin[0];
#pragma unroll
          for (int q = 0; q < CP / 4; ++q) {
            const int4 v = *reinterpret_cast<const int4*>(from + 4 * (q ^ quad_x));
            const int j[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
              cp_async16_row(dst + (4 * q + (i & 2)) * kPassBytes + ((i & 1) ? odd : 0u),
                             src_chunk + static_cast<unsigned long long>(static_cast<uint32_t>(max(j[i], 0))) * A_ROW_BYTES, j[i]);
          }
          // delivered to the barrier by the copy unit once this thread's copies have landed
          cp_async_arrive_noinc(full);
          issued |= 1u << slot.at;
          issued_parity = (issued_parity & ~(1u << slot.at)) | slot.parity << slot.at;
        }
        if (++turn == p.copiers) turn = 0;
        slot.next(p.stages);
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kBarTabEmpty + tab.at));
      tab.next(kTables);
      k0 += GROUP;
      if (k0 >= p.kv) k0 = 0;
    }
    cp_async_wait_all();
    // after a failure: a weight slab still in flight must not land in the next CTA's memory
    if (!ok)
      for (int s = 0; s < p.stages; ++s)
        if (issued >> s & 1u) mbar_wait_timed(bar(kBarFull + s), issued_parity >> s & 1u);
  } else {
    // ---------------- MMA issuer ----------------
    // One thread paces the whole CTA: every instruction between "stage full" and the commit is
    // on the critical path, so the loop carries running descriptor words (a stage advance is one
    // add to the address field) and the reduction steps are unrolled.
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (TcType<T>::fmt << 7) | (TcType<T>::fmt << 10) |
                             ((B_MN ? 1u : 0u) << 16) | (static_cast<uint32_t>(p.n_dim >> 3) << 17) |
                             (static_cast<uint32_t>(kTileM >> 4) << 24);
      const uint32_t a_type = layout_type_for(A_ROW_BYTES);
      const uint32_t b_type = B_MN ? layout_type_for(p.b_row_bytes) : a_type;
      const uint64_t a_desc0 = make_desc(stage0, 16, 8 * A_ROW_BYTES, a_type);
      const uint64_t b_desc0 = B_MN ? make_desc(stage0 + p.a_stage_bytes, EPR * p.b_row_bytes, 8 * p.b_row_bytes, b_type)
                                    : make_desc(stage0 + p.a_stage_bytes, 16, 8 * A_ROW_BYTES, a_type);
      const uint32_t a_hi = static_cast<uint32_t>(a_desc0 >> 32), b_hi = static_cast<uint32_t>(b_desc0 >> 32);
      const uint32_t a_lo0 = static_cast<uint32_t>(a_desc0), b_lo0 = static_cast<uint32_t>(b_desc0);
      const uint32_t stage_step = static_cast<uint32_t>(stage_bytes >> 4);  // address field counts 16-byte units
      const uint32_t b_step = static_cast<uint32_t>(B_MN ? UMMA_K * p.b_row_bytes / 16 : 2);
      uint32_t a_lo = a_lo0, b_lo = b_lo0, full = bar(kBarFull), empty = bar(kBarEmpty);
      uint32_t full_parity = 0;
      int stage = 0;
      Ring acc, tab;
      for (int u = 0; ok && u < my_tiles; ++u) {
        const uint32_t tmem_d = tmem_base + acc.at * p.acc_cols;
        uint32_t accumulate = 0;
        ok = mbar_wait_timed(bar(kBarAccEmpty + acc.at), acc.parity ^ 1);
        tc_fence_after();
        for (int k0 = 0; ok && k0 < p.kv; k0 += GROUP) {
          ok = mbar_wait_timed(bar(kBarTabFull + tab.at), tab.parity);
          if (!ok) break;
          const uint4 v4 = *reinterpret_cast<const uint4*>(votes + tab.at * 4);
          const int n_stages = __popc(v4.x | v4.y | v4.z | v4.w);
          mbar_arrive(bar(kBarTabEmpty + tab.at));
          tab.next(kTables);
          for (int s = 0; s < n_stages; ++s) {
            // a wait that expires here is either a real failure or the copy warps having aborted
            ok = mbar_wait_timed(full, full_parity);
            if (!ok) break;
            // the feature rows were written through the generic proxy (cp.async): order
            // those writes before the tensor core's async-proxy reads
            fence_proxy_async();
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks) {
              const uint64_t a_desc = (static_cast<uint64_t>(a_hi) << 32) | (a_lo + 2u * ks);
              const uint64_t b_desc = (static_cast<uint64_t>(b_hi) << 32) | (b_lo + b_step * ks);
              tc_mma</*TF32=*/false>(tmem_d, a_desc, b_desc, idesc, accumulate);
              accumulate = 1;
            }
            tc_commit(empty);
            a_lo += stage_step;
            b_lo += stage_step;
            full += 8;
            empty += 8;
            if (++stage == p.stages) {
              stage = 0;
              full_parity ^= 1;
              a_lo = a_lo0;
              b_lo = b_lo0;
              full = bar(kBarFull);
              empty = bar(kBarEmpty);
            }
          }
        }
        if (ok) {
          acc_any[acc.at] = static_cast<int>(accumulate);
          mbar_arrive(bar(kBarAccFull + acc.at));
          tc_commit(bar(kBarAccFull + acc.at));  // arrives once every multiplication above has completed
          acc.next(kAccs);
        }
      }
      if (!ok) {
        // nothing may still be multiplying into tensor memory that is given back below
        tc_commit(bar(kBarDrain));
        mbar_wait_timed(bar(kBarDrain), 0);
      }
    }
    __syncwarp();
  }

  if (!ok) atomicExch(p.status, SPC_ERR_DEVICE_WAIT_EXPIRED);
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
}

template <typename T, typename TO, bool B_MN, int LPR>
int launch_rows(const StreamParams& p, const CUtensorMap& map_b, int grid, size_t smem_bytes, cudaStream_t st) {
  static bool configured[kMaxDevices] = {false};  // per instantiation and device
  SPC_CUDA_OK(ensure_dynamic_smem(gather_gemm_stream_kernel<T, TO, B_MN, LPR>, kMostSmem, configured));
  gather_gemm_stream_kernel<T, TO, B_MN, LPR><<<grid, kThreads, smem_bytes, st>>>(p, map_b);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

template <typename T, typename TO, bool B_MN>
int launch(const StreamParams& p, int a_row_bytes, const CUtensorMap& map_b, int grid, size_t smem_bytes, cudaStream_t st) {
  if (a_row_bytes == 128) return launch_rows<T, TO, B_MN, 8>(p, map_b, grid, smem_bytes, st);
  if (a_row_bytes == 64) return launch_rows<T, TO, B_MN, 4>(p, map_b, grid, smem_bytes, st);
  return launch_rows<T, TO, B_MN, 2>(p, map_b, grid, smem_bytes, st);
}

}  // namespace

// Rows of one stage, 16-bit, both accumulators of two CTAs in tensor memory, and tiles enough that a CTA takes several:
// with few, four small CTAs of gemm_tma.cu a multiprocessor are done before the second tile of a long one, the later the less a
// row is (its channels in and out).  Measured (us, that kernel / this one; neighbours a row of a submanifold layer, strided
// layers by their stages a tile):
//   64 -> 128   180 k rows, 1.8 neighbours  46 / 46    7.5   85 /  81    27  106 / 103     strided, 1.4:  197 k  43 / 34
//               205 k                       53 / 53          97 /  94        122 / 116              2:  186 k  50 / 56
//               260 k                       66 / 57         122 / 119        148 / 143                  243 k  66 / 64
//   64 ->  96   180 k                       34 / 37          69 /  62         85 /  79                  186 k  38 / 43
//               205 k                       41 / 41          79 /  71         92 /  87                  243 k  52 / 50
//   32 -> 128   230 k                       38 / 39          62 /  57         83 /  76                  236 k  36 / 38
//               400 k                       61 / 62         106 /  91        138 / 123                  385 k  56 / 57
//   64 ->  64   390 k                       59 / 54         120 / 117        149 / 151
//               700 k                      101 / 96         211 / 205        256 / 252
//   32 ->  64   390 k                       48 / 43          84 /  72        109 /  94
//   32 ->  32   390 k                       42 / 39          71 /  68         87 /  87
//               700 k                       72 / 67         123 / 113        149 / 154
//   16 ->  16   390 k                       36 / 32          55 /  52         73 /  69
// Input gradients (the weight read transposed), outputs and reduction as above: 64 -> 128 at 205 k rows 54 / 55, 103 / 101,
// 129 / 125; 64 -> 64 at 390 k 59 / 54, 123 / 122, 153 / 155; 32 -> 32 at 390 k 43 / 40, 73 / 72, 92 / 93.
bool gather_gemm_stream_takes(int n_dim, int r_dim, long long m_rows, int dtype) {
  if (dtype != SPC_F16 && dtype != SPC_BF16) return false;
  if (r_dim * 2 != row_span(r_dim, 2) || n_dim > 128 || m_rows >= (1ll << 31) - kTileM) return false;
  return ceil_div(m_rows, kTileM) >= (n_dim > 64 && r_dim == 64 ? 11ll : 20ll) * sm_count();
}

int gather_gemm_stream(const void* src, const void* w, const Epilogue& epi, const int32_t* pairs, const int32_t* pairs_rowmajor,
                       const int32_t* order, void* out, long long m_rows, int n_dim, int r_dim, int kv, bool transposed_weight,
                       bool reversed, int dtype, int out_dtype, cudaStream_t st) {
  StreamParams p{};
  p.src = src; p.epi = epi; p.pairs = pairs; p.pairs_rm = pairs_rowmajor; p.kvp = (kv + 3) & ~3; p.order = order; p.out = out;
  p.m_rows = static_cast<int>(m_rows);
  p.tiles = static_cast<int>(ceil_div(m_rows, kTileM));
  p.n_dim = n_dim; p.kv = kv; p.reversed = reversed;
  const int a_row_bytes = 2 * r_dim;
  p.b_row_bytes = transposed_weight ? row_span(n_dim, 2) : a_row_bytes;
  p.a_stage_bytes = static_cast<int>(align_up(static_cast<size_t>(kTileM) * a_row_bytes, 1024));
  p.b_stage_bytes = static_cast<int>(align_up(static_cast<size_t>(n_dim) * a_row_bytes, 1024));
  const int stage_bytes = p.a_stage_bytes + p.b_stage_bytes;
  p.epi_pad = (n_dim + 15) / 16 * 16;
  p.acc_cols = 32;
  while (p.acc_cols < n_dim) p.acc_cols <<= 1;
  p.tmem_cols = kAccs * p.acc_cols;
  // One wave of two CTAs a multiprocessor, all of them: a CTA that takes a tile less ends with the shortest ones.  (As few CTAs
  // as end with the same number of tiles left a part of the chip with one CTA: 64 -> 96, 190 k rows, 74 us and 91 for 68 and 84.)
  const int ctas = 2;
  const int grid = static_cast<int>(std::min<int64_t>(p.tiles, static_cast<int64_t>(ctas) * sm_count()));
  const int row_bytes = n_dim * (out_dtype == SPC_F32 ? 4 : 2);
  p.epi_bytes = 128;
  while (p.epi_bytes > 32 && p.epi_bytes / 2 >= row_bytes) p.epi_bytes /= 2;
  // Everything besides the stages is sized to the layer.  (228 KB a multiprocessor, 1 KB reserved per CTA.)
  const size_t per_cta = std::min<size_t>(kMostSmem, (228 * 1024 - static_cast<size_t>(ctas) * 1024) / ctas - 256);
  const auto fixed = [&] {
    return 1024 + static_cast<size_t>(kTables) * std::min(kv, table_group(a_row_bytes / 16)) * kTileM * 4 +
           static_cast<size_t>(kTileM) * p.epi_bytes + 2 * p.epi_pad * sizeof(float) + kTables * 16 + kBars * 8 + kAccs * 4 + 8;
  };
  const int widest = p.epi_bytes;
  const auto stages = [&] { return static_cast<int>(std::min<size_t>(kMaxStages, (per_cta - fixed()) / stage_bytes)); };
  // a stage per copy warp, if need be with a narrower epilogue (the 16 channels of a step fit it: 32 bytes of 16-bit results,
  // 64 of fp32 ones); where even that leaves two, a wide one
  const int narrowest = 16 * (out_dtype == SPC_F32 ? 4 : 2);
  while (p.epi_bytes > narrowest && stages() < kCopyWarps) p.epi_bytes /= 2;
  if (stages() < kCopyWarps) p.epi_bytes = widest;
  if (p.epi_bytes < narrowest || row_bytes % narrowest != 0) return fail(SPC_ERR_UNSUPPORTED, "TMA gather-GEMM: store of %d channels", n_dim);
  p.stages = stages();
  p.copiers = std::min(p.stages, kCopyWarps);
  const size_t smem_bytes = fixed() + static_cast<size_t>(p.stages) * stage_bytes;
  p.status = device_status_ptr();
  if (p.status == nullptr) return fail(SPC_ERR_CUDA, "TMA gather-GEMM: no device status word");
  CUtensorMap map_b;
  const int rc = weight_map(&map_b, w, n_dim, r_dim, kv, transposed_weight, p.b_row_bytes, r_dim, dtype);
  if (rc != SPC_OK) return rc;
#define SPC_STREAM(T, TO)                                                                             \
  return transposed_weight ? launch<T, TO, true>(p, a_row_bytes, map_b, grid, smem_bytes, st) \
                           : launch<T, TO, false>(p, a_row_bytes, map_b, grid, smem_bytes, st)
  if (dtype == SPC_F16 && out_dtype == SPC_F16) SPC_STREAM(__half, __half);
  if (dtype == SPC_F16 && out_dtype == SPC_F32) SPC_STREAM(__half, float);
  if (dtype == SPC_BF16 && out_dtype == SPC_BF16) SPC_STREAM(__nv_bfloat16, __nv_bfloat16);
  if (dtype == SPC_BF16 && out_dtype == SPC_F32) SPC_STREAM(__nv_bfloat16, float);
#undef SPC_STREAM
  return fail(SPC_ERR_UNSUPPORTED, "TMA gather-GEMM: dtype combination");
}

}  // namespace spc
