// Weight gradient of the sparse convolution on tcgen05 / TMEM.
//
//   dW[n, k, c] = sum over rows m with pair_fwd[k, m] >= 0 of
//                 grad_out[m, n] * features[pair_fwd[k, m], c]
//
// For one kernel offset k this is a dense contraction D[n, c] = G^T F over the
// list of existing (output row, input row) pairs, with the pairs as the
// reduction dimension.  One CTA owns (offset k, a contiguous range of output
// rows, one or two blocks of <= 128 output channels) and keeps D (128 lanes x
// c_in fp32 columns a block) in tensor memory; with 256 output channels both
// blocks multiply the same feature rows, which two CTAs would gather twice.
// Bound by the gathered rows on narrow layers (64 -> 128, 1.6 M pairs of a 27 x 1.36 M
// table: 188 us, 631 MB read, a quarter of it the table; the tensor pipe at 5 %).  k5
// 256 -> 256, 13.6 M pairs: 5.5 ms with a block a CTA, 2.35 now (760 TFLOP/s, 0.46 of
// the measured peak).
// W (four or eight) copy warps and one that multiplies:
//   warps 0 .. W-1  scan pair_fwd[k, lo:hi] 1024 entries a round, compact the
//              existing pairs into a shared-memory ring with warp ballots (no
//              host-side nonzero(), unlike spconv_triton/pytorch/_impl/gemm.py:663),
//              and for every 64 pairs copy the 64 grad_out rows and the 64
//              feature rows into a swizzled stage with 16-byte cp.async
//              (completion delivered by cp.async.mbarrier.arrive.noinc)
//   warp W     issues tcgen05.mma with BOTH operands MN-major: a stage row is
//              one pair and holds its channels contiguously, which is exactly
//              how gathered rows arrive, so nothing is transposed
//   warps 0-3  finally read TMEM and write the fp32 partial tile
//              partial[split, n, k, c]; the partials of the splits are added
//              in a fixed order by the reduction kernel of gemm_simt.cu.
// Rows of the accumulator beyond c_out are computed from whatever the stage
// buffer holds and are never stored.  Every wait is bounded.
#include <algorithm>

#include "common.cuh"
#include "gemm_internal.cuh"
#include "tc_common.cuh"

namespace spc {
namespace {

using namespace tc;

// The number of copy warps is a template parameter: four (160-thread CTAs, three per SM) where a pair
// is at most 384 bytes of rows, eight (two CTAs per SM) for wider rows, which need the copy throughput.
constexpr int kWgMaxIssueWarps = 8;
constexpr int kPairsPerStage = 64;
constexpr int kRing = 2048;                          // capacity of the pair list (power of two, > 64 + 1024)

struct WgParams {
  const void* feats;
  const void* gout;
  const int32_t* pair_fwd;
  float* partial;
  long long n_out, rows_per_split;
  int c_in, c_out, kv, splits;
  int g_row_bytes, f_row_bytes;  // swizzle span of the grad_out / feature rows (32, 64 or 128)
  int n_blocks;  // blocks of 128 output channels of a CTA
  int g_stage_bytes, f_stage_bytes, stages, tmem_cols, cols;
  int* status;
};

__host__ __device__ inline uint32_t wg_layout_type(int row_bytes) {
  return row_bytes == 128 ? 2u : (row_bytes == 64 ? 4u : 6u);
}

// Copies 16-byte pieces of gathered rows into an MN-major stage region: column block b of row p lands at
// base + b * (kPairsPerStage * row_bytes) + p * row_bytes (+ swizzle); rows n .. n_pad are zero filled.
__device__ __forceinline__ uint32_t piece_place(int p, int piece, int row_bytes) {
  const int per_block = row_bytes / 16;  // 2, 4 or 8
  const int lg = per_block == 8 ? 3 : (per_block == 4 ? 2 : 1);
  const uint32_t lin = static_cast<uint32_t>(p * row_bytes + (piece & (per_block - 1)) * 16);
  const uint32_t mask = static_cast<uint32_t>(per_block - 1);
  return static_cast<uint32_t>((piece >> lg) * kPairsPerStage * row_bytes) + (lin ^ (((lin >> 7) & mask) << 4));
}

// A power of two of pieces: a thread keeps its piece and steps over the rows by a multiple of eight, the
// period of the swizzle, so that where it starts is settled once per CTA and a copy costs one list read and
// two additions; four copies at a time, their list entries first, since with one warp on a scheduler every
// dependent instruction is waited for (27 offsets of 45 k rows, 64 -> 64: 109 -> 64 us together with the
// order of the offsets below and twice the splits; 128 -> 128: 169 -> 151 us).
__device__ __forceinline__ void copy_rows(uint32_t to, const uint8_t* at, uint32_t pitch, const int* rows, int n, int n_pad, int first,
                                          int step, uint32_t dst_step) {
  for (int p = first; p < n_pad; p += 4 * step, to += 4 * dst_step) {
    uint32_t row[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) row[u] = p + u * step < n ? static_cast<uint32_t>(rows[p + u * step]) : 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (p + u * step < n_pad)
        cp_async16(to + u * dst_step, at + static_cast<unsigned long long>(row[u]) * pitch, p + u * step < n ? 16u : 0u);
  }
}

// Any number of pieces (48 or 96 channels).
template <int THREADS>
__device__ __forceinline__ void copy_rows_any(uint32_t base, const uint8_t* src, uint32_t pitch, const int* rows, int n, int n_pad,
                                              int pieces, int row_bytes, int tid) {
  for (int q = tid; q < n_pad * pieces; q += THREADS) {
    const int p = q / pieces, piece = q - p * pieces;
    const uint32_t row = p < n ? static_cast<uint32_t>(rows[p]) : 0u;
    cp_async16(base + piece_place(p, piece, row_bytes), src + static_cast<unsigned long long>(row) * pitch + piece * 16, p < n ? 16u : 0u);
  }
}

// SCAN: table entries a thread looks at per scan round.
// The registers of three or two CTAs a multiprocessor: left to the compiler, eight copy warps took 115 a thread, which
// is one CTA (128 -> 128, 383 k rows, 3.8 M pairs: 526 us; two, with 94: 350).
template <typename T, int W, int SCAN>
__global__ void __launch_bounds__(W * 32 + 32, W == 4 ? 3 : 2)
wgrad_tc_kernel(const __grid_constant__ WgParams p) {
  constexpr int kWgIssueWarps = W;
  constexpr int kWgIssueThreads = W * 32;
  constexpr int kWgMmaWarp = W;
  constexpr int kScanEntries = SCAN * kWgIssueThreads;
  constexpr int ELEM = sizeof(T);
  constexpr int UMMA_K = 32 / ELEM;  // 16 pairs per MMA

  extern __shared__ uint8_t smem_raw[];
  // (an offset, not a rounded pointer: the compiler keeps knowing that these are shared-memory addresses)
  uint8_t* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int stage_bytes = p.g_stage_bytes + p.f_stage_bytes;
  uint8_t* stage_base = smem;
  int* ring_m = reinterpret_cast<int*>(smem + static_cast<size_t>(p.stages) * stage_bytes);  // output rows
  int* ring_i = ring_m + kRing;                                                                // input rows
  int* rows_m = ring_i + kRing;            // [stages][64] row lists of the stages in flight
  int* rows_i = rows_m + kMaxStages * kPairsPerStage;
  uint64_t* bars = reinterpret_cast<uint64_t*>(rows_i + kMaxStages * kPairsPerStage);
  StageInfo* info = reinterpret_cast<StageInfo*>(bars + 2 * kMaxStages + 1);
  int* warp_cnt = reinterpret_cast<int*>(info + kMaxStages);  // [SCAN][8]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(warp_cnt + SCAN * kWgIssueWarps);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  // (one thread's reading, acted on by the whole CTA below: threads that saw different values must not part)
  const int stopped = tid == 32 ? *reinterpret_cast<volatile int*>(p.status) : 0;
  // The middle offsets first: the centre of a submanifold kernel has every row, its neighbours most of them,
  // and a CTA of theirs started last would run on alone.
  const int turn = blockIdx.x / p.splits, split = blockIdx.x % p.splits;
  const int k = (turn & 1) ? (p.kv - 1) / 2 + (turn + 1) / 2 : (p.kv - 1) / 2 - turn / 2;
  const int n0 = blockIdx.y * p.n_blocks * kTileM;  // first output channel of this CTA
  const long long lo = split * p.rows_per_split;
  const long long hi = min(p.n_out, lo + p.rows_per_split);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = smem_u32(bars + kMaxStages);
  const uint32_t bar_accum = smem_u32(bars + 2 * kMaxStages);

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(bar_full + 8 * s, kWgIssueThreads + 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_accum, 1);
    fence_mbar_init();
  }
  if (warp == kWgMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish();
  }
  tc_fence_before();
  const int stop = __syncthreads_or(stopped);
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (stop != 0) {
    if (warp == kWgMmaWarp) tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
    return;
  }

  int real_stages = 0;
  if (warp < kWgIssueWarps) {
    int stage = 0;
    uint32_t empty_parity = 1;
    bool ok = true;
    int head = 0, tail = 0;  // ring positions (uniform over the copy threads)
    long long pos = lo;
    const int g_cols = min(p.n_blocks * kTileM, p.c_out - n0);  // output channels this CTA owns
    const int g_pieces = g_cols * ELEM / 16;
    const int f_pieces = p.c_in * ELEM / 16;
    const uint8_t* g_src = static_cast<const uint8_t*>(p.gout) + static_cast<size_t>(n0) * ELEM;
    const uint8_t* f_src = static_cast<const uint8_t*>(p.feats);
    const uint32_t g_pitch = static_cast<uint32_t>(p.c_out) * ELEM, f_pitch = static_cast<uint32_t>(p.c_in) * ELEM;
    const int g_lg = 31 - __clz(g_pieces), g_step = kWgIssueThreads >> g_lg, g_first = tid >> g_lg, g_piece = tid & (g_pieces - 1);
    const bool g_even = (g_pieces & (g_pieces - 1)) == 0 && g_step >= 8;
    const uint32_t g_place = piece_place(g_first, g_piece, p.g_row_bytes);
    const int f_lg = 31 - __clz(f_pieces), f_step = kWgIssueThreads >> f_lg, f_first = tid >> f_lg, f_piece = tid & (f_pieces - 1);
    const bool f_even = (f_pieces & (f_pieces - 1)) == 0 && f_step >= 8;
    const uint32_t f_place = piece_place(f_first, f_piece, p.f_row_bytes);

    // Table entries are fetched one scan round (1024 entries, SCAN per thread) ahead:
    // the loads of the next round are in flight while the stages of this one are built,
    // so the walk over a sparse table does not pay a memory latency per round.
    const int32_t* table = p.pair_fwd + static_cast<long long>(k) * p.n_out;
    int ahead[SCAN];
    auto fetch = [&](long long at) {
#pragma unroll
      for (int j = 0; j < SCAN; ++j) {
        const long long m = at + j * kWgIssueThreads + tid;
        ahead[j] = m < hi ? __ldg(&table[m]) : -1;
      }
    };
    fetch(pos);
    while (pos < hi || tail > head) {
      if (tail - head < kPairsPerStage && pos < hi) {
        // ---- append the existing pairs of one scan round to the ring, in table order ----
        int cur[SCAN];
        unsigned ballot[SCAN];
#pragma unroll
        for (int j = 0; j < SCAN; ++j) {
          cur[j] = ahead[j];
          ballot[j] = __ballot_sync(0xffffffffu, cur[j] >= 0);
          if (lane == 0) warp_cnt[j * kWgIssueWarps + warp] = __popc(ballot[j]);
        }
        const long long at = pos;
        pos += kScanEntries;
        if (pos < hi) fetch(pos);
        named_bar_sync(1, kWgIssueThreads);
        int before[SCAN];
        int run = 0;
#pragma unroll
        for (int j = 0; j < SCAN; ++j) {
#pragma unroll
          for (int w = 0; w < kWgIssueWarps; ++w) {
            if (w == warp) before[j] = run;
            run += warp_cnt[j * kWgIssueWarps + w];
          }
        }
#pragma unroll
        for (int j = 0; j < SCAN; ++j) {
          if (cur[j] >= 0) {
            const int slot = (tail + before[j] + __popc(ballot[j] & ((1u << lane) - 1u))) & (kRing - 1);
            ring_m[slot] = static_cast<int>(at + j * kWgIssueThreads + tid);
            ring_i[slot] = cur[j];
          }
        }
        named_bar_sync(1, kWgIssueThreads);
        tail += run;
        continue;
      }
      // ---- one stage: up to 64 pairs from the head of the ring ----
      const int n = min(kPairsPerStage, tail - head);
      const int n_pad = (n + UMMA_K - 1) / UMMA_K * UMMA_K;  // rows the MMAs will read; the tail is zero filled
      ++real_stages;
      if (ok && !mbar_wait(bar_empty + 8 * stage, empty_parity)) ok = false;
      if (ok) {
        // private copy of the stage's row lists (the ring may be overwritten by the next scan)
        int* sm = rows_m + stage * kPairsPerStage;
        int* si = rows_i + stage * kPairsPerStage;
        if (tid < n) {
          sm[tid] = ring_m[(head + tid) & (kRing - 1)];
          si[tid] = ring_i[(head + tid) & (kRing - 1)];
        }
        named_bar_sync(2, kWgIssueThreads);
        const uint32_t g_dst = smem_u32(stage_base + static_cast<size_t>(stage) * stage_bytes);
        const uint32_t f_dst = g_dst + p.g_stage_bytes;
        const uint32_t full = bar_full + 8 * stage;
        if (g_even)
          copy_rows(g_dst + g_place, g_src + g_piece * 16, g_pitch, sm, n, n_pad, g_first, g_step, g_step * p.g_row_bytes);
        else
          copy_rows_any<kWgIssueThreads>(g_dst, g_src, g_pitch, sm, n, n_pad, g_pieces, p.g_row_bytes, tid);
        if (f_even)
          copy_rows(f_dst + f_place, f_src + f_piece * 16, f_pitch, si, n, n_pad, f_first, f_step, f_step * p.f_row_bytes);
        else
          copy_rows_any<kWgIssueThreads>(f_dst, f_src, f_pitch, si, n, n_pad, f_pieces, p.f_row_bytes, tid);
        cp_async_arrive_noinc(full);
        if (tid == 0) {
          info[stage].ksteps = n_pad / UMMA_K;
          info[stage].last = 0;
          mbar_arrive(full);
        }
        if (++stage == p.stages) {
          stage = 0;
          empty_parity ^= 1;
        }
      } else {
        named_bar_sync(2, kWgIssueThreads);
      }
      head += n;
    }
    // terminator
    if (ok && !mbar_wait(bar_empty + 8 * stage, empty_parity)) ok = false;
    if (ok) {
      mbar_arrive(bar_full + 8 * stage);
      if (tid == 0) {
        info[stage].ksteps = 0;
        info[stage].last = 1;
        mbar_arrive(bar_full + 8 * stage);
      }
    } else {
      atomicExch(p.status, SPC_ERR_DEVICE_WAIT_EXPIRED);
    }
    cp_async_wait_all();

    // ---------------- epilogue (warps 0-3): fp32 partial tile ----------------
    if (warp < 4) {
      bool have_acc = mbar_wait(bar_accum, 0);
      if (!have_acc) atomicExch(p.status, SPC_ERR_DEVICE_WAIT_EXPIRED);
      have_acc = __all_sync(0xffffffffu, have_acc);
      tc_fence_after();
      if (have_acc) {
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
        for (int b = 0; b < p.n_blocks; ++b) {
          const int n = n0 + b * kTileM + tid;  // output channel held by this TMEM lane
          float* dst = p.partial + ((static_cast<long long>(split) * p.c_out + (n < p.c_out ? n : 0)) * p.kv + k) * p.c_in;
          for (int c0 = 0; c0 < p.c_in; c0 += 16) {
            float v[16];
            if (real_stages > 0) {
              uint32_t raw[16];
              tmem_ld16(lane_addr + b * p.cols + c0, raw);
              tmem_ld_wait();
#pragma unroll
              for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(raw[q]);
            } else {
#pragma unroll
              for (int q = 0; q < 16; ++q) v[q] = 0.f;
            }
            if (n < p.c_out) store_row16<float>(dst + c0, v);
          }
        }
      }
      tc_fence_before();
    }
  } else {
    // ---------------- MMA issuer ----------------
    // This one thread paces the CTA: the loop keeps running descriptor words (a stage advance
    // is one add to the address field) and unrolls the four 16-pair steps of a stage.
    if (lane == 0) {
      // fp32 accumulate, both operands MN-major, M = 128, N = c_in
      const uint32_t idesc = (1u << 4) | (TcType<T>::fmt << 7) | (TcType<T>::fmt << 10) | (1u << 15) | (1u << 16) |
                             (static_cast<uint32_t>(p.c_in >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
      const uint32_t g_type = wg_layout_type(p.g_row_bytes), f_type = wg_layout_type(p.f_row_bytes);
      const uint32_t g_addr0 = smem_u32(stage_base);
      const uint64_t a_desc0 = make_desc(g_addr0, kPairsPerStage * p.g_row_bytes, 8 * p.g_row_bytes, g_type);
      const uint64_t b_desc0 = make_desc(g_addr0 + p.g_stage_bytes, kPairsPerStage * p.f_row_bytes, 8 * p.f_row_bytes, f_type);
      const uint32_t a_hi = static_cast<uint32_t>(a_desc0 >> 32), b_hi = static_cast<uint32_t>(b_desc0 >> 32);
      const uint32_t a_lo0 = static_cast<uint32_t>(a_desc0), b_lo0 = static_cast<uint32_t>(b_desc0);
      const uint32_t stage_step = static_cast<uint32_t>(stage_bytes >> 4);
      const uint32_t a_step = static_cast<uint32_t>(UMMA_K * p.g_row_bytes / 16);
      const uint32_t b_step = static_cast<uint32_t>(UMMA_K * p.f_row_bytes / 16);
      const uint32_t a_block = static_cast<uint32_t>(kTileM * ELEM * kPairsPerStage / 16);  // 128 channels of a stage's rows
      const uint32_t info0 = smem_u32(info);
      uint32_t a_lo = a_lo0, b_lo = b_lo0, full = bar_full, empty = bar_empty, inf = info0;
      int stage = 0;
      uint32_t full_parity = 0, accumulate = 0;
      bool ok = true;
      while (true) {
        if (!mbar_wait(full, full_parity)) {
          ok = false;
          break;
        }
        fence_proxy_async();  // stage was written by cp.async (generic proxy)
        tc_fence_after();
        uint32_t ksteps;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(ksteps) : "r"(inf) : "memory");
        if (ksteps == 0) {  // terminator
          tc_commit(bar_accum);
          break;
        }
        for (int b = 0; b < p.n_blocks; ++b) {
          const uint32_t d = tmem_base + static_cast<uint32_t>(b * p.cols), a_at = a_lo + b * a_block;
#pragma unroll
          for (int ks = 0; ks < kPairsPerStage / UMMA_K; ++ks) {
            if (static_cast<uint32_t>(ks) < ksteps) {
              const uint64_t a_desc = (static_cast<uint64_t>(a_hi) << 32) | (a_at + a_step * ks);
              const uint64_t b_desc = (static_cast<uint64_t>(b_hi) << 32) | (b_lo + b_step * ks);
              tc_mma<false>(d, a_desc, b_desc, idesc, ks == 0 ? accumulate : 1u);
            }
          }
        }
        accumulate = 1;
        tc_commit(empty);
        a_lo += stage_step;
        b_lo += stage_step;
        full += 8;
        empty += 8;
        inf += static_cast<uint32_t>(sizeof(StageInfo));
        if (++stage == p.stages) {
          stage = 0;
          full_parity ^= 1;
          a_lo = a_lo0;
          b_lo = b_lo0;
          full = bar_full;
          empty = bar_empty;
          inf = info0;
        }
      }
      if (!ok) {
        atomicExch(p.status, SPC_ERR_DEVICE_WAIT_EXPIRED);
        mbar_arrive(bar_accum);
      }
    }
    __syncwarp();
  }

  __syncthreads();
  if (warp == kWgMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
}

// Swizzle span of rows of `elems` channels: the widest of 128, 64 and 32 bytes that divides them.
int span_of(int elems, int elem_size) {
  const int bytes = elems * elem_size;
  return bytes % 128 == 0 ? 128 : bytes % 64 == 0 ? 64 : bytes % 32 == 0 ? 32 : 0;
}

// Blocks of 128 output channels a CTA takes (two fill tensor memory at 256 input channels: one CTA per SM).
int wg_blocks(int c_out) { return c_out % (2 * tc::kTileM) == 0 ? 2 : 1; }

template <typename T, int W, int SCAN>
int launch_wgrad_tc(const WgParams& p, size_t smem_bytes, cudaStream_t st) {
  static bool configured[kMaxDevices] = {false};  // per instantiation and device
  SPC_CUDA_OK(ensure_dynamic_smem(wgrad_tc_kernel<T, W, SCAN>, 226 * 1024, configured));
  dim3 grid(static_cast<unsigned>(p.kv * p.splits), static_cast<unsigned>(ceil_div(p.c_out, p.n_blocks * kTileM)));
  wgrad_tc_kernel<T, W, SCAN><<<grid, W * 32 + 32, smem_bytes, st>>>(p);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace

bool wgrad_tc_supported(int c_in, int c_out, int kv, int dtype) {
  (void)kv;
  if (dtype != SPC_F16 && dtype != SPC_BF16) return false;
  if (c_in < 16 || c_in > 256 || c_in % 16 != 0 || c_out < 16 || c_out % 16 != 0) return false;
  // a CTA's slice of grad_out columns must also fit a swizzle span
  const int g_cols = std::min(c_out, tc::kTileM);
  if (c_out > tc::kTileM && c_out % tc::kTileM != 0) return false;
  return span_of(c_in, 2) != 0 && span_of(g_cols, 2) != 0;
}

// Split of the row range; same formula family as the CUDA-core kernel, with the
// tensor-core tile (128 output channels x all input channels per CTA).
WgradSplit wgrad_tc_split(int64_t n_out, int c_in, int c_out, int kv) {
  WgradSplit s;
  const int64_t tiles = static_cast<int64_t>(kv) * ceil_div(c_out, wg_blocks(c_out) * tc::kTileM);
  // several CTAs per resident slot: offsets differ a lot in how many pairs they have (the centre
  // offset of a submanifold layer has all of them), and surplus CTAs even that out
  int64_t want = ceil_div(16 * static_cast<int64_t>(sm_count()), std::max<int64_t>(tiles, 1));
  // Two costs: the centre offset's CTAs are the longest chain (as long as a split has rows), and every split writes
  // c_out * kv * c_in partial sums that the reduction reads.  Few table entries (rows times offsets) leave the chip idle
  // with long splits, many pay for short ones; wide layers have the larger sums.  Rows a split 1024 / 2048 / 4096,
  // fp16, submanifold scenes a quarter full, microseconds:
  //                         32->32            64->64          64->128          128->128          256->256
  //   27 offsets, 10 k   27 /  42 /  70   30 /  44 /  74   34 /  50 /  85   38 /  50 /  81   67 /  81 / 130
  //   125, 10 k          36 /  44 /  71   44 /  48 /  77   56 /  58 /  91   83 /  65 /  93  261 / 167 / 153
  //   27, 45 k           40 /  40 /  67   46 /  48 /  71   58 /  56 /  83   93 /  61 /  85  276 / 163 / 130
  //   27, 150 k          81 /  81 /  77   95 /  95 /  87  119 / 119 / 106  177 / 177 / 142  489 / 486 / 359
  //   125, 40 k          89 /  89 /  79  105 / 104 /  89  138 / 138 / 108  212 / 212 / 148  622 / 622 / 400
  // Entries: 0.27, 1.25, 1.2, 4.1 and 5 million; the lines lie between the rows where the better side changes.  Where few of the
  // entries are pairs, the centre's chain is all there is to narrow layers: 100 k rows with 1.5 neighbours, 2048 / 4096, 16 -> 16
  // 30 / 49, 64 -> 64 39 / 56, 64 -> 128 55 / 73 (128 -> 128, with 4096, 86); so these stay at 2048, a tenth behind in full scenes.
  const int64_t entries = n_out * kv, sums = static_cast<int64_t>(c_in) * c_out;
  const bool narrow = sums <= 64 * 128;
  const int64_t few = narrow ? 1250000 : 400000, some = sums <= 128 * 128 ? 2400000 : 600000;
  const int64_t by_len = std::max<int64_t>(1, n_out / (entries <= few ? 1024 : narrow || entries <= some ? 2048 : 4096));
  want = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, by_len), 64));
  s.splits = static_cast<int>(want);
  s.rows_per_split = ceil_div(std::max<int64_t>(n_out, 1), s.splits);
  s.bytes = static_cast<size_t>(s.splits) * c_out * kv * c_in * sizeof(float);
  return s;
}

int wgrad_tc(const void* feats, const void* gout, const int32_t* pair_fwd, float* partial, int64_t n_out, int c_in,
             int c_out, int kv, int dtype, const WgradSplit& split, cudaStream_t st) {
  if (!wgrad_tc_supported(c_in, c_out, kv, dtype)) return fail(SPC_ERR_UNSUPPORTED, "tcgen05 wgrad: unsupported shape");
  if ((reinterpret_cast<uintptr_t>(feats) | reinterpret_cast<uintptr_t>(gout) | reinterpret_cast<uintptr_t>(partial)) & 15u)
    return fail(SPC_ERR_UNSUPPORTED, "tcgen05 wgrad: operands must be 16-byte aligned");
  WgParams p{};
  p.feats = feats; p.gout = gout; p.pair_fwd = pair_fwd; p.partial = partial;
  p.n_out = n_out; p.rows_per_split = split.rows_per_split; p.splits = split.splits;
  p.c_in = c_in; p.c_out = c_out; p.kv = kv; p.n_blocks = wg_blocks(c_out);
  const int g_cols = std::min(c_out, tc::kTileM);
  p.g_row_bytes = span_of(g_cols, 2);
  p.f_row_bytes = span_of(c_in, 2);
  // the A region always spans 128 channels (M = 128); columns beyond c_out hold stale data
  p.g_stage_bytes = static_cast<int>(align_up(static_cast<size_t>(p.n_blocks) * tc::kTileM * 2 * kPairsPerStage, 1024));
  p.f_stage_bytes = static_cast<int>(align_up(static_cast<size_t>(c_in) * 2 * kPairsPerStage, 1024));
  const int stage_bytes = p.g_stage_bytes + p.f_stage_bytes;
  const size_t fixed = 1024 + 2 * kRing * 4 + 2 * tc::kMaxStages * kPairsPerStage * 4 + (2 * tc::kMaxStages + 1) * 8 +
                       tc::kMaxStages * sizeof(tc::StageInfo) + 8 * kWgMaxIssueWarps * 4 + 64;
  const bool narrow = (c_in + p.n_blocks * g_cols) * 2 <= 384;  // bytes of rows per pair
  p.cols = 32;
  while (p.cols < c_in) p.cols <<= 1;
  // three, two or (two blocks of 256 columns) one CTA per SM
  const size_t budget = narrow ? 74 * 1024 : p.n_blocks * p.cols > 256 ? 222 * 1024 : 110 * 1024;
  p.stages = std::max(2, std::min<int>(tc::kMaxStages, static_cast<int>((budget - fixed) / stage_bytes)));
  const size_t smem_bytes = fixed + static_cast<size_t>(p.stages) * stage_bytes;
  p.tmem_cols = p.n_blocks * p.cols;
  p.status = device_status_ptr();
  if (p.status == nullptr) return fail(SPC_ERR_CUDA, "tcgen05 wgrad: no device status word");
  if (narrow) {
    if (dtype == SPC_F16) return launch_wgrad_tc<__half, 4, 8>(p, smem_bytes, st);
    return launch_wgrad_tc<__nv_bfloat16, 4, 8>(p, smem_bytes, st);
  }
  if (dtype == SPC_F16) return launch_wgrad_tc<__half, 8, 4>(p, smem_bytes, st);
  return launch_wgrad_tc<__nv_bfloat16, 8, 4>(p, smem_bytes, st);
}

}  // namespace spc
