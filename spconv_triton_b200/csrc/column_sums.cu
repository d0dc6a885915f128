// Column sums of a row-major matrix: the gradient of a layer's bias.  HBM-bound: one read of the matrix.
//
// A thread owns one 16-byte vector of columns and strides over the rows of its CTA's chunk with four loads in
// flight; the row lanes of a CTA add up in shared memory, the chunks' fp32 sums in a second kernel in chunk
// order (no atomics: the same bits every time).  1.36 M x 128 fp16 (348 MB): 296 us in torch's reduction.
#include <algorithm>

#include "common.cuh"

namespace spc {
namespace {

constexpr int kThreads = 256;

template <typename T, int VEC>
__global__ void __launch_bounds__(kThreads)
column_sums_kernel(const T* __restrict__ x, long long rows, int cols, long long rows_per_chunk, float* __restrict__ partial) {
  struct alignas(sizeof(T) * VEC) Pack { T v[VEC]; };
  extern __shared__ float sums[];  // [row lanes][column vectors of this CTA * VEC]
  const int vecs = cols / VEC;
  const int width = min(vecs, kThreads);                       // column vectors a CTA covers; grid.y covers the rest
  const int lanes = kThreads / width;                          // row lanes
  const int cv = threadIdx.x % width, rl = threadIdx.x / width;
  const int col = (blockIdx.y * width + cv) * VEC;
  const long long lo = blockIdx.x * rows_per_chunk, hi = min(rows, lo + rows_per_chunk);
  float acc[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
  if (rl < lanes && col < cols) {
    const T* at = x + lo * cols + col;
    const long long n = hi - lo;
    long long r = rl;
    constexpr int kAhead = 4;
    for (; r + (kAhead - 1) * lanes < n; r += kAhead * lanes) {
      Pack p[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) p[u] = *reinterpret_cast<const Pack*>(at + (r + u * lanes) * cols);
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[v] += to_float(p[u].v[v]);
    }
    for (; r < n; r += lanes) {
      const Pack p = *reinterpret_cast<const Pack*>(at + r * cols);
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] += to_float(p.v[v]);
    }
#pragma unroll
    for (int v = 0; v < VEC; ++v) sums[(rl * width + cv) * VEC + v] = acc[v];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < width * VEC; i += kThreads) {
    if (blockIdx.y * width * VEC + i >= cols) break;
    float s = 0.f;
    for (int l = 0; l < lanes; ++l) s += sums[l * width * VEC + i];
    partial[blockIdx.x * static_cast<long long>(cols) + blockIdx.y * width * VEC + i] = s;
  }
}

// out[c] = sum of partial[chunk, c]; 32 columns a CTA, 32 chunk lanes with eight loads under way each (eight lanes, four
// loads: 14.6 us for 1184 chunks of 128 columns, all of it waiting).
constexpr int kAddLanes = 32;
template <typename TO>
__global__ void __launch_bounds__(32 * kAddLanes)
add_chunks_kernel(const float* __restrict__ partial, int chunks, int cols, TO* __restrict__ out) {
  __shared__ float s[kAddLanes][32];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), lane = threadIdx.x >> 5;
  float sum = 0.f;
  if (c < cols) {
#pragma unroll 8
    for (int i = lane; i < chunks; i += kAddLanes) sum += __ldg(&partial[static_cast<long long>(i) * cols + c]);
  }
  s[lane][threadIdx.x & 31] = sum;
  __syncthreads();
  if (lane == 0 && c < cols) {
    float all = 0.f;
#pragma unroll
    for (int l = 0; l < kAddLanes; ++l) all += s[l][threadIdx.x & 31];
    out[c] = from_float<TO>(all);
  }
}

int chunks_for(int64_t rows) {
  // eight CTAs a multiprocessor; no chunk below 256 rows
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(ceil_div(rows, 256), 8ll * sm_count())));
}

template <typename T>
int column_sums(const void* x, int64_t rows, int cols, void* out, int out_dtype, float* partial, cudaStream_t st) {
  const int chunks = chunks_for(rows);
  const long long per = ceil_div(rows, chunks);
  constexpr int kFull = 16 / sizeof(T);
  const T* src = static_cast<const T*>(x);
  const bool wide = cols % kFull == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int vecs = wide ? cols / kFull : cols, width = std::min(vecs, kThreads);
  const dim3 grid(chunks, static_cast<unsigned>(ceil_div(vecs, width)));
  const size_t smem = static_cast<size_t>(kThreads) * (wide ? kFull : 1) * 4;
  if (wide) column_sums_kernel<T, kFull><<<grid, kThreads, smem, st>>>(src, rows, cols, per, partial);
  else column_sums_kernel<T, 1><<<grid, kThreads, smem, st>>>(src, rows, cols, per, partial);
  SPC_LAUNCH_OK();
  const unsigned blocks = static_cast<unsigned>(ceil_div(cols, 32));
  switch (out_dtype) {
    case SPC_F16: add_chunks_kernel<<<blocks, 32 * kAddLanes, 0, st>>>(partial, chunks, cols, static_cast<__half*>(out)); break;
    case SPC_BF16: add_chunks_kernel<<<blocks, 32 * kAddLanes, 0, st>>>(partial, chunks, cols, static_cast<__nv_bfloat16*>(out)); break;
    case SPC_F32: add_chunks_kernel<<<blocks, 32 * kAddLanes, 0, st>>>(partial, chunks, cols, static_cast<float*>(out)); break;
    default: return fail(SPC_ERR_UNSUPPORTED, "column_sums: dtype %d not supported", out_dtype);
  }
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace
}  // namespace spc

using namespace spc;

extern "C" size_t spc_column_sums_workspace_bytes(int64_t rows, int cols) {
  if (rows < 0 || cols <= 0) return 0;
  return static_cast<size_t>(chunks_for(rows)) * cols * sizeof(float);
}

extern "C" int spc_column_sums(const void* x, int64_t rows, int cols, int dtype, void* out, int out_dtype, void* workspace,
                               size_t workspace_bytes, void* stream) {
  if (!x || !out || !workspace || rows < 0 || cols <= 0) return fail(SPC_ERR_INVALID_ARGUMENT, "column_sums: bad arguments");
  if (workspace_bytes < spc_column_sums_workspace_bytes(rows, cols))
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "column_sums: workspace of %zu bytes", workspace_bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* partial = static_cast<float*>(workspace);
  switch (dtype) {
    case SPC_F16: return column_sums<__half>(x, rows, cols, out, out_dtype, partial, st);
    case SPC_BF16: return column_sums<__nv_bfloat16>(x, rows, cols, out, out_dtype, partial, st);
    case SPC_F32: return column_sums<float>(x, rows, cols, out, out_dtype, partial, st);
    default: return fail(SPC_ERR_UNSUPPORTED, "column_sums: dtype %d not supported", dtype);
  }
}
