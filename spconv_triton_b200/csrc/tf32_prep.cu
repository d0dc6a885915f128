// Operand preparation for the fp32 convolutions on the tensor cores.
//
// tcgen05.mma kind::tf32 reads fp32 operands and uses their upper 19 bits (sign, 8 exponent
// bits, 10 mantissa bits).  Two preparations make that exact arithmetic on chosen operands:
//
//   SPC_TF32_ROUND   x -> rna(x): every value rounded to the nearest TF32 number (ties away from
//                    zero), the same rounding the reference's Triton dot applies to its operands
//                    when SPCONV_ALLOW_TF32 is set (_impl/gemm.py:55-62).  Without it the tensor
//                    core would truncate, which biases every product towards zero.
//   SPC_TF32_SPLIT_* x -> (hi, lo) with hi = rna(x), lo = rna(x - hi): x = hi + lo up to 2^-22 |x|.
//                    A convolution with reduction [hi_f | lo_f | hi_f] . [hi_w | hi_w | lo_w]
//                    = hi_f hi_w + lo_f hi_w + hi_f lo_w carries fp32-level accuracy (the dropped
//                    lo_f lo_w term is 2^-22 relative) through the TF32 tensor-core path at three
//                    times its work: this is how IEEE-mode fp32 layers reach the tensor cores.
//                    SPLIT_A lays a row out as [hi | lo | hi] (features, gradients), SPLIT_B as
//                    [hi | hi | lo] (weights).
#include <algorithm>

#include "common.cuh"

namespace spc {
namespace {

__device__ __forceinline__ float rna_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// ROUND mode on 16-byte vectors (the whole matrix is one contiguous run), by `blocks` CTAs of which this is `block`
__device__ __forceinline__ void round_rows(const float4* __restrict__ src, float4* __restrict__ dst, long long n4, unsigned block,
                                           unsigned blocks) {
  const long long stride = static_cast<long long>(blocks) * 256;
  for (long long i = block * 256ll + threadIdx.x; i < n4; i += stride) {
    float4 v = __ldg(src + i);
    v.x = rna_tf32(v.x); v.y = rna_tf32(v.y); v.z = rna_tf32(v.z); v.w = rna_tf32(v.w);
    dst[i] = v;
  }
}

// one thread per source element; Index: 32 bits where they hold the element count (four 64-bit divisions in a row
// are as long as the rest of the kernel on few elements)
template <typename Index>
__device__ __forceinline__ void prepare_rows(const float* __restrict__ src, float* __restrict__ dst, long long rows, int cols, int mode,
                                             unsigned block) {
  const Index i = static_cast<Index>(block) * 256 + threadIdx.x;
  if (i >= static_cast<Index>(rows * cols)) return;
  const Index r = i / static_cast<Index>(cols);
  const int c = static_cast<int>(i - r * cols);
  const float x = src[i];
  const float hi = rna_tf32(x);
  if (mode == SPC_TF32_ROUND) {
    dst[i] = hi;
    return;
  }
  const float lo = rna_tf32(x - hi);
  float* row = dst + static_cast<long long>(r) * 3 * cols;
  row[c] = hi;
  row[cols + c] = mode == SPC_TF32_SPLIT_A ? lo : hi;
  row[2 * cols + c] = mode == SPC_TF32_SPLIT_A ? hi : lo;
}

// weight [c_out, kv, c_in] -> dst [c_out, kv, m * c_in], or with `transpose` [c_in, kv, m * c_out]
// (dst[c][k][n] = w[n][k][c]; 2: dst[c][kv - 1 - k][n]): the reduction index innermost, as the forward-form kernel reads it.
template <typename Index>
__device__ __forceinline__ void prepare_weight(const float* __restrict__ w, float* __restrict__ dst, int c_out, int kv, int c_in,
                                               int transpose, int mode, unsigned block) {
  const Index i = static_cast<Index>(block) * 256 + threadIdx.x;
  if (i >= static_cast<Index>(c_out) * kv * c_in) return;
  const Index row_of = i / static_cast<Index>(c_in);  // (output channel, offset)
  const int c = static_cast<int>(i - row_of * c_in);
  const int n = static_cast<int>(row_of / static_cast<Index>(kv));
  const int k = static_cast<int>(row_of - static_cast<Index>(n) * kv);
  const int ko = transpose == 2 ? kv - 1 - k : k;
  const float x = w[i];
  const float hi = rna_tf32(x);
  const int m = mode == SPC_TF32_ROUND ? 1 : 3;
  const int red = transpose ? c_out : c_in;   // reduction extent of the prepared weight
  const int r = transpose ? n : c;            // this element's reduction index
  const int o = transpose ? c : n;            // and its output-channel index
  float* row = dst + (static_cast<long long>(o) * kv + ko) * m * red;
  row[r] = hi;
  if (m == 3) {
    const float lo = rna_tf32(x - hi);
    row[red + r] = mode == SPC_TF32_SPLIT_A ? lo : hi;
    row[2 * red + r] = mode == SPC_TF32_SPLIT_A ? hi : lo;
  }
}

struct Rows {
  const float* src;
  float* dst;
  long long rows;
  int cols, mode;
  bool wide;        // whole 16-byte vectors
  unsigned blocks;
};
struct Weight {
  const float* src;
  float* dst;
  int c_out, kv, c_in, transpose, mode;
  unsigned blocks;
};
// The first CTAs take the rows, the others the weight.
template <typename Index>
__global__ void __launch_bounds__(256) tf32_prepare_kernel(const __grid_constant__ Rows x, const __grid_constant__ Weight w) {
  if (blockIdx.x >= x.blocks)
    prepare_weight<Index>(w.src, w.dst, w.c_out, w.kv, w.c_in, w.transpose, w.mode, blockIdx.x - x.blocks);
  else if (x.wide)
    round_rows(reinterpret_cast<const float4*>(x.src), reinterpret_cast<float4*>(x.dst), x.rows * x.cols / 4, blockIdx.x, x.blocks);
  else
    prepare_rows<Index>(x.src, x.dst, x.rows, x.cols, x.mode, blockIdx.x);
}

int rows_of(const float* src, float* dst, int64_t rows, int cols, int mode, Rows* x) {
  if (!src || !dst || rows < 0 || cols <= 0 || mode < SPC_TF32_ROUND || mode > SPC_TF32_SPLIT_B)
    return fail(SPC_ERR_INVALID_ARGUMENT, "tf32_prepare: bad arguments");
  const long long total = static_cast<long long>(rows) * cols;
  const bool aligned = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
  const bool wide = mode == SPC_TF32_ROUND && total % 4 == 0 && aligned;
  const long long blocks = wide ? std::min<long long>(ceil_div(total / 4, 256), 8ll * sm_count()) : ceil_div(total, 256);
  *x = Rows{src, dst, rows, cols, mode, wide, static_cast<unsigned>(blocks)};
  return SPC_OK;
}
int weight_of(const float* weight, float* dst, int c_out, int kv, int c_in, int transpose, int mode, Weight* w) {
  if (!weight || !dst || c_out <= 0 || kv <= 0 || c_in <= 0 || mode < SPC_TF32_ROUND || mode > SPC_TF32_SPLIT_B)
    return fail(SPC_ERR_INVALID_ARGUMENT, "tf32_prepare_weight: bad arguments");
  const long long total = static_cast<long long>(c_out) * kv * c_in;
  *w = Weight{weight, dst, c_out, kv, c_in, transpose, mode, static_cast<unsigned>(ceil_div(total, 256))};
  return SPC_OK;
}
int launch(const Rows& x, const Weight& w, void* stream) {
  if (x.blocks + w.blocks == 0) return SPC_OK;
  const long long most = std::max<long long>(x.rows * x.cols, static_cast<long long>(w.c_out) * w.kv * w.c_in) + 256;
  const unsigned blocks = x.blocks + w.blocks;
  if (most <= 0xffffffffll) tf32_prepare_kernel<uint32_t><<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, w);
  else tf32_prepare_kernel<unsigned long long><<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, w);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace
}  // namespace spc

using namespace spc;

extern "C" int spc_tf32_prepare(const float* src, float* dst, int64_t rows, int cols, int mode, void* stream) {
  Rows x{};
  const int rc = rows_of(src, dst, rows, cols, mode, &x);
  return rc != SPC_OK ? rc : launch(x, Weight{}, stream);
}

extern "C" int spc_tf32_prepare_weight(const float* weight, float* dst, int c_out, int kv, int c_in, int transpose,
                                       int mode, void* stream) {
  Weight w{};
  const int rc = weight_of(weight, dst, c_out, kv, c_in, transpose, mode, &w);
  return rc != SPC_OK ? rc : launch(Rows{}, w, stream);
}

extern "C" int spc_tf32_prepare_operands(const float* src, float* dst, int64_t rows, int cols, int mode, const float* weight,
                                         float* weight_dst, int c_out, int kv, int c_in, int transpose, int weight_mode, void* stream) {
  Rows x{};
  Weight w{};
  int rc = rows_of(src, dst, rows, cols, mode, &x);
  if (rc == SPC_OK) rc = weight_of(weight, weight_dst, c_out, kv, c_in, transpose, weight_mode, &w);
  return rc != SPC_OK ? rc : launch(x, w, stream);
}
