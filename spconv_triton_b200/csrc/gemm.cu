// C-ABI entry points of the implicit gather-GEMM and the choice between the
// tcgen05 kernel and the CUDA-core kernels.
#include <algorithm>

#include "common.cuh"
#include "gemm_internal.cuh"

using namespace spc;

namespace {

// (the code of a kernel that is gone)
int known_path(int path) { return path == SPC_GEMM_TCGEN05_CPASYNC ? SPC_GEMM_AUTO : path; }

// The tensor-core kernel takes 16-bit inputs always and fp32 inputs only when
// the caller allows TF32; IEEE fp32 stays on the CUDA cores.
bool want_tc(int path, int n_dim, int r_dim, int kv, int dtype, int out_dtype, int precision, bool transposed,
             int* status) {
  *status = SPC_OK;
  const bool ok = gather_gemm_tma_supported(n_dim, r_dim, kv, dtype, out_dtype, precision, transposed);
  if (path == SPC_GEMM_SIMT) return false;
  if (path == SPC_GEMM_TCGEN05) {
    if (!ok) *status = fail(SPC_ERR_UNSUPPORTED, "tcgen05 path does not take this shape/dtype "
                            "(n=%d r=%d kv=%d dtype=%d precision=%d)", n_dim, r_dim, kv, dtype, precision);
    return ok;
  }
  return ok;
}

// (tensors of the caching allocator are; a caller's view need not be)
bool f32_aligned(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) == 0;
}

}  // namespace

extern "C" int spc_conv_small(int64_t rows, int n_dim, int r_dim, int kv) {
  return rows > 0 && n_dim > 0 && r_dim > 0 && kv > 0 && gather_gemm_small_takes(rows, n_dim, r_dim, kv) ? 1 : 0;
}

extern "C" int spc_conv_forward_needs_colmajor(int c_in, int c_out, int kv, int dtype, int out_dtype, int precision,
                                               int path) {
  path = known_path(path);
  if (path != SPC_GEMM_SIMT && gather_gemm_tma_supported(c_out, c_in, kv, dtype, out_dtype, precision, false)) return 0;
  return path == SPC_GEMM_AUTO && gather_gemm_f32_supported(c_out, c_in, dtype, out_dtype) ? 0 : 1;
}

extern "C" int spc_conv_forward(const void* features, const void* weight, const void* bias,
                                const int32_t* pair_fwd, const int32_t* pair_fwd_rowmajor,
                                const int32_t* mask_argsort, void* out,
                                int64_t n_in, int64_t n_out, int c_in, int c_out, int kv, int dtype,
                                int out_dtype, int precision, int path, const float* out_scale,
                                const float* out_shift, int act, float act_alpha, void* stream) {
  return spc_conv_forward_residual(features, weight, bias, pair_fwd, pair_fwd_rowmajor, mask_argsort, out, n_in, n_out,
                                   c_in, c_out, kv, dtype, out_dtype, precision, path, out_scale, out_shift, act,
                                   act_alpha, nullptr, stream);
}

extern "C" int spc_conv_forward_residual(const void* features, const void* weight, const void* bias,
                                         const int32_t* pair_fwd, const int32_t* pair_fwd_rowmajor,
                                         const int32_t* mask_argsort, void* out, int64_t n_in, int64_t n_out,
                                         int c_in, int c_out, int kv, int dtype, int out_dtype, int precision,
                                         int path, const float* out_scale, const float* out_shift, int act,
                                         float act_alpha, const void* residual, void* stream) {
  path = known_path(path);
  if (!features || !weight || !out || n_in < 0 || n_out < 0 || c_in <= 0 || c_out <= 0 || kv <= 0)
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_forward: bad arguments");
  if (!pair_fwd && (!pair_fwd_rowmajor ||
                    spc_conv_forward_needs_colmajor(c_in, c_out, kv, dtype, out_dtype, precision, path)))
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_forward: this layer reads the column-major table");
  if (out_scale != nullptr && out_shift == nullptr)
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_forward: out_scale needs out_shift");
  if (n_out == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Epilogue epi;
  epi.bias = bias; epi.scale = out_scale; epi.shift = out_shift; epi.act = act; epi.alpha = act_alpha;
  epi.residual = residual;
  if (residual != nullptr && (reinterpret_cast<uintptr_t>(residual) & 15u) != 0)
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_forward: the residual must be 16-byte aligned");
  int status;
  if (want_tc(path, c_out, c_in, kv, dtype, out_dtype, precision, false, &status)) {
    return gather_gemm_tma(features, weight, epi, pair_fwd, pair_fwd_rowmajor, mask_argsort, out, n_in, n_out, c_out, c_in, kv,
                           /*transposed_weight=*/false, /*reversed=*/false, dtype, out_dtype, precision, st);
  }
  if (status != SPC_OK) return status;
  if (path == SPC_GEMM_AUTO && dtype == SPC_F32 && out_dtype == SPC_F32 && pair_fwd_rowmajor != nullptr &&
      gather_gemm_small_takes(n_out, c_out, c_in, kv) && f32_aligned(features, weight, pair_fwd_rowmajor))
    return gather_gemm_small(features, weight, epi, pair_fwd_rowmajor, out, n_out, c_out, c_in, kv, false, false, st);
  if (path == SPC_GEMM_AUTO && gather_gemm_f32_supported(c_out, c_in, dtype, out_dtype) && f32_aligned(features, weight, out))
    return gather_gemm_f32(features, weight, epi, pair_fwd, pair_fwd_rowmajor, mask_argsort, out, n_out, c_out, c_in, kv,
                           /*transposed_weight=*/false, /*reversed=*/false, st);
  if (!pair_fwd) return fail(SPC_ERR_INVALID_ARGUMENT, "conv_forward: this layer reads the column-major table");
  // weight[n, k, c]: reduction index c has stride 1, output channel n stride kv*c_in.
  return gather_gemm_simt(features, weight, epi, pair_fwd, mask_argsort, out, n_out, c_out, c_in, kv,
                          /*s_wk=*/c_in, /*s_wr=*/1, /*s_wn=*/static_cast<long long>(kv) * c_in, dtype,
                          out_dtype, st);
}

extern "C" int spc_conv_backward_input(const void* grad_out, const void* weight, const int32_t* pair_bwd,
                                       const int32_t* pair_bwd_rowmajor, const int32_t* mask_argsort, void* din, int64_t n_in, int64_t n_out,
                                       int c_in, int c_out, int kv, int dtype, int precision, int path,
                                       void* stream) {
  if (!pair_bwd) return fail(SPC_ERR_INVALID_ARGUMENT, "conv_backward_input: bad arguments");
  return spc_conv_backward_input_tables(grad_out, weight, pair_bwd, pair_bwd_rowmajor, mask_argsort, din, n_in, n_out, c_in, c_out,
                                        kv, 0, dtype, precision, path, stream);
}

extern "C" int spc_conv_backward_input_needs_colmajor(int c_in, int c_out, int kv, int dtype, int precision, int path) {
  path = known_path(path);
  if (path != SPC_GEMM_SIMT && gather_gemm_tma_supported(c_in, c_out, kv, dtype, dtype, precision, true)) return 0;
  return path == SPC_GEMM_AUTO && gather_gemm_f32_supported(c_in, c_out, dtype, dtype) ? 0 : 1;
}

extern "C" int spc_conv_backward_input_tables(const void* grad_out, const void* weight, const int32_t* pair_bwd,
                                              const int32_t* pair_bwd_rowmajor, const int32_t* mask_argsort, void* din,
                                              int64_t n_in, int64_t n_out, int c_in, int c_out, int kv, int reversed, int dtype,
                                              int precision, int path, void* stream) {
  path = known_path(path);
  if (!grad_out || !weight || !din || n_in < 0 || n_out < 0 || c_in <= 0 || c_out <= 0 || kv <= 0)
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_backward_input: bad arguments");
  if (!pair_bwd && (!pair_bwd_rowmajor || spc_conv_backward_input_needs_colmajor(c_in, c_out, kv, dtype, precision, path)))
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_backward_input: this layer reads the column-major table");
  if (n_in == 0) return SPC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int status;
  if (want_tc(path, c_in, c_out, kv, dtype, dtype, precision, true, &status)) {
    return gather_gemm_tma(grad_out, weight, Epilogue{}, pair_bwd, pair_bwd_rowmajor, mask_argsort, din, n_out, n_in, c_in, c_out, kv,
                           /*transposed_weight=*/true, reversed != 0, dtype, dtype, precision, st);
  }
  if (status != SPC_OK) return status;
  if (path == SPC_GEMM_AUTO && dtype == SPC_F32 && pair_bwd_rowmajor != nullptr && gather_gemm_small_takes(n_in, c_in, c_out, kv) &&
      f32_aligned(grad_out, weight, pair_bwd_rowmajor))
    return gather_gemm_small(grad_out, weight, Epilogue{}, pair_bwd_rowmajor, din, n_in, c_in, c_out, kv, true, reversed != 0, st);
  if (path == SPC_GEMM_AUTO && gather_gemm_f32_supported(c_in, c_out, dtype, dtype) && f32_aligned(grad_out, weight, din))
    return gather_gemm_f32(grad_out, weight, Epilogue{}, pair_bwd, pair_bwd_rowmajor, mask_argsort, din, n_in, c_in, c_out, kv,
                           /*transposed_weight=*/true, reversed != 0, st);
  if (!pair_bwd) return fail(SPC_ERR_INVALID_ARGUMENT, "conv_backward_input: this layer reads the column-major table");
  // output channel is c (stride 1), reduction index is n (stride kv*c_in); reversed offsets: from the last one down
  const char* w = static_cast<const char*>(weight) + (reversed ? static_cast<size_t>(kv - 1) * c_in * dtype_size(dtype) : 0);
  return gather_gemm_simt(grad_out, w, Epilogue{}, pair_bwd, mask_argsort, din, n_in, c_in, c_out, kv,
                          /*s_wk=*/reversed ? -static_cast<long long>(c_in) : c_in, /*s_wr=*/static_cast<long long>(kv) * c_in, /*s_wn=*/1,
                          dtype, dtype, st);
}

extern "C" size_t spc_conv_backward_weight_workspace_bytes(int64_t n_out, int c_in, int c_out, int kv) {
  if (n_out < 0 || c_in <= 0 || c_out <= 0 || kv <= 0) return 0;
  // enough for whichever kernel the call ends up using
  return std::max(std::max(wgrad_split(n_out, c_in, c_out, kv).bytes, wgrad_f32_split(n_out, c_in, c_out, kv).bytes),
                  wgrad_tc_split(n_out, c_in, c_out, kv).bytes);
}

extern "C" int spc_conv_backward_weight(const void* features, const void* grad_out, const int32_t* pair_fwd,
                                        void* dweight, void* workspace, size_t workspace_bytes, int64_t n_in,
                                        int64_t n_out, int c_in, int c_out, int kv, int dtype, int precision,
                                        int path, void* stream) {
  (void)n_in;
  (void)precision;
  path = known_path(path);
  if (!features || !grad_out || !pair_fwd || !dweight || n_out < 0 || c_in <= 0 || c_out <= 0 || kv <= 0)
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_backward_weight: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n_out == 0) {
    SPC_CUDA_OK(cudaMemsetAsync(dweight, 0, static_cast<size_t>(c_out) * kv * c_in * dtype_size(dtype), st));
    return SPC_OK;
  }
  if (path != SPC_GEMM_SIMT && wgrad_tc_supported(c_in, c_out, kv, dtype)) {
    const WgradSplit ts = wgrad_tc_split(n_out, c_in, c_out, kv);
    if (!workspace || workspace_bytes < ts.bytes)
      return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "conv_backward_weight: workspace %zu < %zu bytes", workspace_bytes,
                  ts.bytes);
    const int rc = wgrad_tc(features, grad_out, pair_fwd, static_cast<float*>(workspace), n_out, c_in, c_out, kv,
                            dtype, ts, st);
    if (rc != SPC_OK) return rc;
    return wgrad_reduce(static_cast<const float*>(workspace), dweight, static_cast<long long>(c_out) * kv * c_in,
                        ts.splits, dtype, st);
  }
  if (path == SPC_GEMM_TCGEN05)
    return fail(SPC_ERR_UNSUPPORTED, "conv_backward_weight: the tcgen05 kernel does not take this shape/dtype "
                "(c_in=%d c_out=%d dtype=%d)", c_in, c_out, dtype);
  if (path == SPC_GEMM_AUTO && wgrad_f32_supported(c_in, c_out, dtype) && f32_aligned(features, grad_out, workspace)) {
    const WgradSplit fs = wgrad_f32_split(n_out, c_in, c_out, kv);
    if (!workspace || workspace_bytes < fs.bytes)
      return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "conv_backward_weight: workspace %zu < %zu bytes", workspace_bytes, fs.bytes);
    const int rc = wgrad_f32(features, grad_out, pair_fwd, static_cast<float*>(workspace), n_out, c_in, c_out, kv, fs, st);
    if (rc != SPC_OK) return rc;
    return wgrad_reduce(static_cast<const float*>(workspace), dweight, static_cast<long long>(c_out) * kv * c_in, fs.splits, dtype, st);
  }
  const WgradSplit s = wgrad_split(n_out, c_in, c_out, kv);
  if (!workspace || workspace_bytes < s.bytes)
    return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "conv_backward_weight: workspace %zu < %zu bytes", workspace_bytes,
                s.bytes);
  return wgrad_simt(features, grad_out, pair_fwd, dweight, static_cast<float*>(workspace), n_out, c_in, c_out,
                    kv, dtype, st);
}
