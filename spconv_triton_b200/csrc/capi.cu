// Housekeeping entry points of the C ABI: version, error text, device status, shape formulas.
#include <atomic>

#include "common.cuh"
#include "gemm_internal.cuh"

namespace spc {
char* error_buffer() {
  static thread_local char buf[512] = {0};
  return buf;
}
static std::atomic<long long> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// What a kernel cannot raise itself: a bounded wait that expired, an index row outside the grid.
__device__ int g_device_status = 0;

// Address of the current device's status word (every device that loads the
// library has its own copy of the symbol).
int* device_status_ptr() {
  static int* ptrs[kMaxDevices] = {nullptr};
  const int dev = current_device_slot();
  if (dev < 0) return nullptr;
  if (ptrs[dev] == nullptr) {
    void* raw = nullptr;
    if (cudaGetSymbolAddress(&raw, g_device_status) == cudaSuccess) ptrs[dev] = static_cast<int*>(raw);
  }
  return ptrs[dev];
}

namespace {

__global__ void post_status_kernel(const int* __restrict__ status, int* __restrict__ host_word) {
  *host_word = *status;
  __threadfence_system();
}

int read_device_status(cudaStream_t st, int* host_value) {
  int* ptr = device_status_ptr();
  *host_value = 0;
  if (ptr == nullptr) return SPC_OK;
  SPC_CUDA_OK(cudaMemcpyAsync(host_value, ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  SPC_CUDA_OK(cudaStreamSynchronize(st));
  if (*host_value != 0) SPC_CUDA_OK(cudaMemsetAsync(ptr, 0, sizeof(int), st));
  return SPC_OK;
}

}  // namespace
}  // namespace spc

using namespace spc;

extern "C" int spc_version(void) { return 100; }

extern "C" const char* spc_last_error(void) { return error_buffer(); }

extern "C" long long spc_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

extern "C" int spc_conv_output_size(int ndim, const int32_t* in_shape, const int32_t* ksize,
                                    const int32_t* stride, const int32_t* padding, const int32_t* dilation,
                                    int32_t* out_shape) {
  if (ndim < 1 || !in_shape || !ksize || !stride || !padding || !dilation || !out_shape)
    return fail(SPC_ERR_INVALID_ARGUMENT, "conv_output_size: bad arguments");
  for (int i = 0; i < ndim; ++i) {
    if (ksize[i] == -1) {
      out_shape[i] = 1;
      continue;
    }
    if (stride[i] <= 0) return fail(SPC_ERR_INVALID_ARGUMENT, "conv_output_size: stride must be positive");
    const long long num = static_cast<long long>(in_shape[i]) + 2ll * padding[i] -
                          static_cast<long long>(dilation[i]) * (ksize[i] - 1) - 1;
    // floor division, as Python's // does for negative numerators
    long long q = num / stride[i];
    if ((num % stride[i] != 0) && ((num < 0) != (stride[i] < 0))) --q;
    out_shape[i] = static_cast<int32_t>(q + 1);
  }
  return SPC_OK;
}

extern "C" int spc_deconv_output_size(int ndim, const int32_t* in_shape, const int32_t* ksize,
                                      const int32_t* stride, const int32_t* padding, const int32_t* dilation,
                                      const int32_t* out_padding, int32_t* out_shape) {
  (void)dilation;  // the reference's formula does not use it
  if (ndim < 1 || !in_shape || !ksize || !stride || !padding || !out_padding || !out_shape)
    return fail(SPC_ERR_INVALID_ARGUMENT, "deconv_output_size: bad arguments");
  for (int i = 0; i < ndim; ++i) {
    if (ksize[i] == -1) return fail(SPC_ERR_INVALID_ARGUMENT, "deconv don't support kernel_size < 0");
    out_shape[i] = (in_shape[i] - 1) * stride[i] - 2 * padding[i] + ksize[i] + out_padding[i];
  }
  return SPC_OK;
}

extern "C" int spc_post_device_status(int* pinned_host_word, void* stream) {
  if (pinned_host_word == nullptr) return fail(SPC_ERR_INVALID_ARGUMENT, "post_device_status: null mailbox");
  int* ptr = device_status_ptr();
  if (ptr == nullptr) return SPC_OK;
  // written by a kernel, not copied: a device-to-host copy would wait on the copy engine behind
  // whatever transfer the application has in flight and hold up the stream
  post_status_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(ptr, pinned_host_word);
  SPC_LAUNCH_OK();
  return SPC_OK;
}

extern "C" int spc_check_device_status(void* stream) {
  int value = 0;
  const int rc = read_device_status(static_cast<cudaStream_t>(stream), &value);
  if (rc != SPC_OK) return rc;
  if (value == SPC_ERR_INVALID_ARGUMENT)
    return fail(value, "a rulebook kernel met an index row outside batch_size / spatial_shape (device status %d)", value);
  if (value != 0) return fail(value, "a kernel of this library recorded device status %d (a bounded wait expired)", value);
  return SPC_OK;
}
