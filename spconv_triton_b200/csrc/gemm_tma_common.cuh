// What the two tcgen05 gather-GEMMs share: TMA wrappers, the row copy, and the tensor map of the weight.
#pragma once

#include <cuda.h>

#include "tc_common.cuh"

namespace spc {
namespace tc {

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__host__ __device__ inline uint32_t layout_type_for(int row_bytes) {
  return row_bytes == 128 ? 2u : (row_bytes == 64 ? 4u : 6u);
}

// 16-byte copy into shared memory; zeros instead when row < 0 (the source is then not read).
__device__ __forceinline__ void cp_async16_row(uint32_t dst, const void* src, int row) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.lt.s32 p, %2, 0;\n\t"
      "cp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(dst), "l"(src), "r"(row)
      : "memory");
}

constexpr int kMostSmem = 226 * 1024;  // dynamic shared memory of a CTA

// ---- host side ------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  // The driver call needs the thread's context, which a thread that has made no runtime call yet (autograd's,
  // whose first step may be an input gradient) does not have: an empty free makes it current.
  static thread_local bool current = false;
  if (!current) current = cudaFree(nullptr) == cudaSuccess;
  // (a thread that comes while another looks the function up waits for it)
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* raw = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &raw, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(raw);
  }();
  return fn;
}

inline CUtensorMapSwizzle swizzle_for(int row_bytes) {
  return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                          : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

inline CUtensorMapDataType tma_dtype(int dtype) {
  return dtype == SPC_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                          : (dtype == SPC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32);
}

// Swizzle span of rows holding `elems` contiguous elements: the widest of 128, 64 and 32 bytes that
// divides them (48 channels of 16 bits: 32 bytes, 96 channels: 64), so that no copy is padding.
inline int row_span(int elems, int elem_size) {
  const int bytes = elems * elem_size;
  return bytes % 128 == 0 ? 128 : bytes % 64 == 0 ? 64 : 32;
}

// The KRSC weight [c_out][kv][c_in] as a 3-D tensor (c_in innermost): boxes of `epr` reduction elements of one offset and all
// n_dim output channels, or, read transposed, of one block of output channels and `epr` reduction rows.
inline int weight_map(CUtensorMap* map, const void* w, int n_dim, int r_dim, int kv, bool transposed_weight, int b_row_bytes, int epr, int dtype) {
  const int elem = dtype == SPC_F32 ? 4 : 2;
  const int c_in = transposed_weight ? n_dim : r_dim, c_out = transposed_weight ? r_dim : n_dim;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(c_in), static_cast<cuuint64_t>(kv), static_cast<cuuint64_t>(c_out)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(c_in) * elem, static_cast<cuuint64_t>(kv) * c_in * elem};
  cuuint32_t box[3];
  if (transposed_weight) {
    box[0] = static_cast<cuuint32_t>(b_row_bytes / elem);  // output channels of one column block
    box[1] = 1;
    box[2] = static_cast<cuuint32_t>(epr);                 // reduction rows of one stage
  } else {
    box[0] = static_cast<cuuint32_t>(epr);
    box[1] = 1;
    box[2] = static_cast<cuuint32_t>(n_dim);
  }
  const cuuint32_t estr[3] = {1, 1, 1};
  const EncodeTiledFn encode = encode_fn();
  if (encode == nullptr) return fail(SPC_ERR_CUDA, "the driver has no cuTensorMapEncodeTiled");
  const CUresult r = encode(map, tma_dtype(dtype), 3, const_cast<void*>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 swizzle_for(b_row_bytes), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? SPC_OK : fail(SPC_ERR_CUDA, "cuTensorMapEncodeTiled(B) failed: %d", static_cast<int>(r));
}

}  // namespace tc
}  // namespace spc
