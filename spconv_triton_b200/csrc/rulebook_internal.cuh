// Internal (non-ABI) rulebook entry points for callers inside the library that chain rulebooks.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace spc {

// The strided / transposed layer whose OUTPUT rows, all of them and in its order, are the input rows
// of the rulebook being generated.  When that layer numbered its outputs through a bitmap of its
// output grid, the bitmap and its prefix sums are still in its workspace and are exactly the input
// occupancy bitmap the new rulebook would otherwise build (clear, mark, count, scan) -- and the
// input hash table is not needed either, because the rows are the ranks of the bits.
struct RulebookProducer {
  const spc_geometry* geom;
  const void* workspace;  // as spc_rulebook_prepare left it
  int64_t n_in;           // the n_in that workspace was laid out for
};

// What rulebook_tables_chained writes; every pointer may be null, the row-major tables are 16-byte aligned.
struct RulebookTables {
  int32_t* out_indices;   // [n_out, ndim + 1], strided / transposed layers
  int32_t* fwd_colmajor;  // [kv, n_out]
  int32_t* fwd_rowmajor;  // [n_out, kvp], -1 padded
  int32_t* fwd_order;     // [n_out]: rows grouped so that the 128 rows of a gather-GEMM tile share offsets (kv <= 32)
  int32_t* bwd_colmajor;  // the same for the input side of a strided / transposed layer
  int32_t* bwd_rowmajor;
  int32_t* bwd_order;
};

// spc_rulebook_prepare / spc_rulebook_tables with an optional producer (nullptr = the plain calls).
int rulebook_prepare_chained(const spc_geometry* g, const int32_t* indices, int64_t n_in, void* workspace,
                             size_t workspace_bytes, int64_t* n_out_host, const RulebookProducer* producer,
                             cudaStream_t stream);
// Whether rulebook_prepare_chained would take all it needs from `producer`: it then reads nothing of `indices`.
bool rulebook_adopts(const spc_geometry* g, int64_t n_in, const RulebookProducer* producer);
int rulebook_tables_chained(const spc_geometry* g, const int32_t* indices, int64_t n_in, int64_t n_out, void* workspace,
                            size_t workspace_bytes, const RulebookTables& tables, const RulebookProducer* producer,
                            cudaStream_t stream);

// Numbers that the host needs during a call: kernels write words 1.. of the box and the ticket to word 0 last
// (__threadfence_system between); the wait ends when the ticket is there.
int host_mailbox(volatile int** out, int* ticket);
int wait_for_ticket(volatile int* box, int ticket, cudaStream_t st);

}  // namespace spc
