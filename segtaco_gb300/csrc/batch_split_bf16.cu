// batch_split_bf16.cu -- persistent batched launchers of the split walk, dense operand bf16.
#include "batch.cuh"
#include "internal.h"
#include "spmm_split_launch.cuh"

namespace segtaco {

#define SEGTACO_BATCH_SPLIT_BYTES(V)                                                       \
  (split_bytes<V>(g.items) +                                                               \
   (g.nprobs <= kBatchSmemProblems ? (size_t)g.nprobs * sizeof(long long) : 0))
#define SEGTACO_BATCH_SPLIT_CASE(BT, E, C, G)                                              \
  case SEGTACO_SPLIT_KEY(E, C, G):                                                         \
    spmm_batch_split_kernel<BT, E, C, G>                                                   \
        <<<g.grid, kSpmmCta, SEGTACO_BATCH_SPLIT_BYTES((E) * (C)), s>>>(                   \
            static_cast<const BatchProblem<BT> *>(g.probs), g.item_begin, g.nprobs,        \
            g.total_items, g.queue, g.gate, g.items);                                      \
    break;
#define SEGTACO_BATCH_SPLIT_OCC(BT, E, C, G)                                               \
  case SEGTACO_SPLIT_KEY(E, C, G):                                                         \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(                                     \
        out, spmm_batch_split_kernel<BT, E, C, G>, kSpmmCta,                               \
        SEGTACO_BATCH_SPLIT_BYTES((E) * (C)));                                             \
    break;

int launch_batch_split_bf16(const BatchGroupLaunch &g, cudaStream_t s) {
  switch (SEGTACO_SPLIT_KEY(g.elems, g.V / g.elems, g.G)) {
    SEGTACO_SPLIT_BF16(SEGTACO_BATCH_SPLIT_CASE)
    default:
      return set_error(SEGTACO_EUNSUPPORTED, "batch: no split variant E=%d V=%d G=%d", g.elems,
                       g.V, g.G);
  }
  return check_launch("spmm_batch_split_kernel");
}

int batch_split_blocks_per_sm_bf16(const BatchGroupLaunch &g, int *out) {
  cudaError_t e = cudaErrorInvalidValue;
  switch (SEGTACO_SPLIT_KEY(g.elems, g.V / g.elems, g.G)) {
    SEGTACO_SPLIT_BF16(SEGTACO_BATCH_SPLIT_OCC)
    default: break;
  }
  return check_cuda(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(batch split)");
}

}  // namespace segtaco
