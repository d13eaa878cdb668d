// spmm_split_launch.cuh -- launchers of the split walk (spmm_split.cuh), one
// per dense type (spmm_split_<dtype>.cu), over its compiled lane shapes.
#pragma once

#include "internal.h"
#include "spmm_launch.cuh"
#include "spmm_split.cuh"

// Lane shapes (E, C, G), those that the planner's split_shape chooses: one chunk of
// 16 bytes (bf16: or 8) per lane, or 1- or 2-element chunks, several per lane.
#define SEGTACO_SPLIT_NARROW(X, BT)                                                        \
  X(BT, 1, 1, 1) X(BT, 1, 1, 2) X(BT, 1, 1, 4) X(BT, 1, 1, 8) X(BT, 1, 2, 8) X(BT, 1, 3, 8) \
  X(BT, 1, 2, 16) X(BT, 1, 3, 16) X(BT, 1, 4, 16) X(BT, 1, 3, 32) X(BT, 1, 4, 32)          \
  X(BT, 2, 1, 1) X(BT, 2, 1, 2) X(BT, 2, 1, 4) X(BT, 2, 1, 8) X(BT, 2, 2, 8) X(BT, 2, 3, 8) \
  X(BT, 2, 1, 32) X(BT, 2, 2, 32)
#define SEGTACO_SPLIT_WIDE(X, BT, E)                                                       \
  X(BT, E, 1, 1) X(BT, E, 1, 2) X(BT, E, 1, 4) X(BT, E, 1, 8) X(BT, E, 1, 16)
#define SEGTACO_SPLIT_F32(X)                                                               \
  SEGTACO_SPLIT_WIDE(X, float, 4) X(float, 4, 1, 32) SEGTACO_SPLIT_NARROW(X, float)
#define SEGTACO_SPLIT_BF16(X)                                                              \
  SEGTACO_SPLIT_WIDE(X, uint16_t, 8) SEGTACO_SPLIT_WIDE(X, uint16_t, 4)                    \
  X(uint16_t, 4, 1, 32) SEGTACO_SPLIT_NARROW(X, uint16_t)

#define SEGTACO_SPLIT_KEY(E, C, G) ((E)*10000 + (C)*100 + (G))
#define SEGTACO_SPLIT_RUN(BT, E, C, G, JOIN)                                               \
  case SEGTACO_SPLIT_KEY(E, C, G):                                                         \
    spmm_split_kernel<BT, E, C, G, JOIN>                                                   \
        <<<grid, kSpmmCta, split_bytes<(E) * (C)>(L.split_items), s>>>(a, L.split_items);  \
    break;
#define SEGTACO_SPLIT_CASE(BT, E, C, G) SEGTACO_SPLIT_RUN(BT, E, C, G, false)
#define SEGTACO_JOIN_CASE(BT, E, C, G) SEGTACO_SPLIT_RUN(BT, E, C, G, true)
#define SEGTACO_DEFINE_SPLIT_LAUNCHER(NAME, BT, LIST, CASE)                                \
  namespace segtaco {                                                                      \
  int NAME(const SpmmLaunch &L, cudaStream_t s) {                                          \
    const SpmmArgs<BT> a = make_spmm_args<BT>(L);                                          \
    const long long W = (long long)L.V * L.G;                                              \
    const dim3 grid((unsigned)((L.units + kSpmmWarps - 1) / kSpmmWarps),                   \
                    (unsigned)((L.N + W - 1) / W), 1);                                     \
    const int E = L.split_elems;                                                           \
    switch (SEGTACO_SPLIT_KEY(E, L.V / E, L.G)) {                                          \
      LIST(CASE)                                                                           \
      default:                                                                             \
        return set_error(SEGTACO_EUNSUPPORTED, #NAME ": no variant E=%d V=%d G=%d", E, L.V, L.G); \
    }                                                                                      \
    return check_launch(#NAME);                                                            \
  }                                                                                        \
  }

namespace segtaco {
template <int V> inline size_t split_bytes(int D) {
  return (size_t)kSpmmWarps * split_words<V>(D) * sizeof(int);
}
}  // namespace segtaco
