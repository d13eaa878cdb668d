// spmm_rows_launch.cuh -- launchers of the row-slot walk (spmm_rows.cuh), one per dense
// type (spmm_slots_<dtype>.cu), over the lane shapes of the split walk with at least two
// slots (and the one-slot shapes of 1- and 2-element chunks).
#pragma once

#include "spmm_rows.cuh"
#include "spmm_split_launch.cuh"

#define SEGTACO_ROWS_WIDE(X, BT, E) X(BT, E, 1, 1) X(BT, E, 1, 2) X(BT, E, 1, 4) X(BT, E, 1, 8)
#define SEGTACO_ROWS_F32(X) \
  SEGTACO_ROWS_WIDE(X, float, 4) X(float, 4, 1, 16) SEGTACO_SPLIT_NARROW(X, float)
#define SEGTACO_ROWS_BF16(X)                                                               \
  SEGTACO_ROWS_WIDE(X, uint16_t, 8) X(uint16_t, 8, 1, 16) SEGTACO_ROWS_WIDE(X, uint16_t, 4) \
  X(uint16_t, 4, 1, 16) SEGTACO_SPLIT_NARROW(X, uint16_t)
#define SEGTACO_ROWS_CASE(BT, E, C, G)                                                     \
  case SEGTACO_SPLIT_KEY(E, C, G):                                                         \
    if (L.coop)                                                                            \
      launch_seg(spmm_rows_kernel<BT, E, C, G, true>, grid, s, a, L.carveout);             \
    else                                                                                   \
      launch_seg(spmm_rows_kernel<BT, E, C, G, false>, grid, s, a, L.carveout);            \
    break;
#define SEGTACO_DEFINE_ROWS_LAUNCHER(NAME, BT, LIST)                                       \
  namespace segtaco {                                                                      \
  int NAME(const SpmmLaunch &L, cudaStream_t s) {                                          \
    const SpmmArgs<BT> a = make_spmm_args<BT>(L);                                          \
    const long long W = (long long)L.V * L.G;                                              \
    const dim3 grid((unsigned)((L.units + kSpmmWarps - 1) / kSpmmWarps),                   \
                    (unsigned)((L.N + W - 1) / W), 1);                                     \
    const int E = L.split_elems;                                                           \
    switch (SEGTACO_SPLIT_KEY(E, L.V / E, L.G)) {                                          \
      LIST(SEGTACO_ROWS_CASE)                                                              \
      default:                                                                             \
        return set_error(SEGTACO_EUNSUPPORTED, #NAME ": no variant E=%d V=%d G=%d", E, L.V, L.G); \
    }                                                                                      \
    return check_launch(#NAME);                                                            \
  }                                                                                        \
  }
