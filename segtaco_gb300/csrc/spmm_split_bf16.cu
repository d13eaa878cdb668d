// Split walk of merge-path chunks, bf16 dense operand (bit patterns as uint16_t).
#include "spmm_split_launch.cuh"

SEGTACO_DEFINE_SPLIT_LAUNCHER(launch_spmm_split_bf16, uint16_t, SEGTACO_SPLIT_BF16, SEGTACO_SPLIT_CASE)
