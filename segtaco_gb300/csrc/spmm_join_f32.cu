// Split walk of merge-path chunks whose cut rows are joined, fp32 dense operand.
#include "spmm_split_launch.cuh"

SEGTACO_DEFINE_SPLIT_LAUNCHER(launch_spmm_join_f32, float, SEGTACO_SPLIT_F32, SEGTACO_JOIN_CASE)
