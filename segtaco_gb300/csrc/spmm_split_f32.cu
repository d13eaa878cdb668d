// Split walk of merge-path chunks, fp32 dense operand.
#include "spmm_split_launch.cuh"

SEGTACO_DEFINE_SPLIT_LAUNCHER(launch_spmm_split_f32, float, SEGTACO_SPLIT_F32, SEGTACO_SPLIT_CASE)
