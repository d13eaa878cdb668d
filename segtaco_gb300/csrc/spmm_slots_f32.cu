// Row-slot walk of row blocks, fp32 dense operand.
#include "spmm_rows_launch.cuh"

SEGTACO_DEFINE_ROWS_LAUNCHER(launch_spmm_slots_f32, float, SEGTACO_ROWS_F32)
