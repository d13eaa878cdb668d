// Row-slot walk of row blocks, bf16 dense operand (bit patterns as uint16_t).
#include "spmm_rows_launch.cuh"

SEGTACO_DEFINE_ROWS_LAUNCHER(launch_spmm_slots_bf16, uint16_t, SEGTACO_ROWS_BF16)
