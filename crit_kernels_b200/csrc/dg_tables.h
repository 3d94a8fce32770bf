// Kernel tables: one entry per steps per stage (1, 2; the same for small launches) and activation-row count (1..16), defined
// by the instantiation units (dg_inst_*.cu) and read by the dispatcher (dg_abi.cu).
#pragma once

extern const void* const dg_table_bf16[4][16];
extern const void* const dg_table_fp8_bf16[4][16];
extern const void* const dg_table_fp8_f16[4][16];
extern const void* const dg_table_mxfp8_bf16[4][16];
extern const void* const dg_table_mxfp8_f16[4][16];
extern const void* const dg_table_nvfp4_bf16[4][16];
extern const void* const dg_table_nvfp4_f16[4][16];
extern const void* const dg_batch_table_nvfp4_bf16[2][16];   // gemv_batch_kernel, NVFP4, BF16 activations
