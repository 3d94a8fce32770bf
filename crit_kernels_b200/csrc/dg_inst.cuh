// Expands to the table of the kernels of one format and activation type, by steps per stage (1, 2) and activation rows
// (1..16): instances for 1-4, 5-8 and 9-16 rows. BF16 has stages of one step only.
#pragma once
#include "dg_kernel.cuh"
#include "dg_tables.h"

#define DG_ROWS(A, B, C) {A, A, A, A, B, B, B, B, C, C, C, C, C, C, C, C}
#define DG_K(KERNEL, FMT, NT, M, STEPS, XT)                                                                         \
  reinterpret_cast<const void*>(&dg::KERNEL<FMT, NT, dg::resident_capable(FMT, M), (FMT) == dg::FMT_BF16 ? 1 : STEPS, XT>)
#define DG_STEPS(KERNEL, FMT, STEPS, XT)                                                                            \
  DG_ROWS(DG_K(KERNEL, FMT, 1, 1, STEPS, XT), DG_K(KERNEL, FMT, 1, 5, STEPS, XT), DG_K(KERNEL, FMT, 2, 9, STEPS, XT))
#define DG_TABLE(NAME, FMT, XT) \
  const void* const NAME[2][16] = {DG_STEPS(gemv_kernel, FMT, 1, XT), DG_STEPS(gemv_kernel, FMT, 2, XT)};
#define DG_BATCH_TABLE(NAME, FMT, XT) \
  const void* const NAME[2][16] = {DG_STEPS(gemv_batch_kernel, FMT, 1, XT), DG_STEPS(gemv_batch_kernel, FMT, 2, XT)};
