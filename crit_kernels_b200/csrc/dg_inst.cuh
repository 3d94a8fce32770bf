// Expands to the table of the kernels of one format and activation type, by steps per stage (1, 2), then the same for small
// launches, and activation rows (1..16): instances for 1-4, 5-8 and 9-16 rows. BF16 has stages of one step only; small
// launches only where dg::small_capable.
#pragma once
#include "dg_kernel.cuh"
#include "dg_tables.h"

#define DG_ROWS(A, B, C) {A, A, A, A, B, B, B, B, C, C, C, C, C, C, C, C}
#define DG_K(FMT, NT, M, STEPS, SMALL, XT)                                                                                       \
  reinterpret_cast<const void*>(                                                                                                 \
      &dg::gemv_kernel<FMT, NT, dg::resident_capable(FMT, M), (FMT) == dg::FMT_BF16 ? 1 : STEPS, SMALL, XT>)
#define DG_STEPS(FMT, STEPS, SMALL, XT)                                                                                          \
  DG_ROWS(DG_K(FMT, 1, 1, STEPS, dg::small_capable(1) && SMALL, XT),                                                        \
          DG_K(FMT, 1, 5, STEPS, dg::small_capable(5) && SMALL, XT), DG_K(FMT, 2, 9, STEPS, false, XT))
#define DG_TABLE(NAME, FMT, XT)                                                                                                  \
  const void* const NAME[4][16] = {DG_STEPS(FMT, 1, false, XT), DG_STEPS(FMT, 2, false, XT), DG_STEPS(FMT, 1, true, XT),         \
                                   DG_STEPS(FMT, 2, true, XT)};
#define DG_BATCH_K(FMT, NT, M, STEPS, XT)                                                                                        \
  reinterpret_cast<const void*>(&dg::gemv_batch_kernel<FMT, NT, dg::resident_capable(FMT, M), STEPS, XT>)
#define DG_BATCH_STEPS(FMT, STEPS, XT) \
  DG_ROWS(DG_BATCH_K(FMT, 1, 1, STEPS, XT), DG_BATCH_K(FMT, 1, 5, STEPS, XT), DG_BATCH_K(FMT, 2, 9, STEPS, XT))
#define DG_BATCH_TABLE(NAME, FMT, XT) \
  const void* const NAME[2][16] = {DG_BATCH_STEPS(FMT, 1, XT), DG_BATCH_STEPS(FMT, 2, XT)};
