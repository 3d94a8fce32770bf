// C ABI of the B200 decode GEMVs (include/decode_gemv_b200.h): argument validation, launch planning, dispatch.
//
// Mirrors the reference's raw CUDA API (decode-gemv/decode_gemv_cuda/decode_gemv.cu:378-427): the same refusals
// (cudaErrorInvalidValue for M outside 1..16, N < 1, K not a multiple the format needs, both or neither FP8 scale),
// cudaGetLastError() after the launch, no allocation and no host synchronisation on the enqueue path.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "../../include/decode_gemv_b200.h"
#include "dg_kernel.cuh"
#include "dg_tables.h"

namespace {

using dg::Params;

// Error word the kernels' bounded waits report into: one per device that loads the library.
__device__ int dg_status_word;

constexpr int kMaxDevices = 64;

struct DeviceState {
  std::atomic<int> ready{0};   // 0 unknown, 1 initialised, -1 unusable
  int sms = 0;
  int* status = nullptr;
};

// cuTensorMapEncodeTiled, looked up through the runtime so that the library does not link against libcuda.
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<EncodeTiled>(ptr);
  }();
  return fn;
}

// Tensor maps. An encoded map is a function of the values it is asked for alone, and a decode loop asks for the same few
// maps token after token: each host thread keeps the last ones it encoded (the driver call costs about as much as the
// launch).
struct MapKey {
  const void* base;
  long long a, b, c;       // the sizes the map is made from
  bool operator==(const MapKey& o) const { return base == o.base && a == o.a && b == o.b && c == o.c; }
};
template <typename Encode>
bool kept_map(CUtensorMap* map, const MapKey& key, const Encode& encode) {
  struct Kept { MapKey key{}; CUtensorMap map; };
  constexpr int kKept = 128;
  static thread_local Kept kept[kKept];
  const uintptr_t mixed = reinterpret_cast<uintptr_t>(key.base) >> 8;
  Kept& slot = kept[(mixed ^ (mixed >> 7) ^ (uintptr_t)key.a ^ (uintptr_t)(key.b * 5) ^ (uintptr_t)(key.c >> 4) ^ (uintptr_t)(key.c >> 12)) % kKept];
  if (!(slot.key == key)) {
    EncodeTiled fn = encode_tiled();
    if (!fn || encode(fn, &slot.map) != CUDA_SUCCESS) {
      slot.key = MapKey{};
      return false;
    }
    slot.key = key;
  }
  *map = slot.map;
  return true;
}
// `rows` rows of `row_bytes` bytes (a multiple of 16) as 8-byte elements, box = box_rows rows x box_bytes.
bool encode_rows(CUtensorMap* map, const void* base, int rows, int row_bytes, int box_rows, int box_bytes) {
  return kept_map(map, MapKey{base, rows, row_bytes, box_rows * 4096 + box_bytes}, [&](EncodeTiled fn, CUtensorMap* out) {
    const cuuint64_t dims[2] = {(cuuint64_t)(row_bytes / 8), (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)(box_bytes / 8), (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}
// The activations [M][K] (16-bit elements, rows ldx apart, of K the whole multiples of 64) as [K / 64][M][64], box = `blocks` of them.
bool encode_activations(CUtensorMap* map, const void* base, int M, int K, int ldx, int blocks, bool swizzled) {
  K &= ~63;
  const int row = M > 1 ? ldx : K;     // (one row may come with any distance to a next one)
  return kept_map(map, MapKey{base, ((long long)M << 32) | K, row, swizzled ? -blocks : -blocks - 4096}, [&](EncodeTiled fn, CUtensorMap* out) {
    const cuuint64_t dims[3] = {64, (cuuint64_t)M, (cuuint64_t)(K / 64)};
    const cuuint64_t strides[2] = {(cuuint64_t)row * 2, 128};
    const cuuint32_t box[3] = {64, (cuuint32_t)M, (cuuint32_t)blocks};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}
DeviceState g_devices[kMaxDevices];
std::atomic<int> g_static_weights{0};   // dg_set_static_weights
std::atomic<unsigned long long> g_wait_limit_ns{dg::kWaitLimitNs};   // dg_set_wait_limit_ns
// dg_set_trace: launch i of the GEMV kernels (counted from the call that set the buffer) stamps into region i
std::atomic<unsigned long long*> g_trace_base{nullptr};
std::atomic<int> g_trace_capacity{0}, g_trace_next{0};

const void* const (*const kTables[])[16] = {dg_table_bf16,       dg_table_fp8_bf16,   dg_table_fp8_f16,  dg_table_mxfp8_bf16,
                                      dg_table_mxfp8_f16,  dg_table_nvfp4_bf16, dg_table_nvfp4_f16};

// Per device, once: SM count, the address of the status word, and the opt-in to 227 KB of dynamic shared memory for
// every kernel. None of this is a stream operation. Returns nullptr when the device cannot run sm_100a code.
DeviceState* device_state() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  DeviceState& st = g_devices[dev];
  int ready = st.ready.load(std::memory_order_acquire);
  if (ready == 1) return &st;
  if (ready == -1) return nullptr;
  int major = 0, sms = 0;
  void* status = nullptr;
  bool ok = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) == cudaSuccess && major == 10 &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0 &&
            cudaGetSymbolAddress(&status, dg_status_word) == cudaSuccess;
  // (the whole of an SM's 228 KB as shared memory: two small blocks, or one, and no change between launches)
  auto opt_in = [&](const void* const (*table)[16], int rows) {
    const void* done = nullptr;    // (a table's neighbours share their kernel)
    for (int i = 0; ok && i < 16 * rows; ++i) {
      if (table[i / 16][i % 16] == done) continue;
      done = table[i / 16][i % 16];
      ok = cudaFuncSetAttribute(done, cudaFuncAttributeMaxDynamicSharedMemorySize, dg::kSmemLimit) ==
               cudaSuccess &&
           cudaFuncSetAttribute(done, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared) == cudaSuccess;
    }
  };
  for (const void* const (*table)[16] : kTables) opt_in(table, 4);
  opt_in(dg_batch_table_nvfp4_bf16, 2);
  if (!ok) {
    cudaGetLastError();
    st.ready.store(-1, std::memory_order_release);
    return nullptr;
  }
  st.sms = sms;
  st.status = static_cast<int*>(status);
  st.ready.store(1, std::memory_order_release);
  return &st;
}

struct FormatInfo {
  int e, step, x_row;   // elements per 16-byte block, bytes of a step of a weight row and of an activation row
};
template <int FMT>
constexpr FormatInfo info_of() { return {dg::Format<FMT>::E, dg::Format<FMT>::STEP, dg::Format<FMT>::XROW}; }
constexpr FormatInfo kFormats[4] = {info_of<0>(), info_of<1>(), info_of<2>(), info_of<3>()};

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Bytes kept behind the ring for resident activations: whole steps of [M][x_row bytes], and a byte per step, in sixteens, which
// nothing uses (the exponents lie in static shared memory); it stays in the plans that callers know.
int resident_bytes_of(int fmt, int M, int nblk) {
  const int row_steps = ceil_div(nblk * 16, kFormats[fmt].step);
  return row_steps * M * kFormats[fmt].x_row + ((row_steps + 15) & ~15);
}

// How row-major block scales reach a stage: by tensor copy when every window of every row starts on 16 bytes and is a multiple of 16
// bytes long (K a multiple of 256, MXFP8 512; base on 16 bytes), else two warps copy them.
int row_major_scales(int fmt, int K, bool on_16_bytes) {
  if (fmt != dg::FMT_NVFP4 && fmt != dg::FMT_MXFP8) return dg::SCALES_NONE;
  return K % (fmt == dg::FMT_NVFP4 ? 256 : 512) == 0 && on_16_bytes ? dg::SCALES_STAGED : dg::SCALES_DIRECT;
}

// Launch shape: a speed choice from (format, M, N, K, SM count, how scales travel, SwiGLU) only; no row's bits depend on it.
//   CTAs            one per SM, fewer when the matrix has under four rows per SM
//   tile rows       64 to 40 (less when a CTA's range is shorter): what takes the fewest eighths of 8 rows, a tile costing as much
//                   as one eighth (its sums) plus, where its activations are converted on the way, as much as these cost
//                   (57344 x 8192 NVFP4 in tiles of 56 and of 64 rows, both seven: 8 rows 64.8 and 63.8 us, 16 rows 93.3 and 91)
//   steps           512-byte steps per ring stage (BF16: one of 1 KB): two, one where the ring would have fewer than three
//                   stages otherwise: a consumer warp's fixed costs per stage then weigh half. A CTA's whole range in one tile
//                   is worth more than two steps (8192 x 8192 NVFP4, 2 / 3 / 4 rows, 56 matrix rows per CTA: tiles of 40 and 16
//                   in two steps 12.65 / 14.35 / 14.9 us, one tile in one step 11.7 / 12.45 / 13.15; FP8 with 4 rows 17.3 and
//                   14.8), and from 16 steps of K on two steps are worth more than a third stage where the ring does not have
//                   to hold a finished tile's sums as well (8192 x 28672 NVFP4, 4 rows: three stages of 40 rows 41.8, two of 56
//                   31.2). NVFP4 from five rows on: one, but for the shortest ranges. Its windows of activations leave two steps
//                   only low tiles (57344 x 8192, 5 rows 66.4 and 61.6 us; gate_up with SwiGLU had tiles of 16 columns), and a layer's
//                   projections are one kernel then: three layers at 8 rows take 374 us with two steps for K = 28672, 366 without
//                   (31.1 and 32.1 alone), with SwiGLU in gate_up 419 and 371.5
//   stages          as many as fit in shared memory, at most kMaxStages
// Activations stay resident (FP8, NVFP4, up to four rows) where that leaves three stages of two steps, or four of one (from three rows on,
// where they would take a fifth and more of a stage, and where a CTA's range is one tile in stages of one step only); otherwise, and
// where a CTA's range is short (below), a window of them passes through every stage.
// `grid` > 0: the launch is a batch's (that many CTAs whatever N; the caller sizes the ring for all its GEMVs and
// decides about resident activations: `allow_resident` is its wish, and no rule about stages is applied here).
bool make_plan(int fmt, int M, int N, int K, int sms, Params& p, int& ctas, int& smem, int grid = 0,
               bool allow_resident = true) {
  const FormatInfo f = kFormats[fmt];
  const long long row_bits = (long long)K * 128 / f.e;   // 16 bytes per e elements
  p.row_bytes = (int)(row_bits / 8);
  p.nblk = p.row_bytes / 16;
  p.M = M;
  const int regions = p.pairs ? 2 : 1;    // N counts columns; gate_up matrices have two rows to a column
  ctas = grid > 0 ? grid : sms < ceil_div(N, 4) ? sms : ceil_div(N, 4);   // grid: the launch is shared (batch)
  const int cols_per_cta = ceil_div(N, ctas), all_rows = regions * ceil_div(cols_per_cta, dg::kBoxRows) * dg::kBoxRows;
  p.cols_each = N / ctas;
  p.cols_more = N % ctas;
  const int row_steps = ceil_div(p.row_bytes, f.step);
  // Tuning aid: DG_FORCE_PLAN="rows,steps" fixes the rows of a tile and the steps of a stage (read once).
  static const char* forced = std::getenv("DG_FORCE_PLAN");
  int force_rows = 0, force_steps = 0;
  if (forced) std::sscanf(forced, "%d,%d", &force_rows, &force_steps);
  const int resident_bytes = resident_bytes_of(fmt, M, p.nblk);
  // (a batch shares one ring and one resident area between GEMVs of different K: only the smaller ones stay resident)
  // (one row's activations are a thirtieth of a stage: not worth a lower tile)
  const int room = dg::kSmemLimit - dg::kSmemHeader;
  // Where a CTA's range is short, bringing and converting all activations before its first product takes longer than windows (us
  // resident and in windows: NVFP4 600 x 8192 with 4 rows 7.7 and 6.4, 3 rows 7.1 and 6.2, 2 rows 6.2 and 6.1, one 5.35 and 6.1; 4096 x 8192, 28
  // matrix rows per CTA, 4 rows 9.8 and 8.65, one 7.8 and 8.4; 1152 x 2048 with 1 / 4 rows 3.55 / 3.9 and 3.3 / 3.4; FP8 4096 x 4096 with
  // 3 / 4 rows 6.4 / 6.5 and 6.3 / 6.3, 2368 x 8192 with 4 rows 8.1 and 8.5).
  const bool short_range = grid == 0 && ((all_rows <= 48 && M >= 4) || (all_rows <= 32 && M == 3)) && (fmt == dg::FMT_NVFP4 || row_steps <= 8);
  const bool shortest = grid == 0 && fmt == dg::FMT_NVFP4 && all_rows * row_steps <= 32;
  const bool may_reside = !short_range && !shortest && allow_resident && dg::resident_capable(fmt, M) && K % 64 == 0 &&
                          resident_bytes <= (grid > 0 ? dg::kResidentLimit / 2 - 15 * 1024 : dg::kResidentLimit) &&
                          (M > 1 || 3 * 56 * (dg::weight_pitch(fmt, 2) + dg::scale_pitch(fmt, 2)) + resident_bytes <= room);
  int best_cost = 0, best_merit = 0;
  p.tile_rows = 0;
  // whether stages of the range's only tile fit, `need` of them
  auto one_tile_fits = [&](bool resident, int steps, int need) {
    if (all_rows > 64 || grid > 0 || force_steps > 0 || p.pairs) return false;
    int bytes = all_rows * (dg::weight_pitch(fmt, steps) + dg::scale_pitch(fmt, steps));
    if (!resident) bytes = (dg::x_offset(bytes) + steps * M * f.x_row + 1023) & ~1023;
    return need * ((bytes + 127) & ~127) <= room - (resident ? resident_bytes : 0);
  };
  // resident with two steps, with one, not resident with two, with one: the first that has the stages it asks for
  for (int attempt = may_reside ? 0 : 2; attempt < 4 && p.tile_rows == 0; ++attempt) {
    const bool resident = attempt < 2;
    const int steps = fmt == dg::FMT_BF16 ? 1 : 2 - attempt % 2;
    // (a batch's GEMVs share one instance: the same steps for all, whatever their K)
    if (grid > 0 ? steps != (M <= 4 ? 2 : 1) : force_steps > 0 ? steps != std::min(force_steps, row_steps)
                                                               : steps == 2 && row_steps == 1 && fmt != dg::FMT_BF16) continue;
    int need = grid > 0 || force_steps > 0 ? 2 : attempt == 0 ? 3 : attempt == 1 ? (M >= 3 ? 4 : dg::kMaxStages + 1)
                                               : attempt == 2 ? 3 : 2;
    if (grid == 0 && force_steps == 0 && fmt == dg::FMT_NVFP4 && M >= 5 && steps == 2 && all_rows > 32) continue;
    // (from 13 rows on the windows of FP8 leave three stages of two steps 40 rows only: us with 16 rows so and in one step, 12288 x 5120 22.8 and
    // 18.3, 28672 x 8192 56.5 and 54.8, 20000 x 2048 14.2 and 13.2; with 12 rows 12288 x 5120 17.3 and 18.0; one tile, 8192 x 8192, 16.1 and 16.8)
    if (grid == 0 && force_steps == 0 && fmt == dg::FMT_FP8 && M >= 13 && steps == 2 && all_rows > 64) continue;
    const bool one_step_tile = fmt != dg::FMT_BF16 && one_tile_fits(resident, 1, resident ? 4 : 3);
    if (steps == 2 && fmt != dg::FMT_BF16 && row_steps > 1 && !one_tile_fits(resident, 2, 3)) {
      if (!resident && row_steps >= 16 && one_tile_fits(false, 2, 2)) need = 2;
      else if (one_step_tile) continue;
    }
    if (attempt == 1 && one_step_tile) need = 4;
    const int convert = resident || fmt == dg::FMT_BF16 ? 0 : M <= 8 ? 5 : 7;   // of a tile, in halves of a group
    for (int rows = 64; rows >= 40; rows -= 8) {
      int tile_rows = std::min(force_rows >= 16 && force_rows <= 64 ? force_rows & ~7 : rows, all_rows);
      if (p.pairs) tile_rows &= ~15;                            // the same for both regions
      int stage_bytes = tile_rows * (dg::weight_pitch(fmt, steps) + dg::scale_pitch(fmt, steps));
      if (!resident) stage_bytes = dg::x_offset(stage_bytes) + steps * M * f.x_row;
      const int unit = resident ? 128 : 1024;
      stage_bytes = (stage_bytes + unit - 1) / unit * unit;
      const int stages = std::min((room - (resident ? resident_bytes : 0)) / stage_bytes, dg::kMaxStages);
      if (stages < need) continue;
      const int cap = tile_rows / regions, tiles = ceil_div(cols_per_cta, cap), rem = cols_per_cta - (tiles - 1) * cap;
      const int eights = (tiles - 1) * tile_rows / 8 + ceil_div((regions - 1) * cap + rem, 8);
      // of equals the one with the fewest tiles of an odd number of eighths where NVFP4's activations come in windows (their last
      // group's products are made whole), then the one whose last tile is the fullest: a window of a few rows takes as long as its latency
      const int odd = resident || fmt != dg::FMT_NVFP4 ? 0 : (tiles - 1) * (tile_rows / 8 & 1) + (ceil_div((regions - 1) * cap + rem, 8) & 1);
      const int merit = 64 * (64 - std::min(odd, 63)) + rem;
      const int cost = eights + (1 + convert) * tiles;
      if (p.tile_rows == 0 || cost < best_cost || (cost == best_cost && merit > best_merit)) {
        best_cost = cost;
        best_merit = merit;
        p.tile_rows = tile_rows;
        p.last_rows = ceil_div(rem, dg::kBoxRows) * dg::kBoxRows;
        p.steps = steps;
        p.stage_bytes = stage_bytes;
        p.stages = stages;
        p.x_mode = resident ? dg::X_RESIDENT : K % 64 == 0 ? dg::X_TENSOR : dg::X_COPIED;
      }
    }
  }
  if (p.tile_rows == 0) return false;
  // Small launches: a stage for every window, in half of the shared memory, so that the next launch's CTA fits beside.
  if (grid == 0 && dg::small_capable(M) && all_rows <= dg::kSmallRows &&
      (fmt != dg::FMT_NVFP4 || (row_steps <= 2 && all_rows * row_steps <= dg::kSmallNvfp4 && !p.pairs)) && K % 64 == 0 && p.scale_mode != dg::SCALES_DIRECT &&
      p.scale_mode != dg::SCALES_BLOCKED && force_steps == 0) {
    const int steps = fmt == dg::FMT_BF16 || row_steps == 1 ? 1 : 2, windows = std::max(2, ceil_div(row_steps, steps));
    const int rows = regions * ceil_div(all_rows / regions, dg::kBoxRows) * dg::kBoxRows;
    const bool resident = may_reside;
    int stage_bytes = rows * (dg::weight_pitch(fmt, steps) + dg::scale_pitch(fmt, steps));
    if (!resident) stage_bytes = (dg::x_offset(stage_bytes) + steps * M * f.x_row + 1023) / 1024 * 1024;
    stage_bytes = (stage_bytes + 127) / 128 * 128;
    if (windows <= dg::kMaxStages &&
        dg::kSmemHeader + windows * stage_bytes + (resident ? resident_bytes : 0) <= dg::kSmallSmem) {
      p.small = 1;
      p.tile_rows = rows;
      p.last_rows = rows / regions;
      p.steps = steps;
      p.stage_bytes = stage_bytes;
      p.stages = windows;
      p.x_mode = resident ? dg::X_RESIDENT : dg::X_TENSOR;
    }
  }
  p.x_res_off = dg::kSmemHeader + p.stages * p.stage_bytes;
  smem = p.x_res_off + (p.x_mode == dg::X_RESIDENT ? resident_bytes : 0);
  return true;
}

bool aligned(const void* ptr, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(ptr) % bytes == 0; }

// From this many bytes on a launch's weights and scales leave L2 first, NVFP4's always. In the usual order they drive out what the next
// launches need, the kernels' code above all: a launch of another kernel than the one before took 1.4 to 4.2 us longer than one of
// the same, with them first 0.7 to 1.9. But a few smaller matrices used in turn stay in L2, and leave it too early so.
// us in the usual order and leaving first, three matrices in turn, eager / so many that they exceed L2, in a graph: BF16 3072 x 3072, one
// row 5.0 / 5.93 and 6.0 / 5.92; FP8 4096 x 4096 4.9 / 5.55 and 5.3 / 5.3, 5120 x 4096 5.65 / 6.1 and 6.05 / 5.95, 4096 x 8192 8.3 / 8.6 and
// 8.1 / 8.45, 28672 x 8192 40.4 and 38.4; MXFP8 5120 x 5120, two rows 8.04 / 8.11 and 8.44 / 8.07; BF16 4096 x 4096 8.13 / 8.29 and 8.08 /
// 8.14, 8192 x 8192 23.0 and 21.9. NVFP4, which its consumers bound: 4096 x 4096 5.24 / 5.74 and 5.25 / 5.50, 8192 x 4096 7.16 / 7.74 and
// 7.34 / 7.46, 10240 x 8192 14.05 / 13.7 and 13.3 / 13.0, four layers of four projections 488 and 464.
constexpr long long kStreamed = 32ll << 20;
long long weight_bytes(const Params& p) {
  return (long long)(p.pairs ? 2 * p.pairs : p.N) * (p.row_bytes + (p.scale_mode == dg::SCALES_NONE ? 0 : p.scale_row_bytes));
}

// Everything of a launch but the launch: plan, tensor maps, process-wide settings. `grid` > 0 fixes the CTA count.
int prepare(int fmt, Params& p, int M, int& ctas, int& smem, int grid = 0, bool allow_resident = true) {
  DeviceState* st = device_state();
  if (!st) return (int)cudaErrorInvalidDevice;
  if (!make_plan(fmt, M, p.N, p.K, st->sms, p, ctas, smem, grid, allow_resident)) return (int)cudaErrorInvalidValue;
  p.status = st->status;
  // Tensor maps for the copies of whole boxes and of the activations' windows.
  const int matrix_rows = p.pairs ? 2 * p.pairs : p.N;
  const int full_rows = p.tile_rows / (p.pairs ? 2 : 1), w_box = dg::weight_pitch(fmt, p.steps), sc_box = dg::scale_pitch(fmt, p.steps);
  if (!encode_rows(&p.tmap_w, p.w, matrix_rows, p.row_bytes, full_rows, w_box) ||
      !encode_rows(&p.tmap_w_last, p.w, matrix_rows, p.row_bytes, p.last_rows, w_box) ||
      (p.scale_mode == dg::SCALES_STAGED &&
       (!encode_rows(&p.tmap_sc, p.scales, matrix_rows, p.scale_row_bytes, full_rows, sc_box) ||
        !encode_rows(&p.tmap_sc_last, p.scales, matrix_rows, p.scale_row_bytes, p.last_rows, sc_box))))
    return (int)cudaErrorNotSupported;
  const int step_blocks = kFormats[fmt].x_row / 128;
  if (p.x_mode == dg::X_COPIED) {
    // (rows of any distance, none at all among them, may come to the copying warps)
    p.x_box_steps = p.K / 64 >= p.steps * step_blocks && (M == 1 || p.ldx > 0) &&
                    encode_activations(&p.tmap_x, p.x, M, p.K, p.ldx, p.steps * step_blocks, true) ? p.steps : 0;
  } else {
    const int steps = ceil_div(p.row_bytes, kFormats[fmt].step);
    p.x_box_steps = std::min(steps, 256 / step_blocks);           // whole boxes only: the space ends with the last step
    while (steps % p.x_box_steps) --p.x_box_steps;
    const bool resident = p.x_mode == dg::X_RESIDENT;
    if (!encode_activations(&p.tmap_x, p.x, M, p.K, p.ldx, (resident ? p.x_box_steps : p.steps) * step_blocks, !resident))
      return (int)cudaErrorNotSupported;
  }
  p.streamed = fmt == dg::FMT_NVFP4 || weight_bytes(p) >= kStreamed;
  p.early_weights = g_static_weights.load(std::memory_order_relaxed);
  p.wait_limit_ns = g_wait_limit_ns.load(std::memory_order_relaxed);
  return 0;
}

// Programmatic dependent launch: the kernel may start while the previous kernel of the stream drains (its launch,
// barrier set-up and, with static weights, its first weight copies overlap that tail); it waits for the previous
// kernel before it reads activations or scales from global memory and before it writes.
int launch_pdl(const void* kernel, void** args, int ctas, int threads, int smem, cudaStream_t stream) {
  static const bool no_pdl = std::getenv("DG_NO_PDL") != nullptr;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(ctas);
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = (size_t)smem;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = no_pdl ? 0 : 1;
  const cudaError_t e = cudaLaunchKernelExC(&config, kernel, args);
  return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

int launch(int table, int fmt, Params& p, int M, cudaStream_t stream) {
  int ctas = 0, smem = 0;
  if (const int code = prepare(fmt, p, M, ctas, smem)) return code;
  if (unsigned long long* base = g_trace_base.load(std::memory_order_acquire)) {
    const int index = g_trace_next.fetch_add(1, std::memory_order_relaxed);
    if (index < g_trace_capacity.load(std::memory_order_relaxed))
      p.trace = base + (size_t)index * DG_TRACE_CTAS * dg::kTraceSlots;
  }
  void* args[] = {&p};
  // Up to four rows whose activations come in windows run the kernel for five to eight, the bits being the same: its code for such
  // windows is the better one (NVFP4 8192 x 28672, one row 32.5 us in the kernel for up to four and 30.5 in this one, 12490 x 5088 with one /
  // four rows 13.5 / 14.1 and 12.7 / 13.4, 20000 x 1056 10.8 / 11.2 and 9.7 / 10.1; FP8 20000 x 9200 35.3 / 35.6 and 34.1 / 34.4).
  const bool windows = p.x_mode != dg::X_RESIDENT;
  const int rows = windows ? std::max(M, 5) : M;
  return launch_pdl(kTables[table][p.steps - 1 + 2 * p.small][rows - 1], args, ctas, p.small ? dg::kSmallThreads : dg::kThreads, smem,
                    stream);
}

// Argument rules of the NVFP4 GEMV (dg_enqueue_nvfp4) and the fields they determine.
bool fill_nvfp4(Params& p, const void* x, int ldx, int x_is_bf16, const uint8_t* codes, const uint8_t* scales, int blocked,
                const float* inverse, int out_kind, int M, int N, int K) {
  if (M < 1 || M > DG_MAX_ROWS || N < 1 || K < 32 || K % 32) return false;
  if (!x || !codes || !scales || !inverse || ldx % 8 || !aligned(x, 16) || !aligned(codes, 16) || !aligned(scales, 2) ||
      !aligned(inverse, 4) || (out_kind != 0 && out_kind != 1))
    return false;
  p.x = x; p.ldx = ldx; p.w = codes; p.scales = scales; p.row_scale = inverse;
  p.out_kind = out_kind == 0 ? dg::OUT_F32 : (x_is_bf16 ? dg::OUT_BF16 : dg::OUT_F16);
  p.N = N; p.K = K;
  p.scale_row_bytes = K / 16;
  p.ct = blocked ? (K / 16 + 3) / 4 : 0;
  p.scale_mode = blocked ? dg::SCALES_BLOCKED : row_major_scales(dg::FMT_NVFP4, K, aligned(scales, 16));
  return true;
}

// Head of an encoded batch (dg_encode_nvfp4_batch); the GEMVs' launch parameters follow at kBatchHead bytes.
constexpr unsigned int kBatchMagic = 0x44474232u;   // "DGB2": goes up with the layout of Params
constexpr size_t kBatchHead = 256;
struct BatchHead {
  unsigned int magic;
  int count, M, steps, ctas, smem, threads, device;
  const void* device_blob;
};
static_assert(sizeof(BatchHead) <= kBatchHead && kBatchHead % alignof(Params) == 0, "batch head layout");

}  // namespace

extern "C" {

int dg_enqueue_nvfp4(const void* x, int ldx, int x_is_bf16, const uint8_t* codes, const uint8_t* scales, int blocked,
                     const float* inverse, void* out, int ldo, int out_kind, int M, int N, int K, void* stream) {
  Params p{};
  if (!out || !fill_nvfp4(p, x, ldx, x_is_bf16, codes, scales, blocked, inverse, out_kind, M, N, K))
    return (int)cudaErrorInvalidValue;
  p.out = out; p.ldo = ldo;
  return launch(x_is_bf16 ? 5 : 6, dg::FMT_NVFP4, p, M, static_cast<cudaStream_t>(stream));
}

int dg_enqueue_nvfp4_allgather(const void* x, int ldx, int x_is_bf16, const uint8_t* codes, const uint8_t* scales,
                               int blocked, const float* inverse, void* const* peer_out, void* const* peer_flags,
                               int world, int rank, int slot, int out_kind, int M, int N, int K, void* stream) {
  Params p{};
  if (!peer_out || !peer_flags || world < 1 || world > dg::kMaxRanks || rank < 0 || rank >= world || slot < 0 ||
      slot > 3 || !fill_nvfp4(p, x, ldx, x_is_bf16, codes, scales, blocked, inverse, out_kind, M, N, K))
    return (int)cudaErrorInvalidValue;
  p.ldo = N;
  p.world = world; p.rank = rank; p.gather_slot = slot & 1; p.gather_nowait = slot >> 1;
  for (int q = 0; q < world; ++q) {
    if (!peer_out[q] || !peer_flags[q] || !aligned(peer_flags[q], 4)) return (int)cudaErrorInvalidValue;
    p.peer_out[q] = peer_out[q];
    p.peer_flag[q] = static_cast<unsigned int*>(peer_flags[q]);
  }
  p.out = peer_out[rank];
  return launch(x_is_bf16 ? 5 : 6, dg::FMT_NVFP4, p, M, static_cast<cudaStream_t>(stream));
}

// Waits (bounded) until counter `slot` of this rank's block holds `expected` arrivals, then takes them off.
__global__ void gather_wait_kernel(unsigned int* counter, unsigned int expected, int* status,
                                   unsigned long long limit_ns) {
  const unsigned long long start = dg::global_ns();
  bool done = false;
  for (unsigned int i = 1; !done; ++i) {
    unsigned int seen;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
    done = seen >= expected;
    if (!done && (i & 63u) == 0u && dg::global_ns() - start > limit_ns) break;
  }
  if (done) atomicSub_system(counter, expected);
  else if (status) atomicOr(status, dg::kStatusGatherTimeout);
  __threadfence_system();
}

int dg_enqueue_gather_wait(void* flags, int slot, unsigned int expected, void* stream) {
  DeviceState* st = device_state();
  if (!st) return (int)cudaErrorInvalidDevice;
  if (!flags || !aligned(flags, 4) || (slot != 0 && slot != 1) || expected == 0) return (int)cudaErrorInvalidValue;
  gather_wait_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<unsigned int*>(flags) + slot, expected,
                                                                    st->status,
                                                                    g_wait_limit_ns.load(std::memory_order_relaxed));
  return (int)cudaGetLastError();
}

int dg_reset_counters(void* flags, void* stream) {
  if (!flags || !aligned(flags, 4)) return (int)cudaErrorInvalidValue;
  return (int)cudaMemsetAsync(flags, 0, 4 * sizeof(unsigned int), static_cast<cudaStream_t>(stream));
}

// ---- the entry point that allocates nothing ---------------------------------------------------------------------
// Arrival counters for dg_enqueue_nvfp4_allgather_noalloc: DG_NOALLOC_CHANNELS blocks of four 32-bit counters that live
// in the library's image on every GPU that loads it (1 KB per GPU, held until the process exits), zero when the
// module is loaded and re-armed to zero by every call that completes. In host code `dg_gather_scratch` is only a
// handle for the runtime, not a device address: the address a kernel may use comes from cudaGetSymbolAddress, asked
// once per device with that device current.
static __device__ __align__(256) unsigned int dg_gather_scratch[4 * DG_NOALLOC_CHANNELS];
static std::atomic<unsigned int*> g_gather_scratch[kMaxDevices];   // per device, filled by the first call that names it

static cudaError_t gather_scratch_of(int device, unsigned int** out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  if (!g_gather_scratch[device].load(std::memory_order_acquire)) {
    int previous = 0;
    cudaError_t e = cudaGetDevice(&previous);
    if (e == cudaSuccess && previous != device) e = cudaSetDevice(device);
    void* address = nullptr;
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&address, dg_gather_scratch);
    if (previous != device) {
      const cudaError_t back = cudaSetDevice(previous);
      if (e == cudaSuccess) e = back;
    }
    if (e != cudaSuccess) return e;
    g_gather_scratch[device].store(static_cast<unsigned int*>(address), std::memory_order_release);
  }
  *out = g_gather_scratch[device].load(std::memory_order_acquire);
  return cudaSuccess;
}

int dg_enqueue_nvfp4_allgather_noalloc(const void* x, int ldx, int x_is_bf16, const uint8_t* codes,
                                       const uint8_t* scales, int blocked, const float* inverse,
                                       void* const* peer_out, const int* devices, int world, int rank, int channel,
                                       int slot, int out_kind, int M, int N, int K, void* stream) {
  if (!devices || world < 1 || world > dg::kMaxRanks || channel < 0 || channel >= DG_NOALLOC_CHANNELS)
    return (int)cudaErrorInvalidValue;   // more ranks or channels than the built-in counters cover
  // Only the waiting forms: a signal-only call (slot 2, 3) would leave arrivals on counters that no caller can
  // reach to collect, and the channel's next waiting call would then end before its data has landed.
  if (slot != 0 && slot != 1) return (int)cudaErrorInvalidValue;
  int current = -1;
  if (rank < 0 || rank >= world || cudaGetDevice(&current) != cudaSuccess || current != devices[rank])
    return (int)cudaErrorInvalidValue;   // the kernel counts its CTAs on the current device's block
  void* flags[dg::kMaxRanks];
  for (int q = 0; q < world; ++q) {
    unsigned int* base = nullptr;
    const cudaError_t e = gather_scratch_of(devices[q], &base);
    if (e != cudaSuccess) return (int)e;
    flags[q] = base + 4 * channel;
  }
  return dg_enqueue_nvfp4_allgather(x, ldx, x_is_bf16, codes, scales, blocked, inverse, peer_out, flags, world, rank,
                                    slot, out_kind, M, N, K, stream);
}

int dg_enqueue_nvfp4_gate_up_swiglu(const void* x, int ldx, int x_is_bf16, const uint8_t* codes, const uint8_t* scales,
                                    int blocked, const float* inverse, void* out, int ldo, int out_kind, int M, int I,
                                    int K, void* stream) {
  Params p{};
  if (!out || I < 1 || I > (1 << 29) ||
      !fill_nvfp4(p, x, ldx, x_is_bf16, codes, scales, blocked, inverse, out_kind, M, 2 * I, K))
    return (int)cudaErrorInvalidValue;
  p.out = out; p.ldo = ldo;
  p.pairs = I;
  p.N = I;                 // (output columns)
  return launch(x_is_bf16 ? 5 : 6, dg::FMT_NVFP4, p, M, static_cast<cudaStream_t>(stream));
}

unsigned long long dg_batch_blob_bytes(int count) { return count > 0 ? kBatchHead + (size_t)count * sizeof(Params) : 0; }

int dg_encode_nvfp4_batch(const DgNvfp4BatchItem* items, int count, int x_is_bf16, int out_kind, int M, int world, int rank,
                          void* const* peer_flags, int slot, const void* device_blob, void* host_blob) {
  if (!items || count < 1 || !device_blob || !host_blob || !aligned(device_blob, 256) || !aligned(host_blob, 8) ||
      !x_is_bf16 || world < 0 || world > dg::kMaxRanks || (world > 0 && (rank < 0 || rank >= world || !peer_flags)) ||
      slot < 0 || slot > 3)
    return (int)cudaErrorInvalidValue;
  DeviceState* st = device_state();
  if (!st) return (int)cudaErrorInvalidDevice;
  BatchHead head{};
  Params* out = reinterpret_cast<Params*>(static_cast<unsigned char*>(host_blob) + kBatchHead);
  int stage_bytes = 0, resident_bytes = 0, stages = 0;
  // One ring for all: the largest stage any GEMV needs, as many of them as fit. Behind the ring: room for the largest
  // resident activations (every GEMV brings its own when its turn comes). If the resident ones cost the ring its third
  // stage, once more without them.
  for (int attempt = 0; attempt < 2; ++attempt) {
    stage_bytes = 0; resident_bytes = 0;
    for (int g = 0; g < count; ++g) {
      const DgNvfp4BatchItem& it = items[g];
      Params p{};
      if (!fill_nvfp4(p, it.x, it.ldx, x_is_bf16, it.codes, it.scales, it.blocked, it.inverse, out_kind, M, it.N, it.K))
        return (int)cudaErrorInvalidValue;
      if (world > 0) {
        if (!it.peer_out) return (int)cudaErrorInvalidValue;
        p.ldo = it.N;
        p.world = world; p.rank = rank; p.gather_slot = slot & 1; p.gather_nowait = slot >> 1;
        for (int q = 0; q < world; ++q) {
          if (!it.peer_out[q] || !peer_flags[q] || !aligned(peer_flags[q], 4)) return (int)cudaErrorInvalidValue;
          p.peer_out[q] = it.peer_out[q];
          p.peer_flag[q] = static_cast<unsigned int*>(peer_flags[q]);
        }
        p.out = it.peer_out[rank];
      } else {
        if (!it.out) return (int)cudaErrorInvalidValue;
        p.out = it.out; p.ldo = it.ldo;
      }
      int ctas = 0, smem = 0;
      // one grid for all: a CTA per SM, whatever a GEMV's size (a CTA without rows of a GEMV passes it by)
      if (const int code = prepare(dg::FMT_NVFP4, p, M, ctas, smem, st->sms,
                                   attempt == 0))
        return code;
      stage_bytes = std::max(stage_bytes, (p.stage_bytes + 1023) & ~1023);   // (where stages hold activations)
      if (p.x_mode == dg::X_RESIDENT) resident_bytes = std::max(resident_bytes, resident_bytes_of(dg::FMT_NVFP4, M, p.nblk));
      out[g] = p;
    }
    stages = (dg::kSmemLimit - dg::kSmemHeader - resident_bytes) / stage_bytes;
    if (stages > dg::kMaxStages) stages = dg::kMaxStages;
    if (resident_bytes == 0 || stages >= 3) break;
  }
  if (stages < 2) return (int)cudaErrorInvalidValue;
  for (int g = 0; g < count; ++g) {
    out[0].batch_copies |= out[g].x_mode == dg::X_COPIED || out[g].scale_mode != dg::SCALES_STAGED;
    out[g].stage_bytes = stage_bytes;
    out[g].stages = stages;
    out[g].x_res_off = dg::kSmemHeader + stages * stage_bytes;
  }
  head.magic = kBatchMagic; head.count = count; head.M = M; head.steps = out[0].steps; head.ctas = st->sms;
  head.smem = dg::kSmemHeader + stages * stage_bytes + resident_bytes;
  head.threads = dg::kThreads;
  head.device_blob = device_blob;
  cudaGetDevice(&head.device);
  *reinterpret_cast<BatchHead*>(host_blob) = head;
  return 0;
}

int dg_enqueue_batch(const void* host_blob, void* stream) {
  if (!host_blob) return (int)cudaErrorInvalidValue;
  const BatchHead head = *reinterpret_cast<const BatchHead*>(host_blob);
  int device = -1;
  if (head.magic != kBatchMagic || head.count < 1 || head.M < 1 || head.M > DG_MAX_ROWS || head.steps < 1 ||
      head.steps > 2 ||
      cudaGetDevice(&device) != cudaSuccess || device != head.device)
    return (int)cudaErrorInvalidValue;
  if (!device_state()) return (int)cudaErrorInvalidDevice;
  const Params* items = reinterpret_cast<const Params*>(static_cast<const unsigned char*>(head.device_blob) + kBatchHead);
  int count = head.count;
  void* args[] = {&items, &count};
  return launch_pdl(dg_batch_table_nvfp4_bf16[head.steps - 1][head.M - 1], args, head.ctas, head.threads, head.smem,
                    static_cast<cudaStream_t>(stream));
}

int dg_enqueue_fp8(const void* x, int ldx, int x_is_bf16, const uint8_t* codes, const float* row_scale,
                   const uint8_t* mx_scale, void* out, int ldo, int out_kind, int M, int N, int K, void* stream) {
  if (M < 1 || M > DG_MAX_ROWS || N < 1 || K < 16 || K % 16 || (mx_scale && K % 32) || (!row_scale == !mx_scale))
    return (int)cudaErrorInvalidValue;
  if (!x || !codes || !out || ldx % 8 || !aligned(x, 16) || !aligned(codes, 16) || !aligned(row_scale, 4) ||
      (out_kind != 0 && out_kind != 1))
    return (int)cudaErrorInvalidValue;
  Params p{};
  p.x = x; p.ldx = ldx; p.w = codes; p.scales = mx_scale; p.row_scale = row_scale; p.out = out; p.ldo = ldo;
  p.out_kind = out_kind == 0 ? dg::OUT_F32 : (x_is_bf16 ? dg::OUT_BF16 : dg::OUT_F16);
  p.N = N; p.K = K;
  p.scale_row_bytes = K / 32;
  const int fmt = mx_scale ? dg::FMT_MXFP8 : dg::FMT_FP8;
  p.scale_mode = row_major_scales(fmt, K, aligned(mx_scale, 16));
  return launch((mx_scale ? 3 : 1) + (x_is_bf16 ? 0 : 1), fmt, p, M, static_cast<cudaStream_t>(stream));
}

int dg_enqueue_bf16(const void* x, int ldx, const void* w, void* out, int ldo, int out_kind, int M, int N, int K,
                    void* stream) {
  if (M < 1 || M > DG_MAX_ROWS || N < 1 || K < 8 || K % 8) return (int)cudaErrorInvalidValue;
  if (!x || !w || !out || ldx % 8 || !aligned(x, 16) || !aligned(w, 16) || (out_kind != 0 && out_kind != 1))
    return (int)cudaErrorInvalidValue;
  Params p{};
  p.x = x; p.ldx = ldx; p.w = static_cast<const uint8_t*>(w); p.out = out; p.ldo = ldo;
  p.out_kind = out_kind == 0 ? dg::OUT_F32 : dg::OUT_BF16;
  p.N = N; p.K = K;
  p.scale_mode = dg::SCALES_NONE;
  return launch(0, dg::FMT_BF16, p, M, static_cast<cudaStream_t>(stream));
}

int dg_hardware_decode(void) { return device_state() ? 1 : -1; }

int dg_plan(int fmt, int M, int N, int K, int plan[6]) {
  static const int kmult[4] = {8, 16, 32, 32};
  if (fmt < 0 || fmt > 3 || M < 1 || M > DG_MAX_ROWS || N < 1 || K < kmult[fmt] || K % kmult[fmt] || !plan)
    return (int)cudaErrorInvalidValue;
  int sms = 148;
  if (DeviceState* st = device_state()) sms = st->sms;
  Params p{};
  p.N = N; p.K = K;
  p.scale_mode = row_major_scales(fmt, K, true);
  int ctas = 0, smem = 0;
  if (!make_plan(fmt, M, N, K, sms, p, ctas, smem)) return (int)cudaErrorInvalidValue;
  plan[0] = ctas; plan[1] = ceil_div(p.tile_rows, dg::kGroupRows); plan[2] = p.steps; plan[3] = p.stages; plan[4] = p.stage_bytes;
  plan[5] = smem;
  return 0;
}

int dg_take_status(void) {
  DeviceState* st = device_state();
  if (!st) return -(int)cudaErrorInvalidDevice;
  int word = 0;
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(&word, st->status, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && word) e = cudaMemset(st->status, 0, sizeof(int));
  return e == cudaSuccess ? word : -(int)e;
}

int dg_reset_noalloc_channel(int channel, void* stream) {
  if (channel < 0 || channel >= DG_NOALLOC_CHANNELS) return (int)cudaErrorInvalidValue;
  int current = 0;
  cudaError_t e = cudaGetDevice(&current);
  unsigned int* base = nullptr;
  if (e == cudaSuccess) e = gather_scratch_of(current, &base);
  if (e != cudaSuccess) return (int)e;
  return dg_reset_counters(base + 4 * channel, stream);
}

unsigned long long dg_set_wait_limit_ns(unsigned long long limit_ns) {
  return g_wait_limit_ns.exchange(limit_ns ? limit_ns : dg::kWaitLimitNs, std::memory_order_relaxed);
}

int dg_set_static_weights(int enabled) {
  return g_static_weights.exchange(enabled ? 1 : 0, std::memory_order_relaxed);
}

int dg_set_trace(void* buffer, int launches) {
  g_trace_base.store(nullptr, std::memory_order_release);
  g_trace_next.store(0, std::memory_order_relaxed);
  g_trace_capacity.store(buffer && launches > 0 ? launches : 0, std::memory_order_relaxed);
  if (buffer && launches > 0) g_trace_base.store(static_cast<unsigned long long*>(buffer), std::memory_order_release);
  return 0;
}

int dg_version(void) { return 103; }

}  // extern "C"
