// Weight-only decode GEMV for B200 (sm_100a): out[m][n] = scale[n] * sum_k x[m][k] * w[n][k] for 1..16 activation
// rows, weights stored as BF16, FP8 E4M3 (row scale), MXFP8 (E8M0 per 32) or NVFP4 (E2M1 codes, E4M3 per 16).
//
// Replaces the kernels of the reference package decode-gemv (decode_gemv_cuda/decode_gemv.cu:85 gemv_kernel,
// :191 bf16_kernel, :285 fp8_kernel). Same formats, same contract (FP32 sums whose order never depends on the row
// count), a different machine mapping:
//
//   * one persistent CTA per SM: 8 consumer warps, a warp that feeds the ring and 3 that finish tiles. The matrix rows are
//     split into one contiguous range per CTA; a range is walked in tiles of up to 64 rows and each tile in K windows.
//   * the feeding warp streams every window of a tile into a shared-memory ring, one tensor copy (TMA, mbarrier
//     complete_tx) for the weights and one for the block scales, plus the matching window of the activations. Bytes in
//     flight are set by the ring (up to ~200 KB per SM), not by registers.
//   * a 512-byte step of a row is eight chunks of 64 bytes; consumer warp w owns chunk w of every step, for all rows of
//     the tile, and multiplies it on the tensor cores (dg_mma.cuh): the activations of a chunk are then loaded and
//     converted by one warp, once per tile. At the end of a tile the eight warps' sums of every output meet in shared
//     memory (in the ring stage just consumed), where the finishing warps add them in a fixed tree; the row scale
//     multiplies once and the result is rounded once to the output type.
//
// A row's summation order is therefore a function of K and the format alone: it does not depend on M, on the rows a
// tile holds, on the tile or window sizes the launch picked, on the CTA count, or on which slice of the matrix a
// device holds.
#pragma once

#include <cuda.h>   // CUtensorMap (type only; the driver entry point is looked up at run time)
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "dg_mma.cuh"
#include "dg_swiglu.cuh"

namespace dg {

enum : int { FMT_BF16 = 0, FMT_FP8 = 1, FMT_MXFP8 = 2, FMT_NVFP4 = 3 };
enum : int { SCALES_NONE = 0, SCALES_STAGED = 1, SCALES_DIRECT = 2, SCALES_BLOCKED = 3 };
enum : int { OUT_F32 = 0, OUT_BF16 = 1, OUT_F16 = 2 };

constexpr int kMaxStages = 12;
constexpr int kConsumers = 8;              // = chunks of a step: the slices of K whose sums are added at the end
// Warps of a block: the consumers, one that feeds the ring, and three that finish tiles; in launches with something to copy
// that bulk copies cannot bring, two of these copy instead.
constexpr int kFeeder = kConsumers, kFinisher = kConsumers + 1, kFinishers = 3, kFirstCopier = kConsumers + 2, kCopyWarps = 2;
constexpr int kThreads = 32 * (kConsumers + 1 + kFinishers);
// Small launches: a CTA's whole share is one tile of at most 32 rows, brought by bulk copies alone, and fits in half of the
// SM's shared memory. Their blocks have fewer warps (the finisher only starts the activations) and fewer registers, so that
// two fit on an SM: the next launch of the stream then waits there for this one to finish, its barriers set up and its weights
// on their way into L2.
constexpr int kSmallThreads = 32 * (kConsumers + 2), kSmallRows = 32;
// NVFP4: only very short launches, of up to two steps of K and 48 matrix rows times steps in a CTA's share. Its decoding spills some of
// the 96 registers, and where calls come about as fast as a launch takes, the next launch's CTAs are placed when this one has left some
// SMs and not others; some SMs then hold two CTAs of a launch and as many hold none, and so do all launches after it, whose CTAs take
// the places that are left. us as an ordinary and as a small launch, in a graph / eager calls: 1024 x 1024, one row 3.47 / 4.92 and
// 2.82 / 4.93, 2368 x 2048, 32 rows times steps, 3.69 / 5.28 and 3.21 / 5.32, 3552 x 2048, 48, 4 rows 4.18 / 5.34 and 3.83 / 5.36; 1184 x
// 6144, 48 in six steps, 2 rows 5.55 / 5.74 and 5.31 / 7.50, 2368 x 4096, 64, 8 rows 4.80 / 5.31 and 4.70 / 6.62, 2560 x 2560, 72, one row
// 5.31 / 5.50 and 5.48 / 6.95 (129 SMs of 148 had work).
__host__ __device__ constexpr bool small_capable(int m) { return m <= 8; }
constexpr int kSmallNvfp4 = 48;
constexpr int kSmallSmem = 111 * 1024;     // dynamic shared memory: 228 KB for two, less 1 KB and the static part each
constexpr int kBoxRows = 8;                // tile rows come in multiples of these
constexpr int kGroupRows = 16;             // rows of one mma tile
constexpr int kMaxGroups = 4;              // mma tiles of rows a warp holds at most
constexpr int kSmemHeader = 256;           // mbarriers + abort flag
constexpr int kStaticSmem = 1024;          // room left for the kernels' static shared memory
constexpr int kSmemLimit = 232448 - kStaticSmem;   // dynamic shared memory per CTA (sm_100 has 227 KB in all)
constexpr unsigned long long kWaitLimitNs = 2000000000ull;   // bounded waits give up after this (default; the host
                                                             // can set another limit, Params::wait_limit_ns)

// status word bits written on a wait that ran out (never expected; the host can read the word)
constexpr int kStatusProducerTimeout = 1;
constexpr int kStatusConsumerTimeout = 2;
constexpr int kStatusGatherTimeout = 4;
constexpr int kMaxRanks = 8;
// Time stamps (%globaltimer, ns) a CTA leaves in Params::trace when a trace buffer is set: kernel entry, the wait for
// the previous kernel of the stream passed, first stage full, last stage consumed, last warp done; then the SM id.
constexpr int kTraceSlots = 8;
enum : int { TRACE_ENTRY = 0, TRACE_DEP = 1, TRACE_FIRST_FULL = 2, TRACE_LAST_CONSUMED = 3, TRACE_EXIT = 4, TRACE_SM = 5 };

// E: elements of a 16-byte block; STEP: bytes of one step of a row (eight chunks, one per consumer warp; BF16's are twice
// as long, so that its sums take no more additions than the other formats'); SCB: scale bytes of one step; PAD: bytes a row's window is stored apart
// beyond its length, so that the eight lanes of one shared-memory access phase fall into different banks (two rows'
// 64-byte chunks, four rows' 32-byte blocks for MXFP8). The copies bring the padding from the next window.
template <int FMT> struct Format;
template <> struct Format<FMT_BF16>  { static constexpr int STEP = 1024, E = 8,  SCB = 0,  PAD = 16;  static constexpr int XROW = STEP / 16 * E * 2; };
template <> struct Format<FMT_FP8>   { static constexpr int STEP = 512, E = 16, SCB = 0,  PAD = 16;  static constexpr int XROW = STEP / 16 * E * 2; };
template <> struct Format<FMT_MXFP8> { static constexpr int STEP = 512, E = 16, SCB = 16, PAD = 32;  static constexpr int XROW = STEP / 16 * E * 2; };
template <> struct Format<FMT_NVFP4> { static constexpr int STEP = 512, E = 32, SCB = 64, PAD = 16;  static constexpr int XROW = STEP / 16 * E * 2; };
constexpr int kScalePad = 16;

// Shared-memory distance of two rows of a window of `steps` steps: weights, and staged scales.
__host__ __device__ constexpr int step_bytes(int fmt) { return fmt == FMT_BF16 ? 1024 : 512; }
__host__ __device__ constexpr int weight_pitch(int fmt, int steps) { return steps * step_bytes(fmt) + (fmt == FMT_MXFP8 ? 32 : 16); }
__host__ __device__ constexpr int scale_pitch(int fmt, int steps) {
  return fmt == FMT_NVFP4 ? steps * 64 + kScalePad : fmt == FMT_MXFP8 ? steps * 16 + kScalePad : 0;
}
// Columns (activation rows, in eights) an instance multiplies.
__host__ __device__ constexpr int column_tiles(int m) { return m <= 8 ? 1 : 2; }
__host__ __device__ constexpr bool split_columns(int fmt) { return fmt == FMT_BF16 || fmt == FMT_MXFP8; }   // see fragment_column
// Ways of the activations into shared memory (Params::x_mode).
enum : int { X_RESIDENT = 0, X_TENSOR = 1, X_COPIED = 2 };

// Offset of the activations in a stage: the ring starts kSmemHeader bytes into shared memory, stages are multiples of 1024
// bytes where they hold activations, which must start on such a multiple (the swizzle goes by address).
__host__ __device__ constexpr int x_offset(int before) { return ((before + kSmemHeader + 1023) & ~1023) - kSmemHeader; }

// Resident activations (X_RESIDENT, decided by the launch plan): FP8 / NVFP4 at up to 4 rows, where the whole
// [M][K] activations are small, keep them in shared memory behind the ring for the whole kernel instead of copying a
// window of them into every ring stage: one tensor copy brings them, and the consumer warps put them into the form the
// tensor cores take (see prepare_resident) while the first weights are on their way.
__host__ __device__ constexpr bool resident_capable(int fmt, int m) { return (fmt == FMT_FP8 || fmt == FMT_NVFP4) && m <= 4; }
constexpr int kResidentLimit = 96 * 1024;   // bytes behind the ring that resident activations take at most
// The exponents of resident BF16 activations (see prepare_resident): a byte per consumer warp, step and row.
constexpr int kResidentExps = kResidentLimit / Format<FMT_FP8>::XROW * kConsumers;
static_assert(kResidentExps + (kMaxStages + 1) * 8 <= kStaticSmem, "static shared memory");

struct Params {
  const void* x;             // [M][ldx] BF16 or FP16
  const uint8_t* w;          // weight rows, row_bytes apart
  const uint8_t* scales;     // NVFP4 E4M3 [N][K/16] (or tiled), MXFP8 E8M0 [N][K/32]; else null
  const float* row_scale;    // FP8 row scale / NVFP4 inverse global scale [N]; else null
  void* out;                 // [M][ldo]
  int* status;               // device word for kStatus* bits
  int ldx, ldo, out_kind;
  int N, K;
  int row_bytes;             // bytes of one weight row
  int nblk;                  // 16-byte blocks per row
  int scale_row_bytes;       // bytes of one row-major scale row
  int scale_mode;            // SCALES_*
  int ct;                    // tiled scales: 4-block tiles per tile row
  int M;                     // activation rows
  int cols_each, cols_more;  // the CTAs' output columns (see Walk)
  int small;                 // 1: a small launch (see kSmallThreads)
  int batch_copies;          // batched launches, first GEMV: some GEMV of the batch needs the copying warps (copies_needed)
  int steps;                 // 512-byte steps per ring stage
  int stages;                // ring depth
  int tile_rows;             // rows of a full tile (a multiple of 8; gate_up: of 16, for both regions), at most 16 * kMaxGroups
  int stage_bytes;           // bytes of one ring stage
  int early_weights;         // 1: weight copies may be issued before the previous kernel of the stream completed
  int streamed;              // 1: weights and scales leave L2 first (see kStreamed in dg_abi.cu); NVFP4's always do
  int last_rows;             // rows of the copies of a tile that is not full (per region; a multiple of 8)
  // SwiGLU epilogue (pairs > 0): the matrix is a gate_up projection of 2 * pairs rows, gate rows [0, pairs) and up rows
  // [pairs, 2 pairs); N counts its output columns (= pairs). A tile holds row k of both halves and writes
  // out[m][k] = silu(gate) * up (FP32, one rounding) instead of the two sums: `pairs` columns.
  int pairs;
  // Activations: X_RESIDENT (resident_capable; the kernel's dynamic shared memory holds, x_res_off bytes in, the steps of
  // M x XROW bytes, unswizzled, FP16), or a
  // window of them in every ring stage, by one tensor copy (X_TENSOR). Where K is no multiple of 64 (X_COPIED) the copying warps bring
  // the windows that a row ends in (see tensor_windows).
  int x_mode, x_res_off;
  int x_box_steps;           // X_RESIDENT: steps of one copy of the activations; X_COPIED: 0 where there is no map for a window
  unsigned long long* trace; // diagnostic (dg_set_trace): kTraceSlots time stamps per CTA, or null
  unsigned long long wait_limit_ns;   // every wait in the kernel gives up after this long (status word, then leaves)
  // All-gather epilogue (world >= 1, 0 = off): this rank's [M][N] results go into slot `rank` of its own
  // [world][M][N] buffer; every CTA then copies its rows to the same slot of every other rank's buffer (peer_out[q],
  // peer-mapped addresses) and counts itself done in word 2 of this rank's counter block; the last CTA adds 1 to
  // word `gather_slot` (0 or 1) of every rank's block (peer_flag[q]) and waits until its own word holds `world`, then
  // clears it: when the kernel ends, every rank's data has landed here.
  int world, rank, gather_slot, gather_nowait;   // nowait: signal only; dg_enqueue_gather_wait collects later
  void* peer_out[kMaxRanks];
  unsigned int* peer_flag[kMaxRanks];
  // Tensor maps over the weight rows and the row-major scale rows as 8-byte elements: box = one window and its padding of
  // a full tile's rows (per region, see Walk), or of last_rows rows. Rows are 16-byte multiples apart, as the encoder asks.
  alignas(64) CUtensorMap tmap_w, tmap_w_last, tmap_sc, tmap_sc_last;
  // The activations as [K / 64][M][64 elements]. X_TENSOR, X_COPIED: 128-byte swizzled, box = the blocks of one window (X_COPIED: a map
  // only where a row has one); X_RESIDENT: as they are, box = those of x_box_steps steps.
  alignas(64) CUtensorMap tmap_x;
};

// ---------------------------------------------------------------------------------------------------------------
// PTX wrappers: mbarriers, tensor copies (TMA), cp.async tied to an mbarrier.

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_count(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait. False when it gave up or another thread of the CTA already had: the caller leaves its loops.
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void trace_stamp(unsigned long long* trace, int slot) {   // the latest stamp of a slot wins
  if (trace) atomicMax(trace + (size_t)blockIdx.x * kTraceSlots + slot, global_ns());
}
// The limit sits in shared memory right after the abort flag (written once by the kernel's first thread).
static __device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const unsigned long long start = global_ns();
  const unsigned long long limit = *reinterpret_cast<const volatile unsigned long long*>(abort_flag + 2);
  do {
    if (*abort_flag) return false;
#pragma unroll 1
    for (int i = 0; i < 64; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (mbar_try_wait(bar, parity)) return true;
    }
  } while (global_ns() - start <= limit);
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, abort_flag);
}
// The policy of copies of what is read once and leaves L2 first.
__device__ __forceinline__ uint64_t read_once() {
  uint64_t policy;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
// 2-D tiled tensor copy: box of the tensor map at element column x, row y.
__device__ __forceinline__ void tensor_g2s(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar, bool streamed, uint64_t policy) {
  if (streamed)
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar), "l"(policy)
                 : "memory");
  else
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
// The same box into L2 only. (Without the hint: 4096 x 4096 NVFP4, one row, eager 5.37 with it, 5.25 without; large ones the same.)
__device__ __forceinline__ void tensor_prefetch(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
// 3-D: from (0, 0, z) on.
__device__ __forceinline__ void tensor3_g2s(uint32_t dst, const CUtensorMap* map, int z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(0), "r"(z), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// `valid` of the bytes, zeros for the rest
__device__ __forceinline__ void cp_async16_part(uint32_t dst, const void* src, int valid) {
  const void* granule = reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(granule), "r"(valid) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Offset of the byte of 16-block j (j even) of row n in cuBLASLt's 128 x 4 tiled scale layout, ct tiles per tile
// row: the layout the reference reads at decode_gemv.cu:78-82.
__device__ __forceinline__ size_t tiled_scale_offset(int n, int j, int ct) {
  const int r = n & 127;
  return ((size_t)(n >> 7) * ct + (j >> 2)) * 512 + (size_t)(r & 31) * 16 + (r >> 5) * 4 + (j & 3);
}
__device__ __forceinline__ void store_out(void* out, int kind, size_t idx, float v) {
  if (kind == OUT_F32) reinterpret_cast<float*>(out)[idx] = v;
  else if (kind == OUT_BF16) reinterpret_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(out)[idx] = __float2half_rn(v);
}

// A CTA's barriers (shared-memory addresses, 8 bytes per stage) and abort word. full: the stage's window has come; empty: its
// eight consumers have left it (a tile's last window: the finishing warps have, for all eight); sums: in a tile's last
// window, its eight consumers have left their sums in it.
struct Bars {
  uint32_t full, empty, sums, x;   // x (one for the CTA): the resident activations have come
  uint32_t exps;                   // the resident activations' exponents (kResidentExps bytes)
  volatile int* abort_flag;
};

// ---------------------------------------------------------------------------------------------------------------
// Tile walk shared by all warps: CTA c owns the output columns [lo, hi), walked in tiles of `cap` columns, the last one what is
// left. A tile's rows in the stage: its columns' matrix rows (regions = 1), or, for a gate_up matrix with the SwiGLU epilogue
// (regions = 2), its columns' gate rows and, from row cap on, their up rows.

// First column of CTA c: the first cols_more CTAs have cols_each + 1, the others cols_each.
__device__ __forceinline__ int first_column(const Params& p, unsigned c) { return (int)c * p.cols_each + min((int)c, p.cols_more); }

struct Walk {
  int lo, hi, cap, regions, ntiles, nwin;
  int pairs;                     // SwiGLU epilogue: rows per half of the gate_up matrix (0: an ordinary matrix)
  __device__ __forceinline__ Walk(const Params& p, int window_bytes) {
    pairs = p.pairs;
    lo = first_column(p, blockIdx.x);
    hi = first_column(p, blockIdx.x + 1);
    regions = pairs ? 2 : 1;
    cap = pairs ? p.tile_rows >> 1 : p.tile_rows;
    ntiles = (int)((unsigned)(hi - lo + cap - 1) / (unsigned)cap);
    nwin = (p.row_bytes + window_bytes - 1) / window_bytes;
  }
  // First column and width of tile t.
  __device__ __forceinline__ void tile(int t, int& col0, int& cols) const {
    col0 = lo + t * cap;
    cols = min(cap, hi - col0);
  }
  // Rows a tile of `cols` columns takes in the stage, and the matrix row of one of them (where there is one).
  __device__ __forceinline__ int rows(int cols) const { return (regions - 1) * cap + cols; }
  __device__ __forceinline__ int matrix_row(int col0, int cols, int r) const {
    return r < cap ? col0 + min(r, cols - 1) : pairs + col0 + (r - cap);
  }
};

// Shared-memory stage: [weights, rows weight_pitch apart][scales, rows scale_pitch apart][x: per step XROW / 128 blocks of
// K, each M rows of 128 bytes, on a multiple of 1024 bytes]. Boxes of kBoxRows rows start on 128 bytes, as tensor copies
// ask.
template <int FMT, int STEPS>
struct StageLayout {
  static constexpr int W_ROW = weight_pitch(FMT, STEPS), SC_ROW = scale_pitch(FMT, STEPS);
  int sc_off, x_off;
  __device__ __forceinline__ StageLayout(const Params& p) {
    sc_off = p.tile_rows * W_ROW;
    x_off = x_offset(p.tile_rows * (W_ROW + SC_ROW));
  }
};

// Where 16-byte slot s (0..7) of row r of the activation blocks lies: the 128-byte swizzle of the tensor copies.
__device__ __forceinline__ int x_slot(int r, int s) { return r * 128 + ((s ^ (r & 7)) << 4); }

// ---------------------------------------------------------------------------------------------------------------
// Producer warps.

// Programmatic dependent launch: the next kernel of the stream may start while this one runs, and this one may have
// started while the previous one ran. `griddep_wait` returns once the previous kernel has completed and its writes
// are visible; without the launch attribute both are no-ops.
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Block scales that bulk copies cannot bring (row-major rows that are no multiples of 16 bytes or lie off 16 bytes, or
// cuBLASLt's tiles): the activation producers copy them themselves.
template <int FMT>
__device__ __forceinline__ bool scales_gathered(const Params& p) {
  return Format<FMT>::SCB != 0 && p.scale_mode != SCALES_STAGED;
}

// Resident activations: all of them, in as few copies as boxes allow (one thread).
template <int FMT>
__device__ __forceinline__ void copy_resident(const Params& p, const Params& maps, unsigned char* smem, const Bars& bars) {
  constexpr int XROW = Format<FMT>::XROW;
  const int steps = (p.row_bytes + Format<FMT>::STEP - 1) / Format<FMT>::STEP, bytes = p.M * XROW;
  mbar_arrive_expect_tx(bars.x, (uint32_t)(steps * bytes));
  for (int st = 0; st < steps; st += p.x_box_steps)
    tensor3_g2s(smem_addr(smem) + (uint32_t)(p.x_res_off + st * bytes), &maps.tmap_x, st * (XROW / 128), bars.x);
}

// Windows whose activations one tensor copy brings: all, or where K is no multiple of 64 those that lie within the rows (past their end a
// copy would bring the next row's values). The two copying warps, 16 bytes a copy, cannot keep up with more than a few rows: us at
// 12490 x 5088 with 8 / 16 rows, all windows by them and only the last: NVFP4 24.0 / 37.9 and 15.2 / 23.4, FP8 19.0 / 45.3 and 16.2 / 20.8,
// MXFP8 22.7 / 42.6 and 17.3 / 22.6, BF16 24.1 / 36.2 and 23.5 / 26.8; NVFP4 40000 x 8160 93 / 144 and 56 / 81.
template <int FMT, int STEPS, bool RESIDENT>
__device__ __forceinline__ int tensor_windows(const Params& p) {
  if constexpr (RESIDENT) return 0;
  constexpr int WINDOW = STEPS * Format<FMT>::XROW / 2;                   // elements
  return p.x_mode == X_TENSOR ? (p.K + WINDOW - 1) / WINDOW : p.x_mode == X_COPIED && p.x_box_steps ? p.K / WINDOW : 0;
}

// A kernel's first activations, the moment the previous kernel of the stream has finished (the finishing warp has nothing else
// to do then): the resident ones, or those of the windows that fill the ring.
template <int FMT, int STEPS, bool RESIDENT>
__device__ __forceinline__ void start_activations(const Params& p, const Params& maps, unsigned char* smem, const Bars& bars) {
  constexpr int X_BLOCKS = STEPS * Format<FMT>::XROW / 128;
  const int by_tensor = tensor_windows<FMT, STEPS, RESIDENT>(p);
  const bool resident = RESIDENT || p.x_mode == X_RESIDENT;
  if ((threadIdx.x & 31) == 0 && (by_tensor > 0 || resident)) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.tmap_x) : "memory");
  const Walk wk(p, STEPS * Format<FMT>::STEP);
  griddep_wait();
  if ((threadIdx.x & 31) != 0) return;
  if (resident && wk.ntiles > 0) copy_resident<FMT>(p, maps, smem, bars);
  if (by_tensor == 0) return;
  const uint32_t at = smem_addr(smem) + kSmemHeader +
                      (uint32_t)x_offset(p.tile_rows * (weight_pitch(FMT, STEPS) + scale_pitch(FMT, STEPS)));
  const int windows = min(p.stages, wk.ntiles * wk.nwin);
  for (int i = 0, win = 0; i < windows; ++i) {
    if (win < by_tensor) tensor3_g2s(at + (uint32_t)i * p.stage_bytes, &maps.tmap_x, win * X_BLOCKS, bars.full + 8u * i);
    if (++win == wk.nwin) win = 0;
  }
}

// The ring's first filling is paced: asked for all at once, the first windows came as late as the last, up to 3 us later on some
// SMs than on others. 22 bytes per clock and SM are 6.4 TB/s from 148 SMs at 1965 MHz, just under what HBM gives (6.55); fewer SMs
// or a lower clock ask for less, and so do weights that lie in L2, for the first filling only. Measured at 1965 MHz, us with 19 /
// 22 / 26 bytes and without pacing: NVFP4 10240 x 8192, one row 13.6 / 13.8 / 14.2 / 14.2, 8192 x 8192, 8 rows 12.7 / 12.6 / 12.2 /
// 12.5; FP8 4096 x 4096, one row 5.62 / 5.74 / 5.87 / 5.88, 8 rows 7.1 / 6.6 / 6.2 / 6.7, 4096 x 14336, one row 13.5 / 13.0 / 12.5 /
// 12.6; BF16 4096 x 2048, one row 5.24 / 5.27 / 5.39 / 5.45, 8 rows 5.87 / 5.51 / 5.20 / 5.49: few rows like it slower, many faster.
constexpr int kUnpaced = 32 * 1024, kPace = 22;   // bytes at once, bytes per clock

// The feeding warp: weight (and staged scale) copies of every window of one GEMV, in order, and the activations' tensor
// copies. A tile's rows travel as ONE 2-D tensor copy per region (and one for their scales): a copy costs the SM about 150
// clocks to start whatever its size (as boxes of 8 rows, 12 to 16 a window, or with single rows for a tile's remainder they
// bounded the whole kernel at 1 us a window). A box is always brought whole: columns past the matrix row's end and rows past
// the matrix come as zeros and count; rows past the tile are not used. One arrival carries the byte count of all copies;
// completions may land before it (the phase cannot end while it is outstanding). The activations of a kernel's first windows
// are not its business (see start_activations): the previous kernel of the stream may not have been waited for yet when
// the ring fills. The ring position (stage s, its phase parity) is the caller's and
// carries on from one GEMV of a batch to the next (`first`: its first; `wait`: the previous kernel of the stream has to be
// waited for); `maps`: where the tensor maps are read from.
template <int FMT, int STEPS, bool RESIDENT>
__device__ __forceinline__ bool feed_weights(const Params& p, const Params& maps, unsigned char* smem, const Bars& bars,
                                             bool first, bool wait, int& s, uint32_t& parity) {
  constexpr int SCB = Format<FMT>::SCB, WIN = STEPS * Format<FMT>::STEP, SC_WIN = STEPS * SCB;
  constexpr int W_ROW = weight_pitch(FMT, STEPS), SC_ROW = scale_pitch(FMT, STEPS), XROW = Format<FMT>::XROW;
  const Walk wk(p, WIN);
  const int lane = threadIdx.x & 31, stage_bytes = p.stage_bytes, stages = p.stages;
  const bool staged = SCB != 0 && p.scale_mode == SCALES_STAGED;
  const uint32_t ring = smem_addr(smem) + kSmemHeader, sc_off = (uint32_t)(p.tile_rows * W_ROW);
  // activations by tensor copy: a window at a time
  constexpr int X_BLOCKS = STEPS * XROW / 128;
  const uint32_t x_off = (uint32_t)x_offset(p.tile_rows * (W_ROW + SC_ROW));
  const uint32_t x_bytes = (uint32_t)(X_BLOCKS * 128 * p.M);
  const int by_tensor = tensor_windows<FMT, STEPS, RESIDENT>(p);
  auto activations = [&](int at, int win) {
    if (win >= by_tensor || lane != 31) return;
    // (the copying warps may have written there before)
    if (p.x_mode == X_COPIED) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tensor3_g2s(ring + (uint32_t)at * stage_bytes + x_off, &maps.tmap_x, win * X_BLOCKS, bars.full + 8u * at);
  };
  // or all at once: when nobody reads the previous GEMV's any more, which is known once the last of its stages is empty
  bool x_due = p.x_mode == X_RESIDENT && wk.ntiles > 0 && !first;
  auto resident = [&] {
    if (x_due && lane == 31) copy_resident<FMT>(p, maps, smem, bars);
    x_due = false;
  };
  auto wait_empty = [&](int at, uint32_t use) {
    if (mbar_wait(bars.empty + 8u * at, use ^ 1u, bars.abort_flag)) return true;
    if (lane == 0 && p.status) atomicOr(p.status, kStatusProducerTimeout);
    return false;
  };
  const uint64_t policy = read_once();
  if (wait) griddep_wait();   // (with everything worked out)
  int filled = 0;
  const long long start = clock64();
  // (in code of its own for streamed weights: a branch at every copy took BF16 2816 x 11264 with 5 rows from 13.6 to 13.8 us)
  auto copies = [&](auto kind) {
    constexpr bool streamed = decltype(kind)::value;
    for (int t = 0; t < wk.ntiles; ++t) {
      int col0, cols;
      wk.tile(t, col0, cols);
      const bool full_tile = cols == wk.cap;
      const CUtensorMap* const map_w = full_tile ? &maps.tmap_w : &maps.tmap_w_last;
      const CUtensorMap* const map_sc = full_tile ? &maps.tmap_sc : &maps.tmap_sc_last;
      const uint32_t bytes = wk.regions * (full_tile ? wk.cap : p.last_rows) * (uint32_t)(W_ROW + (staged ? SC_ROW : 0));
      // lanes 0, 1: the regions' weights; 2, 3: their scales
      const int region = lane & 1, n0 = region * wk.pairs + col0, row0 = region * wk.cap;
      for (int win = 0; win < wk.nwin; ++win) {
        if (!wait_empty(s, parity)) return false;
        if (++filled == stages) resident();
        if (first && filled == stages + 1) griddep_wait();   // (passed by now, but not by this warp)
        if (first && filled > 1 && filled <= stages && !p.small) {   // (see kPace)
          const int due = ((filled - 1) * stage_bytes - kUnpaced) / kPace;
          while ((int)(clock64() - start) < due) {}
        }
        const uint32_t full = bars.full + 8u * s, stage = ring + (uint32_t)s * stage_bytes;
        if (lane == 0) mbar_arrive_expect_tx(full, bytes + (win < by_tensor ? x_bytes : 0u));
        __syncwarp();
        if (!first || filled > stages) activations(s, win);
        if (region < wk.regions) {
          if (lane < 2) tensor_g2s(stage + row0 * W_ROW, map_w, (win * WIN) >> 3, n0, full, streamed, policy);
          else if (lane < 4 && staged) tensor_g2s(stage + sc_off + row0 * SC_ROW, map_sc, (win * SC_WIN) >> 3, n0, full, streamed, policy);
        }
        if (++s == stages) { s = 0; parity ^= 1u; }
      }
    }
    return true;
  };
  if (FMT == FMT_NVFP4 || p.streamed != 0) {
    if (!copies(std::true_type())) return false;
  } else {
    if (!copies(std::false_type())) return false;
  }
  if (x_due) {                     // fewer windows than stages
    int at = s;
    uint32_t use = parity;
    for (int i = filled; i < stages - 1; ++i)
      if (++at == stages) { at = 0; use ^= 1u; }
    if (!wait_empty(at, use)) return false;
    resident();
  }
  return true;
}

// The first window's weights (and staged scales; a small launch: all of them) into L2, before the wait for the previous kernel
// of the stream: what that kernel may still write reaches the same L2, so the copies after the wait read its values, from L2
// instead of HBM. (Further windows would come late for the kernels still running. Small windows are not worth the traffic: 2048 x 2048 FP8 takes 4.7 us
// without and 5.0 with, 8192 x 8192 NVFP4 13.4 and 12.4.) And the tensor maps, on their way to be used.
constexpr int kPrefetchFrom = 32 * 1024;   // bytes of a stage
template <int FMT, int STEPS>
__device__ __forceinline__ void prefetch_weights(const Params& p) {
  constexpr int SCB = Format<FMT>::SCB, WIN = STEPS * Format<FMT>::STEP;
  const int lane = threadIdx.x & 31;
  if (lane < 4) {               // the maps themselves: half a microsecond at their first use
    const CUtensorMap* map = lane == 0 ? &p.tmap_w : lane == 1 ? &p.tmap_w_last : lane == 2 ? &p.tmap_sc : &p.tmap_sc_last;
    if (lane < 2 || (SCB != 0 && p.scale_mode == SCALES_STAGED)) asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
  }
  if (lane != 0 || (!p.small && p.stage_bytes < kPrefetchFrom)) return;
  const Walk wk(p, WIN);
  if (wk.ntiles == 0) return;
  int col0, cols;
  wk.tile(0, col0, cols);
  for (int win = 0; win < (p.small ? wk.nwin : 1); ++win)
    for (int region = 0; region < wk.regions; ++region) {
      const int n0 = region * wk.pairs + col0;
      tensor_prefetch(cols == wk.cap ? &p.tmap_w : &p.tmap_w_last, (win * WIN) >> 3, n0);
      if (SCB != 0 && p.scale_mode == SCALES_STAGED)
        tensor_prefetch(cols == wk.cap ? &p.tmap_sc : &p.tmap_sc_last, (win * STEPS * SCB) >> 3, n0);
    }
}

// The other producer warps, where they are needed: the windows' activations where no tensor copy can bring them, 16 bytes
// (8 elements) per copy, and the scales that are gathered; then every lane's arrival, which fires when its copies have
// landed.
template <int FMT, bool RESIDENT>
__device__ __forceinline__ bool copies_needed(const Params& p) { return (!RESIDENT && p.x_mode == X_COPIED) || scales_gathered<FMT>(p); }

// (zeros past the row's end, by stores, which the lane's arrival on the stage's barrier must follow: returns true then)
template <int FMT, int STEPS>
__device__ __forceinline__ bool copy_activations(const Params& p, uint32_t dst, int win, int warp, int lane) {
  constexpr int SLOTS = STEPS * Format<FMT>::XROW / 16;
  const int M = p.M, k0 = win * SLOTS * 8, slots = min(SLOTS, (p.K - k0) >> 3);
  for (int m = warp; m < M; m += kCopyWarps) {
    const unsigned char* src = reinterpret_cast<const unsigned char*>(p.x) + ((size_t)m * p.ldx + k0) * 2;
    for (int i = lane; i < SLOTS; i += 32) {
      const uint32_t to = dst + x_slot((i >> 3) * M + m, i & 7);
      if (i < slots) cp_async16(to, src + (size_t)i * 16);
      else sts128(to, make_uint4(0u, 0u, 0u, 0u));
    }
  }
  return slots < SLOTS;
}

// Whether gathered row-major scales travel in whole 16-byte granules: a row's place in the stage is then as far off 16 bytes
// as its address is (scale_shift), which rows eight apart share (their distance is a multiple of 16 bytes; MXFP8: of 8).
template <int FMT>
__device__ __forceinline__ bool scale_granules(const Params& p) {
  return Format<FMT>::SCB != 0 && p.scale_mode == SCALES_DIRECT && (((size_t)p.pairs * p.scale_row_bytes) & 15) == 0;
}
__device__ __forceinline__ uint32_t scale_shift(const Params& p, int n) {
  return (uint32_t)(reinterpret_cast<uintptr_t>(p.scales) + (size_t)n * p.scale_row_bytes) & 15u;
}

// Scale bytes of the window for every row of the tile, zeros past the row's end. Row-major rows: 16 bytes at a time, from the
// granule the window starts in on. Tiles: four blocks' bytes of a row at a time; a lane stays with its row. What neither fits
// goes byte by byte through registers, to the places a bulk copy would use; the lane's arrival on the stage's barrier must
// follow the stores (returns true then). One warp issues few instructions while the others compute, so the loops are kept
// short: with addresses worked out anew for each four bytes, 20000 x 6016 took 30 us (now 21), and from rows off four bytes,
// byte by byte, 40000 x 4128 took 137 us (now 36).
template <int FMT, int STEPS>
__device__ __forceinline__ bool gather_scales(const Params& p, const Walk& wk, uint32_t dst, int col0, int cols, int win,
                                              int warp, int lane) {
  constexpr int SCB = Format<FMT>::SCB, SC_ROW = scale_pitch(FMT, STEPS), WINDOW = STEPS * SCB;
  const int rows = wk.rows(cols), byte0 = win * WINDOW, sc_bytes = p.row_bytes * SCB / Format<FMT>::STEP;   // of a row's scales
  const bool tiled = p.scale_mode == SCALES_BLOCKED;
  if (scale_granules<FMT>(p)) {
    constexpr int GRANULES = WINDOW / 16 + 1;
    const uint8_t* base = p.scales + byte0;
    for (int i = warp * 32 + lane; i < rows * GRANULES; i += 32 * kCopyWarps) {
      const int r = i / GRANULES, g = i - r * GRANULES;
      const uint8_t* row = base + (size_t)wk.matrix_row(col0, cols, r) * p.scale_row_bytes;
      const int off = 16 * g - (int)(reinterpret_cast<uintptr_t>(row) & 15);        // of the granule from the window's start
      const int valid = max(0, min(16, sc_bytes - byte0 - off));
      cp_async16_part(dst + (uint32_t)(r * SC_ROW + 16 * g), row + (valid > 0 ? off : 0), valid);
    }
    return false;
  }
  if (tiled && (reinterpret_cast<uintptr_t>(p.scales) & 3) == 0) {
    for (int r = lane; r < rows; r += 32) {
      const int n = wk.matrix_row(col0, cols, r);
      const uint8_t* src = p.scales + tiled_scale_offset(n, byte0 + 4 * warp, p.ct);
      uint32_t to = dst + (uint32_t)(r * SC_ROW + 4 * warp);
      int left = sc_bytes - byte0 - 4 * warp;
#pragma unroll 4
      for (int u = warp; u < WINDOW / 4; u += kCopyWarps) {
        cp_async4(to, left > 0 ? src : p.scales, max(0, min(4, left)));
        src += 512 * kCopyWarps;
        to += 4 * kCopyWarps;
        left -= 4 * kCopyWarps;
      }
    }
    return false;
  }
  for (int r = warp; r < rows; r += kCopyWarps) {
    const int n = wk.matrix_row(col0, cols, r);
    for (int b = lane; b < WINDOW; b += 32) {
      const int j = byte0 + b;
      const uint8_t* src = p.scales + (tiled ? tiled_scale_offset(n, j & ~1, p.ct) + (j & 1) : (size_t)n * p.scale_row_bytes + j);
      sts_u8(dst + (uint32_t)(r * SC_ROW + b), j < sc_bytes ? (uint32_t)*src : 0u);
    }
  }
  return true;
}

template <int FMT, int STEPS, bool RESIDENT>
__device__ __forceinline__ bool feed_activations(const Params& p, unsigned char* smem, const Bars& bars, int warp, int& s,
                                                 uint32_t& parity) {
  const Walk wk(p, STEPS * Format<FMT>::STEP);
  const StageLayout<FMT, STEPS> lay(p);
  const int lane = threadIdx.x & 31;
  const bool gathered = scales_gathered<FMT>(p);
  const int by_tensor = tensor_windows<FMT, STEPS, RESIDENT>(p);
  const uint32_t ring = smem_addr(smem) + kSmemHeader;
  for (int t = 0; t < wk.ntiles; ++t) {
    int col0, cols;
    wk.tile(t, col0, cols);
    for (int win = 0; win < wk.nwin; ++win) {
      if (!mbar_wait(bars.empty + 8u * s, parity ^ 1u, bars.abort_flag)) {
        if (lane == 0 && p.status) atomicOr(p.status, kStatusProducerTimeout);
        return false;
      }
      const uint32_t full = bars.full + 8u * s, stage = ring + (uint32_t)s * p.stage_bytes;
      bool stored = false;
      if constexpr (Format<FMT>::SCB != 0) {
        if (gathered) stored = gather_scales<FMT, STEPS>(p, wk, stage + lay.sc_off, col0, cols, win, warp, lane);
      }
      if (!RESIDENT && p.x_mode == X_COPIED && win >= by_tensor) stored |= copy_activations<FMT, STEPS>(p, stage + lay.x_off, win, warp, lane);
      if (stored) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        mbar_arrive(full);
      } else {
        cp_async_arrive_noinc(full);
      }
      if (++s == p.stages) { s = 0; parity ^= 1u; }
    }
  }
  return true;
}

// ---------------------------------------------------------------------------------------------------------------
// Consumers.

// What a consumer lane needs of the launch, held in registers or as constants of the tile.
struct Lane {
  int g, t, warp;              // lane / 4, lane % 4, consumer warp
  __device__ __forceinline__ Lane() : g((threadIdx.x & 31) >> 2), t(threadIdx.x & 3), warp(threadIdx.x >> 5) {}
};
// Tile row (of eight) that lane group g supplies. Rows lie PAD bytes off a multiple of 128 apart: with 16 the rows that
// share an access phase (g = 2q, 2q + 1) must be four apart to lie 64 bytes apart; with 32 (MXFP8, four rows a phase)
// the natural order does.
template <int FMT>
__device__ __forceinline__ int fragment_row(int g) {
  return FMT == FMT_MXFP8 ? g : (g >> 1) | ((g & 1) << 2);
}

// Activation row (of eight) that lane group g supplies, likewise: the two of a phase lie in 128-byte rows whose slots the
// swizzle permutes by row; where a lane's slots are four apart (BF16, MXFP8) the two must differ in bit 2.
template <int FMT>
__device__ __forceinline__ int fragment_column(int g) {
  return split_columns(FMT) ? (g >> 1) | ((g & 1) << 2) : g;
}

// A lane's share of one chunk of 16 rows: PIECES times 16 bytes of rows g and g + 8, with their scales (NVFP4: two E4M3
// of the two 16-blocks in the low 16 bits; MXFP8: two E8M0 of the chunk's two blocks).
template <int FMT> struct Fragment {
  static constexpr int CHUNK = Format<FMT>::STEP / kConsumers, PIECES = CHUNK / 64;
  static constexpr int NB = PIECES * Format<FMT>::E / 2, SUB = NB / 4;   // pairs a lane holds per row; eights of them
};
template <int FMT> struct RawRows { uint4 lo[Fragment<FMT>::PIECES], hi[Fragment<FMT>::PIECES]; uint32_t slo, shi; };

template <int FMT>
__device__ __forceinline__ uint4 load_piece(uint32_t row, int t, int piece) {   // `row`: the chunk of one row
  if constexpr (FMT == FMT_MXFP8) {
    const uint2 a = lds64(row + t * 8), b = lds64(row + 32 + t * 8);
    return make_uint4(a.x, a.y, b.x, b.y);
  } else {
    return lds128(row + piece * 64 + t * 16);
  }
}

// Weights of sub-block q (8 per row: four pairs) in the tensor cores' 16-bit type.
template <int FMT>
__device__ __forceinline__ void decode_sub(const uint4 (&v)[Fragment<FMT>::PIECES], uint32_t scale2, int q, uint32_t (&h)[4]) {
  if constexpr (FMT == FMT_BF16) {
    h[0] = v[q].x; h[1] = v[q].y; h[2] = v[q].z; h[3] = v[q].w;
  } else if constexpr (FMT == FMT_NVFP4) {
    decode_e2m1_h(q == 0 ? v[0].x : q == 1 ? v[0].y : q == 2 ? v[0].z : v[0].w, h);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = mul_half2(h[i], scale2);
  } else {
    decode_e4m3_h(q ? v[0].z : v[0].x, q ? v[0].w : v[0].y, h);
  }
}

// One chunk of 16 rows into the running sums: acc[nt][0] rows g, acc[nt][1] rows g + 8, columns (2 t, 2 t + 1) + 8 nt.
// ACTS: the activations are used as they came (ACTS_PLAIN), are FP16 times the usual power of two (ACTS_USUAL) or one of their
// column, which `unscale` takes off again (ACTS_SCALED), or are BF16 beside weights that decode to FP16 (ACTS_WIDE).
enum : int { ACTS_PLAIN = 0, ACTS_USUAL = 1, ACTS_SCALED = 2, ACTS_WIDE = 3 };
// HALF: there are no rows g + 8; their products are neither made nor added.
template <int FMT, int NT, int ACTS, bool HALF>
__device__ __forceinline__ void chunk_rows(const RawRows<FMT>& raw, const uint32_t (&b)[NT][Fragment<FMT>::NB],
                                           const pk2 (&unscale)[NT], pk2 (&acc)[NT][2]) {
  constexpr int SUB = Fragment<FMT>::SUB, PER = SUB / 2;   // two chains: of four steps (NVFP4) or two
  constexpr bool BF = FMT == FMT_BF16 || ACTS == ACTS_WIDE;
  uint32_t s2lo[2] = {0u, 0u}, s2hi[2] = {0u, 0u};
  if constexpr (FMT == FMT_NVFP4) {
    const uint32_t a = e4m3x2_to_half2(raw.slo);
    s2lo[0] = __byte_perm(a, a, 0x1010); s2lo[1] = __byte_perm(a, a, 0x3232);
    if constexpr (!HALF) {
      const uint32_t c = e4m3x2_to_half2(raw.shi);
      s2hi[0] = __byte_perm(c, c, 0x1010); s2hi[1] = __byte_perm(c, c, 0x3232);
    }
  }
  float part[2][NT][4];
#pragma unroll
  for (int q = 0; q < SUB; ++q) {
    const int chain = q / PER;
    uint32_t lo[4], hi[4];
    decode_sub<FMT>(raw.lo, s2lo[q >> 1 & 1], q, lo);
    if constexpr (!HALF) {
      decode_sub<FMT>(raw.hi, s2hi[q >> 1 & 1], q, hi);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) hi[i] = lo[i];
    }
    if constexpr (ACTS == ACTS_WIDE) {
#pragma unroll
      for (int i = 0; i < 4; ++i) { lo[i] = half2_to_bf162(lo[i]); hi[i] = half2_to_bf162(hi[i]); }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (q % PER == 0) mma_step<BF, true>(part[chain][nt], lo[0], hi[0], lo[1], hi[1], b[nt][4 * q], b[nt][4 * q + 1]);
      else mma_step<BF, false>(part[chain][nt], lo[0], hi[0], lo[1], hi[1], b[nt][4 * q], b[nt][4 * q + 1]);
      mma_step<BF, false>(part[chain][nt], lo[2], hi[2], lo[3], hi[3], b[nt][4 * q + 2], b[nt][4 * q + 3]);
    }
  }
  const pk2 usual = pack2(kWindowUnscale, kWindowUnscale);
  pk2 mx[2][2];                           // MXFP8: [block][rows g, g + 8] scales, powers of two
  if constexpr (FMT == FMT_MXFP8) {
    e8m0x2_to_f32(raw.slo, mx[0][0], mx[1][0]);
    if constexpr (!HALF) e8m0x2_to_f32(raw.shi, mx[0][1], mx[1][1]);
    if (ACTS == ACTS_USUAL) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int half = 0; half < (HALF ? 1 : 2); ++half) mx[c][half] = fmul2(mx[c][half], usual);
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int half = 0; half < (HALF ? 1 : 2); ++half) {
      pk2 v0 = pack2(part[0][nt][2 * half], part[0][nt][2 * half + 1]);
      pk2 v1 = pack2(part[1][nt][2 * half], part[1][nt][2 * half + 1]);
      if constexpr (FMT == FMT_MXFP8) {
        // (a column's power of two first: the product with the block's scale is then the true one)
        if (ACTS == ACTS_SCALED) { v0 = fmul2(v0, unscale[nt]); v1 = fmul2(v1, unscale[nt]); }
        acc[nt][half] = ffma2(v1, mx[1][half], ffma2(v0, mx[0][half], acc[nt][half]));
      } else {
        v0 = fadd2(v0, v1);
        acc[nt][half] = ACTS == ACTS_USUAL || ACTS == ACTS_SCALED
                            ? ffma2(v0, ACTS == ACTS_USUAL ? usual : unscale[nt], acc[nt][half])
                            : fadd2(v0, acc[nt][half]);
      }
    }
}

// Where the lane's activations of its warp's chunk lie in a step: columns (fragment_column of g) + 8 nt, NJ slots of 16
// bytes. Columns past the last activation row repeat it: nobody reads their sums.
// (Window by window they are swizzled, see x_slot; resident ones lie as they came.)
template <int FMT, int NT, bool RES>
struct XOffsets {
  static constexpr int NJ = Fragment<FMT>::NB / 4;
  uint32_t off[NT][NJ];
  __device__ __forceinline__ XOffsets(const Lane& ln, int M) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int m = min(fragment_column<FMT>(ln.g) + 8 * nt, M - 1);
        const int slot = ln.warp * 4 * NJ + (split_columns(FMT) ? 4 * j + ln.t : NJ * ln.t + j);   // of the step's
        off[nt][j] = (uint32_t)(RES ? ((slot >> 3) * M + m) * 128 + (slot & 7) * 16 : x_slot((slot >> 3) * M + m, slot & 7));
      }
  }
};
// The activations as stored, NB pairs per column. (Past the row's end there are zeros, as in the weights and scales.)
template <int FMT, int NT, bool RES>
__device__ __forceinline__ void load_x(uint32_t xs, const XOffsets<FMT, NT, RES>& xo, uint32_t (&b)[NT][Fragment<FMT>::NB]) {
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int j = 0; j < Fragment<FMT>::NB / 4; ++j) {
      const uint4 v = lds128(xs + xo.off[nt][j]);
      b[nt][4 * j] = v.x; b[nt][4 * j + 1] = v.y; b[nt][4 * j + 2] = v.z; b[nt][4 * j + 3] = v.w;
    }
}

// The powers of two to take off the lane's sums' columns (2 t, 2 t + 1) again, from the lanes that hold these columns.
__device__ __forceinline__ pk2 column_unscale(uint32_t e, const Lane& ln) {
  e = e == kWide ? kWindowExp : e;          // (such a column is zeros)
  return pack2(exp_unscale(__shfl_sync(0xffffffffu, e, 8 * ln.t)), exp_unscale(__shfl_sync(0xffffffffu, e, 8 * ln.t + 4)));
}

__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kConsumers) : "memory"); }
// Resident activations have come as they are in global memory. BF16 ones: every consumer warp puts its own slice of K into the
// form the tiles read, FP16 times 2^7 or the chunk's own power of two, whose exponent it then leaves in `exps`, one byte
// per warp, step and row (kWide: the chunk stays BF16). No other warp reads that slice, so nobody waits for anybody. The lanes of
// a group g take activation row g % M, chunks of 8 / M steps at a time, slot by slot in place. Returns the steps (modulo 32)
// with another exponent than the usual one. (Rolled loops: this runs once per kernel, from cold instruction caches; unrolled
// over a lane's slots it took 1.0 us for a single step, now 0.6.)
template <int FMT>
__device__ __forceinline__ uint32_t prepare_resident(const Params& p, unsigned char* smem, uint32_t exps) {
  constexpr int XROW = Format<FMT>::XROW, NJ = Fragment<FMT>::NB / 4;
  const Lane ln;
  const int M = p.M, by = M == 1 ? 32 : M == 2 ? 16 : M == 3 ? 11 : 8, q = ln.g * by >> 5, m = ln.g - q * M;   // q: g / M
  const int together = M == 1 ? 8 : M == 2 ? 4 : 2, steps = (p.row_bytes + Format<FMT>::STEP - 1) / Format<FMT>::STEP;
  const int slot0 = ln.warp * 4 * NJ + NJ * ln.t;
  const uint32_t at0 = smem_addr(smem) + (uint32_t)(p.x_res_off + ((slot0 >> 3) * M + m) * 128 + (slot0 & 7) * 16);
  const uint32_t mine0 = exps + (uint32_t)(ln.warp * steps * M);
  uint32_t spread = 0u;
  bool noted = false;             // the exponents have been set to the usual one
#pragma unroll 1
  for (int st0 = 0; st0 < steps; st0 += together) {
    const int st = st0 + q;
    const bool mine = q < together && st < steps;
    const uint32_t at = at0 + (uint32_t)(st * M * XROW);
    uint32_t left = 0u;          // bit j: slot j is as it came
    if (mine) {
#pragma unroll 1
      for (int j = 0; j < NJ; ++j) {
        const uint4 v = lds128(at + 16 * j);
        if ((window_bits(v.x) | window_bits(v.y) | window_bits(v.z) | window_bits(v.w)) & kOutside)
          left |= 1u << j;
        else
          sts128(at + 16 * j, make_uint4(scaled_half2(v.x, kWindowScale), scaled_half2(v.y, kWindowScale),
                                         scaled_half2(v.z, kWindowScale), scaled_half2(v.w, kWindowScale)));
      }
    }
    if (__any_sync(0xffffffffu, left != 0u)) {
      auto slot = [&](int j, uint32_t (&v)[4]) {     // as it came
        const uint4 h = lds128(at + 16 * j);
        v[0] = h.x; v[1] = h.y; v[2] = h.z; v[3] = h.w;
        if ((left >> j & 1u) == 0u) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = window_back(v[i]);
        }
      };
      uint32_t range = 0u;
      if (mine) {
#pragma unroll 1
        for (int j = 0; j < NJ; ++j) {
          uint32_t v[4];
          slot(j, v);
          range = __vmaxu2(range, chunk_range<4>(v));
        }
      }
      const uint32_t e = chunk_exp(range);
      if (mine) {
#pragma unroll 1
        for (int j = 0; j < NJ; ++j) {
          uint32_t v[4];
          slot(j, v);
          if (e != kWide) {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = scaled_half2(v[i], exp_scale(e));
          }
          sts128(at + 16 * j, make_uint4(v[0], v[1], v[2], v[3]));
        }
      }
      if (!noted) {
        noted = true;
        for (int i = threadIdx.x & 31; i < steps * M; i += 32) sts_u8(mine0 + i, kWindowExp);
        __syncwarp();
      }
      if (mine && e != kWindowExp) {
        spread |= 1u << (st & 31);
        if (ln.t == 0) sts_u8(mine0 + st * M + m, e);
      }
    }
  }
  return __reduce_or_sync(0xffffffffu, spread);
}

// A row's two scale bytes of the lane. (Gathered MXFP8 rows may lie on odd addresses.)
template <int FMT>
__device__ __forceinline__ uint32_t load_scales(uint32_t at) {
  return FMT == FMT_MXFP8 ? lds_u8(at) | lds_u8(at + 1) << 8 : lds_u16(at);
}
// Rows g and (unless HALF) g + 8, hi_row rows further on, of the chunk at wrow / srow; sc_hi: what the latter's scales lie
// further off than srow's.
template <int FMT, int STEPS, bool HALF>
__device__ __forceinline__ void load_rows(RawRows<FMT>& raw, uint32_t wrow, uint32_t srow, int hi_row, int sc_hi, int t) {
#pragma unroll
  for (int i = 0; i < Fragment<FMT>::PIECES; ++i) {
    raw.lo[i] = load_piece<FMT>(wrow, t, i);
    if constexpr (!HALF) raw.hi[i] = load_piece<FMT>(wrow + hi_row * weight_pitch(FMT, STEPS), t, i);
  }
  if constexpr (Format<FMT>::SCB != 0) {
    raw.slo = load_scales<FMT>(srow);
    if constexpr (!HALF) raw.shi = load_scales<FMT>(srow + hi_row * scale_pitch(FMT, STEPS) + (FMT == FMT_MXFP8 ? sc_hi : 0));
  }
}

// A tile is finished when every output's sums over the eight consumer warps have been added, in a fixed tree, multiplied by
// the row's scale and rounded once to the output type. In units of 32 columns x four activation rows, one warp each; unit u:
// columns 32 (u % 2) + lane (SwiGLU tiles have no more than 32), activation rows from 4 (u / 2) (SwiGLU: 4 u) on.
__device__ __forceinline__ int finish_units(const Params& p, const Walk& wk) { return (p.M + 3) / 4 * (wk.pairs ? 1 : 2); }
__device__ __forceinline__ int unit_column(const Walk& wk, int u) { return (threadIdx.x & 31) + (wk.pairs ? 0 : 32 * (u & 1)); }
// (Behind the wait for the previous kernel, as it is written: a load that the compiler places cost the resident kernels up to 5 %,
// 28672 x 8192 NVFP4 with four rows 35.6 and 34.8 us.)
__device__ __forceinline__ float load_f32(const float* at) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(at));
  return v;
}
// Scale of the lane's column (SwiGLU: of its gate and up row).
__device__ __forceinline__ void finish_scales(const Params& p, const Walk& wk, int col0, int cols, int u, float (&f)[2]) {
  const int c = unit_column(wk, u);
  f[0] = f[1] = 1.f;
  if (p.row_scale && c < cols) {
    f[0] = load_f32(p.row_scale + col0 + c);
    if (wk.pairs) f[1] = load_f32(p.row_scale + wk.pairs + col0 + c);
  }
}
template <int FMT, int STEPS>
__device__ __forceinline__ void finish_unit(const Params& p, const Walk& wk, uint32_t stage, int col0, int cols, int u,
                                            const float (&f)[2]) {
  constexpr int W_ROW = weight_pitch(FMT, STEPS), CHUNK = Fragment<FMT>::CHUNK;
  const int c = unit_column(wk, u), m = wk.pairs ? 4 * u : u / 2 * 4, M = p.M;
  if (c >= cols) return;
  auto sums = [&](int r, float scale, float (&v)[4]) {
    float a[kConsumers][4];
#pragma unroll
    for (int w = 0; w < kConsumers; ++w) {
      const uint4 q = lds128(stage + (uint32_t)(r * W_ROW + w * CHUNK + m * 4));
      a[w][0] = __uint_as_float(q.x); a[w][1] = __uint_as_float(q.y); a[w][2] = __uint_as_float(q.z); a[w][3] = __uint_as_float(q.w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = (((a[0][i] + a[1][i]) + (a[2][i] + a[3][i])) + ((a[4][i] + a[5][i]) + (a[6][i] + a[7][i]))) * scale;
  };
  float v[4];
  sums(c, f[0], v);
  if constexpr (FMT == FMT_NVFP4) {
    if (wk.pairs) {
      float up[4];
      sums(wk.cap + c, f[1], up);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = swiglu_value(v[i], up[i]);
    }
  }
  const size_t at = (p.world < 1 ? 0 : (size_t)p.rank * M * p.ldo) + (size_t)m * p.ldo + col0 + c;
  auto store = [&](auto kind) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (m + i < M) store_out(p.out, decltype(kind)::value, at + (size_t)i * p.ldo, v[i]);
  };
  if (p.out_kind == OUT_F32) store(std::integral_constant<int, OUT_F32>());
  else if (p.out_kind == OUT_BF16) store(std::integral_constant<int, OUT_BF16>());
  else store(std::integral_constant<int, OUT_F16>());
}

enum : int { RES_NONE = 0, RES_USUAL = 1, RES_MIXED = 2 };
// Where chunks with values outside the usual window are multiplied: nowhere (there are none); resident ones by the usual chunks' code,
// which then has the columns' powers of two in registers; those that come in windows in code of its own (with the powers
// in registers for every chunk, 28672 x 8192 NVFP4 with 8 rows took 38.4 us, without 37.4, a batched pass over 32 GEMVs at one row
// 849, without 831; but the code of its own is one more thing to fetch, which a launch for few rows pays for with a single such
// chunk: 4096 x 4096, one row, resident, 7.1 and 6.4 us).
// NVFP4 28672 x 8192 at 1 / 8 / 16 rows, us: N(0, 1) activations 31.1 / 37.6 / 53.4, one value of 300 in each row 33.2 / 38.5 /
// 54.3, all above 2^8 36.5 / 45.0 / 67.3, chunks over more than 32 binades 56.6 / 64.9 / 80.8. (As passes after the tile, from global
// memory, they took 68 / 72 / 117, 320 / 316 / 645 and 949 / 1087 / 2158.)
enum : int { ODD_NONE = 0, ODD_SHARED = 1, ODD_APART = 2 };
// One tile of up to 8 EIGHTS rows: the windows in turn; at the end the warp leaves its sums in the stage it has just consumed,
// in its own chunk of each row (which no other warp reads), one FP32 per activation row, and tells the finishing warps, to
// which the stage then belongs (the last tile: the consumers finish it, a unit each, when all have come so far). RES: the
// activations are resident (RES_MIXED: `spread` has the steps, modulo 32, with chunks of another exponent than the usual one). FRESH:
// the lane's places are worked out anew for every tile. Otherwise the compiler works out once what a kernel's tile codes share and
// keeps it all the time, which costs registers: the NVFP4 kernel for resident activations and two steps spilled 84 bytes a thread, and
// none so (us without and with: 8192 x 8192, one row 10.8 and 10.55, 4096 x 4096 5.04 and 4.84, 5920 x 4096 5.73 and 5.70). The others spill
// less, and some are slower so: one step, 8567 x 17728, two rows 24.6 and 27.0; FP16 in windows, 8567 x 17728, 8 rows 22.8 and 24.5.
template <int FMT, int NT, int EIGHTS, int STEPS, typename XT, int RES, bool FRESH>
__device__ __forceinline__ void consume_tile(const Params& p, const Walk& wk, const StageLayout<FMT, STEPS>& lay,
                                             unsigned char* smem, int col0, int cols, bool last, uint32_t spread, const Bars& bars, int& s, uint32_t& parity,
                                             bool first_window, bool& ok) {
  constexpr int SCB = Format<FMT>::SCB, STEP = Format<FMT>::STEP, XROW = Format<FMT>::XROW, WIN = STEPS * STEP;
  constexpr int NB = Fragment<FMT>::NB, CHUNK = Fragment<FMT>::CHUNK, W_ROW = weight_pitch(FMT, STEPS), SC_ROW = scale_pitch(FMT, STEPS);
  constexpr int G = (EIGHTS + 1) / 2;
  constexpr bool ODD = EIGHTS % 2 != 0;       // the last group has no second half
  // BF16 activations of the formats whose weights become FP16
  constexpr bool CONVERT = FMT != FMT_BF16 && std::is_same<XT, __nv_bfloat16>::value;
  constexpr int ODDITIES = !CONVERT || RES == RES_USUAL ? ODD_NONE : RES == RES_MIXED ? ODD_SHARED : ODD_APART;
  Lane ln;
  if constexpr (FRESH) asm volatile("" : "+r"(ln.g), "+r"(ln.t), "+r"(ln.warp));
  const int M = p.M, stage_bytes = p.stage_bytes, stages = p.stages;
  if (last && p.row_scale && unit_column(wk, ln.warp) < cols) {    // (needed at the tile's end)
    const float* at = p.row_scale + col0 + unit_column(wk, ln.warp);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
    if (wk.pairs) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + wk.pairs));
  }
  const uint32_t ring = smem_addr(smem) + kSmemHeader;
  const int frow = fragment_row<FMT>(ln.g);
  // this lane's places in a stage: weights, scales, activations (or among the resident ones)
  const uint32_t w_off = (uint32_t)(frow * W_ROW + ln.warp * CHUNK);
  uint32_t sc_off = (uint32_t)(lay.sc_off + frow * SC_ROW + (FMT == FMT_NVFP4 ? ln.warp * 8 + ln.t * 2 : ln.warp * 2));
  int sc_hi = 0;
  if (scale_granules<FMT>(p)) {
    const uint32_t shift = scale_shift(p, col0 + frow);
    sc_off += shift;
    if (FMT == FMT_MXFP8) sc_hi = (int)scale_shift(p, col0 + frow + 8) - (int)shift;
  }
  const XOffsets<FMT, NT, RES != RES_NONE> xo(ln, M);
  uint32_t res = smem_addr(smem) + (uint32_t)p.x_res_off;    // of the next step
  const uint32_t x_step = (uint32_t)(M * XROW);
  pk2 acc[G][NT][2];
#pragma unroll
  for (int r = 0; r < G; ++r)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[r][nt][0] = acc[r][nt][1] = pack2(0.f, 0.f);

  for (int win = 0, left = p.row_bytes;; ++win) {
    // (after a wait that ran out the warp goes on without waiting: what it then reads and writes is not used)
    ok &= mbar_wait(bars.full + 8u * s, parity, bars.abort_flag);
    if (first_window && win == 0 && threadIdx.x == 0) trace_stamp(p.trace, TRACE_FIRST_FULL);
    const uint32_t stage = ring + (uint32_t)s * stage_bytes;
    // (not unrolled: the steps' code, twice, would not stay in the instruction caches)
#pragma unroll 1
    for (int st = 0; st < STEPS && left > st * STEP; ++st) {
      const uint32_t wrow = stage + w_off + st * STEP, srow = stage + sc_off + st * SCB;
      uint32_t b[NT][NB];
      const uint32_t xs = (RES ? res : stage + lay.x_off) + st * x_step;
      load_x<FMT, NT, RES != RES_NONE>(xs, xo, b);
      RawRows<FMT> raw[2];
      pk2 unscale[NT] = {};
      auto first_rows = [&] { load_rows<FMT, STEPS, ODD && G == 1>(raw[0], wrow, srow, 8, sc_hi, ln.t); };
      // the groups' products in turn: the next group's rows are loaded while one's are multiplied
      auto multiply = [&](auto acts) {
        constexpr int ACTS = decltype(acts)::value;
#pragma unroll
        for (int r = 0; r < G; ++r) {
          constexpr int kRow = kGroupRows;
          const int cur = r & 1;
          if (r + 2 < G || (r + 2 == G && !ODD))
            load_rows<FMT, STEPS, false>(raw[cur ^ 1], wrow + (r + 1) * kRow * W_ROW, srow + (r + 1) * kRow * SC_ROW, 8, sc_hi, ln.t);
          else if (r + 2 == G)
            load_rows<FMT, STEPS, true>(raw[cur ^ 1], wrow + (r + 1) * kRow * W_ROW, srow + (r + 1) * kRow * SC_ROW, 8, sc_hi, ln.t);
          if (ODD && r == G - 1) chunk_rows<FMT, NT, ACTS, true>(raw[cur], b, unscale, acc[r]);
          else chunk_rows<FMT, NT, ACTS, false>(raw[cur], b, unscale, acc[r]);
        }
      };
      // The same for columns that stay BF16, rolled: its registers and its instructions would be taken from the other chunks (five
      // rows, 28672 x 8192 NVFP4, N(0, 1) activations: 38.7 us unrolled, 36.5 rolled; chunks that stay BF16 56 and 64). An odd
      // tile's last group has its lower rows twice.
      auto multiply_wide = [&] {
#pragma unroll 1
        for (int r = 0; r < G; ++r) {
          pk2 sum[NT][2];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) sum[nt][0] = sum[nt][1] = pack2(0.f, 0.f);
          const bool half = ODD && r == G - 1;
          load_rows<FMT, STEPS, false>(raw[0], wrow + r * kGroupRows * W_ROW, srow + r * kGroupRows * SC_ROW, half ? 0 : 8, half ? 0 : sc_hi, ln.t);
          chunk_rows<FMT, NT, ACTS_WIDE, false>(raw[0], b, unscale, sum);
#pragma unroll
          for (int i = 0; i < G; ++i)
            if (i == r) {
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                acc[i][nt][0] = fadd2(sum[nt][0], acc[i][nt][0]);
                acc[i][nt][1] = fadd2(sum[nt][1], acc[i][nt][1]);
              }
            }
        }
      };
      using Scaled = std::integral_constant<int, ACTS_SCALED>;
      using Usual = std::integral_constant<int, CONVERT ? ACTS_USUAL : ACTS_PLAIN>;
      // of a chunk as stored: has it values outside the usual window (zeros among them)
      auto outside = [&] {
        uint32_t bits = 0u;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int i = 0; i < NB; ++i) bits |= window_bits(b[nt][i]);
        return __any_sync(0xffffffffu, (bits & kOutside) != 0u);
      };
      // columns that stay BF16, or the others
      auto keep = [&](const uint32_t (&e)[NT], bool wide) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int i = 0; i < NB; ++i) b[nt][i] = (e[nt] == kWide) == wide ? b[nt][i] : 0u;
      };
      if constexpr (ODDITIES == ODD_SHARED) {
        first_rows();                       // (on their way meanwhile)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) unscale[nt] = pack2(kWindowUnscale, kWindowUnscale);
        const int step = win * STEPS + st;
        if (__builtin_expect((spread >> (step & 31) & 1u) != 0u, 0)) {
          uint32_t e[NT];
          bool any = false, all = true;      // are kWide
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const int steps = (p.row_bytes + STEP - 1) / STEP;
            e[nt] = lds_u8(bars.exps + (uint32_t)((ln.warp * steps + step) * M + min(fragment_column<FMT>(ln.g), M - 1)));
            const uint32_t wide = __ballot_sync(0xffffffffu, e[nt] == kWide);
            any |= wide != 0u;
            all &= wide == 0xffffffffu;
          }
          if (any) {
            keep(e, true);
            multiply_wide();
            if (all) continue;
            load_x<FMT, NT, true>(xs, xo, b);
            first_rows();
            keep(e, false);
          }
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) unscale[nt] = column_unscale(e[nt], ln);
        }
        multiply(Scaled());
      } else {
        if constexpr (ODDITIES == ODD_APART) {
          if (__builtin_expect(outside(), 0)) {
            uint32_t e[NT];
            bool odd = false, any = false, all = true;       // not the usual exponent; are kWide
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              e[nt] = chunk_exp(chunk_range<NB>(b[nt]));
              odd |= e[nt] != kWindowExp;
            }
            if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                const uint32_t wide = __ballot_sync(0xffffffffu, e[nt] == kWide);
                any |= wide != 0u;
                all &= wide == 0xffffffffu;
              }
              if (any) {
                keep(e, true);
                multiply_wide();
                if (all) continue;
                load_x<FMT, NT, false>(xs, xo, b);           // (registers for both would be taken from every chunk)
              }
              first_rows();
              keep(e, false);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                unscale[nt] = column_unscale(e[nt], ln);
                const float scale = exp_scale(e[nt] == kWide ? kWindowExp : e[nt]);
#pragma unroll
                for (int i = 0; i < NB; ++i) b[nt][i] = scaled_half2(b[nt][i], scale);
              }
              multiply(Scaled());
              continue;
            }
          }
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < NB; ++i) b[nt][i] = scaled_half2(b[nt][i], kWindowScale);
        }
        first_rows();
        multiply(Usual());
      }
    }
    left -= WIN;
    if (RES) res += STEPS * x_step;
    __syncwarp();
    if (left <= 0) break;
    if ((threadIdx.x & 31) == 0) mbar_arrive(bars.empty + 8u * s);
    if (++s == stages) { s = 0; parity ^= 1u; }
  }
  float scales[2];
  if (last) finish_scales(p, wk, col0, cols, ln.warp, scales);
  const uint32_t at = ring + (uint32_t)s * stage_bytes + w_off;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    // the fragments' columns 2 t and 2 t + 1
    const int m0 = 8 * nt + fragment_column<FMT>(2 * ln.t), m1 = 8 * nt + fragment_column<FMT>(2 * ln.t + 1);
#pragma unroll
    for (int r = 0; r < G; ++r)
#pragma unroll
      for (int half = 0; half < (ODD && r == G - 1 ? 1 : 2); ++half) {
        float a, c;
        unpack2(acc[r][nt][half], a, c);
        const uint32_t row = at + (uint32_t)((r * kGroupRows + half * 8) * W_ROW);
        if (m0 < M) sts_f32(row + m0 * 4, a);
        if (m1 < M) sts_f32(row + m1 * 4, c);
      }
  }
  if (last) {
    consumer_barrier();
    if (ln.warp < finish_units(p, wk)) finish_unit<FMT, STEPS>(p, wk, ring + (uint32_t)s * stage_bytes, col0, cols, ln.warp, scales);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the stage's next contents come by bulk copies
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive((last ? bars.empty : bars.sums) + 8u * s);
  if (++s == stages) { s = 0; parity ^= 1u; }
}

// The consumer warps' walk over one GEMV, tile by tile. The ring position (s, parity) carries over from one GEMV of a
// batch to the next; `first`: the kernel's first GEMV.
template <int FMT, int NT, bool CAN_RES, int STEPS, bool SMALL, bool BATCH, typename XT>
__device__ __forceinline__ bool consume_gemv(const Params& p, unsigned char* smem, const Bars& bars,
                                             int& s, uint32_t& parity, uint32_t& x_parity, bool first) {
  const Walk wk(p, STEPS * Format<FMT>::STEP);
  const StageLayout<FMT, STEPS> lay(p);
  if (first) griddep_wait();   // consumers read scales and write results in global memory: after the previous kernel
  bool resident = CAN_RES;        // (a launch of its own for up to four rows whose activations come in windows has the kernel for five to eight)
  uint32_t spread = 0u;           // (see prepare_resident)
  bool ok = true;
  if (first && threadIdx.x == 0) trace_stamp(p.trace, TRACE_DEP);
  if constexpr (CAN_RES) {
    if constexpr (BATCH) resident = p.x_mode == X_RESIDENT;
    if (resident && wk.ntiles > 0) {
      ok = mbar_wait(bars.x, x_parity, bars.abort_flag);
      x_parity ^= 1u;
      if constexpr (std::is_same<XT, __nv_bfloat16>::value) spread = prepare_resident<FMT>(p, smem, bars.exps);
      __syncwarp();
    }
  }
  for (int t = 0; t < wk.ntiles; ++t) {
    int col0, cols;
    wk.tile(t, col0, cols);
    auto tile = [&](auto res) {
      constexpr int RES = decltype(res)::value;
      auto run = [&](auto e) {
        consume_tile<FMT, NT, decltype(e)::value, STEPS, XT, RES, FMT == FMT_NVFP4 && CAN_RES && STEPS == 2 && !SMALL && !BATCH>(p, wk, lay, smem, col0, cols, t + 1 == wk.ntiles, spread, bars, s, parity,
                                                                  first && t == 0, ok);
      };
      const int eights = (wk.rows(cols) + 7) / 8;
      if constexpr (!SMALL) {
        if (eights == 8) return run(std::integral_constant<int, 8>());
        if (eights == 7) return run(std::integral_constant<int, 7>());
        if (eights == 6) return run(std::integral_constant<int, 6>());
        if (eights == 5) return run(std::integral_constant<int, 5>());
      }
      if (eights >= 4) return run(std::integral_constant<int, 4>());
      if (eights == 3) return run(std::integral_constant<int, 3>());
      if (eights == 2) return run(std::integral_constant<int, 2>());
      run(std::integral_constant<int, 1>());
    };
    if constexpr (CAN_RES) {
      // (the usual case in code of its own: what a launch fetches of the other costs it 0.6 us)
      if (resident && spread == 0u) tile(std::integral_constant<int, RES_USUAL>());
      else if (resident && std::is_same<XT, __nv_bfloat16>::value) tile(std::integral_constant<int, RES_MIXED>());
      else if constexpr (BATCH) tile(std::integral_constant<int, RES_NONE>());
    } else {
      tile(std::integral_constant<int, RES_NONE>());
    }
  }
  if (!ok && (threadIdx.x & 31) == 0 && p.status) atomicOr(p.status, kStatusConsumerTimeout);
  return ok;
}

// The finishing warps' walk over one GEMV: every tile but the last, which the consumers finish themselves. They are at the
// next tile's windows meanwhile (with the consumers finishing every tile between two barriers a tile of 64 rows took 0.6 us
// longer). `team`: how many warps finish; `sums_parity`: a phase bit per stage.
template <int FMT, int STEPS>
__device__ __forceinline__ bool finish_gemv(const Params& p, unsigned char* smem, const Bars& bars, int worker, int team, int& s,
                                            uint32_t& sums_parity) {
  const Walk wk(p, STEPS * Format<FMT>::STEP);
  const int lane = threadIdx.x & 31, stages = p.stages, skip = wk.nwin % stages;
  // of the eight arrivals that a stage's return takes
  const int arrivals = kConsumers / team + (worker < kConsumers % team ? 1 : 0);
  for (int t = 0; t < wk.ntiles; ++t) {
    int col0, cols;
    wk.tile(t, col0, cols);
    s += skip - 1;                 // the tile's last window
    if (s < 0) s += stages;
    if (s >= stages) s -= stages;
    if (t + 1 < wk.ntiles) {
      if (!mbar_wait(bars.sums + 8u * s, sums_parity >> s & 1u, bars.abort_flag)) {
        if (lane == 0 && p.status) atomicOr(p.status, kStatusConsumerTimeout);
        return false;
      }
      const uint32_t stage = smem_addr(smem) + kSmemHeader + (uint32_t)s * p.stage_bytes;
      for (int u = worker; u < finish_units(p, wk); u += team) {
        float f[2];
        finish_scales(p, wk, col0, cols, u, f);
        finish_unit<FMT, STEPS>(p, wk, stage, col0, cols, u, f);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the stage's next contents come by bulk copies
      __syncwarp();
      if (lane == 0) mbar_arrive_count(bars.empty + 8u * s, arrivals);
      sums_parity ^= 1u << s;
    }
    if (++s == stages) s = 0;
  }
  return true;
}

// All-gather epilogue: all rows of the CTA have been written (every warp but the feeding one).
__device__ __forceinline__ void finished_barrier() { asm volatile("bar.sync 3, %0;" ::"r"(blockDim.x - 32) : "memory"); }

// All-gather epilogue, first half: the CTA's rows [lo, hi) of this rank's slot are complete in the local buffer; all
// consumer threads copy them into the same place of every other rank's buffer: 16 bytes per store where the rows'
// addresses allow it (every rank's buffer has the layout and alignment of this one), else element by element.
__device__ __forceinline__ void gather_copy(const Params& p) {
  const int tid = threadIdx.x, M = p.M;                       // consumer threads are 0 .. 255
  finished_barrier();
  if (p.world < 2) return;
  const int lo = first_column(p, blockIdx.x), rows = first_column(p, blockIdx.x + 1) - lo;
  const int esize = p.out_kind == OUT_F32 ? 4 : 2;
  const size_t slot0 = (size_t)p.rank * M * p.ldo + lo;
  bool vector = true;                                // all buffers equally placed within 16 bytes
  for (int q = 0; q < p.world; ++q)
    vector &= ((reinterpret_cast<uintptr_t>(p.peer_out[q]) ^ reinterpret_cast<uintptr_t>(p.out)) & 15) == 0;
  // warp w copies activation rows w, w + 8, ...; its lanes run along the CTA's rows (consecutive addresses)
  const int lane = tid & 31, warp = tid >> 5;
  for (int m = warp; m < M; m += kConsumers) {
    const size_t byte0 = (slot0 + (size_t)m * p.ldo) * esize;
    const unsigned char* src = reinterpret_cast<const unsigned char*>(p.out) + byte0;
    const int bytes = rows * esize;
    // head up to the next 16-byte boundary, 16-byte body, tail
    const int head = vector ? min(bytes, (int)((16 - (reinterpret_cast<uintptr_t>(src) & 15)) & 15)) : bytes;
    const int body = (bytes - head) >> 4;
    for (int i = lane * esize; i < head; i += 32 * esize) {
      if (esize == 4) {
        const uint32_t v = *reinterpret_cast<const uint32_t*>(src + i);
        for (int q = 0; q < p.world; ++q)
          if (q != p.rank) *reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(p.peer_out[q]) + byte0 + i) = v;
      } else {
        const uint16_t v = *reinterpret_cast<const uint16_t*>(src + i);
        for (int q = 0; q < p.world; ++q)
          if (q != p.rank) *reinterpret_cast<uint16_t*>(static_cast<unsigned char*>(p.peer_out[q]) + byte0 + i) = v;
      }
    }
    for (int i = lane; i < body; i += 32) {
      const uint4 v = *reinterpret_cast<const uint4*>(src + head + 16 * i);
      for (int q = 0; q < p.world; ++q)
        if (q != p.rank)
          *reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.peer_out[q]) + byte0 + head + 16 * i) = v;
    }
    for (int i = head + 16 * body + lane * esize; i < bytes; i += 32 * esize) {
      if (esize == 4) {
        const uint32_t v = *reinterpret_cast<const uint32_t*>(src + i);
        for (int q = 0; q < p.world; ++q)
          if (q != p.rank) *reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(p.peer_out[q]) + byte0 + i) = v;
      } else {
        const uint16_t v = *reinterpret_cast<const uint16_t*>(src + i);
        for (int q = 0; q < p.world; ++q)
          if (q != p.rank) *reinterpret_cast<uint16_t*>(static_cast<unsigned char*>(p.peer_out[q]) + byte0 + i) = v;
      }
    }
  }
}

// Second half: one thread publishes the CTA's copies and counts the CTA done; the rank's last CTA sends `arrivals`
// arrivals to every rank (one per gathered GEMV) and waits, bounded, until its own counter holds arrivals x world.
__device__ __forceinline__ void gather_signal(const Params& p, volatile int* abort_flag, unsigned int arrivals) {
  asm volatile("bar.sync 1, %0;" ::"n"(kConsumers * 32) : "memory");
  if (threadIdx.x != 0) return;
  // System-scope operations cost about a microsecond each and this is the kernel's tail, so the chain is kept short:
  // fence (the CTA's peer copies), one acquire-release count per CTA, then the last CTA fences once and sends one
  // relaxed arrival per rank.
  unsigned int* mine = p.peer_flag[p.rank];
  if (p.world > 1) __threadfence_system();           // the CTA's copies, before it counts as done
  unsigned int before;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(mine + 2) : "memory");
  if (before != gridDim.x - 1) return;
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(mine + 2), "r"(0u) : "memory");   // re-arm the CTA count
  // One system-scope fence orders every CTA's copies (observed through the count) before the arrivals; the
  // arrivals themselves are relaxed, so that they leave back to back (a release per arrival serialised eight
  // round trips on eight GPUs).
  __threadfence_system();
  for (int q = 0; q < p.world; ++q)
    asm volatile("red.relaxed.sys.global.add.u32 [%0], %1;" ::"l"(p.peer_flag[q] + p.gather_slot), "r"(arrivals)
                 : "memory");
  if (p.gather_nowait) return;
  const unsigned int want = (unsigned int)p.world * arrivals;
  const unsigned long long start = global_ns();
  bool done = false;
  for (unsigned int i = 1; !done; ++i) {
    unsigned int seen;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(mine + p.gather_slot) : "memory");
    done = seen >= want;
    if (!done && (i & 63u) == 0u && (*abort_flag || global_ns() - start > p.wait_limit_ns)) break;
  }
  if (done)
    asm volatile("red.relaxed.sys.global.add.u32 [%0], %1;" ::"l"(mine + p.gather_slot), "r"(0u - want) : "memory");
  else if (p.status)
    atomicOr(p.status, kStatusGatherTimeout);
}

// Barriers and the abort word of a CTA; the first thread sets them up. `copies`: the copying warps take part.
__device__ __forceinline__ Bars ring_setup(const Params& p, bool copies, unsigned char* smem, uint64_t* sums, const uint8_t* exps) {
  Bars bars;
  bars.exps = smem_addr(exps);
  bars.x = smem_addr(sums + kMaxStages);
  bars.full = smem_addr(smem);
  bars.empty = bars.full + 8u * kMaxStages;
  bars.sums = smem_addr(sums);
  bars.abort_flag = reinterpret_cast<volatile int*>(smem + 2 * kMaxStages * 8);
  if (threadIdx.x == 0) {
    if (p.trace) {
      unsigned int sm;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
      p.trace[(size_t)blockIdx.x * kTraceSlots + TRACE_SM] = sm;
      trace_stamp(p.trace, TRACE_ENTRY);
    }
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(bars.full + 8u * s, 1 + (copies ? 32 * kCopyWarps : 0));   // the expect_tx arrival + the copying lanes'
                                                                           // cp.async arrivals
      mbar_init(bars.empty + 8u * s, kConsumers);
      mbar_init(bars.sums + 8u * s, kConsumers);
    }
    mbar_init(bars.x, 1);
    *bars.abort_flag = 0;
    *reinterpret_cast<volatile unsigned long long*>(bars.abort_flag + 2) = p.wait_limit_ns;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  griddep_launch_dependents();
  return bars;
}

// NT: column tiles of 8 activation rows; CAN_RES: the launch keeps the activations resident (resident_capable).
template <int FMT, int NT, bool CAN_RES, int STEPS, bool SMALL, typename XT>
__global__ void __launch_bounds__(SMALL ? kSmallThreads : kThreads, SMALL ? 2 : 1) gemv_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t sums[kMaxStages + 1];   // and the resident activations' barrier
  __shared__ uint8_t exps[CAN_RES ? kResidentExps : 1];
  const bool copies = !SMALL && copies_needed<FMT, CAN_RES>(p);
  const Bars bars = ring_setup(p, copies, smem, sums, exps);
  int s = 0;
  uint32_t parity = 0, x_parity = 0;
  const int warp = (int)(threadIdx.x >> 5);
  if (warp == kFeeder) {
    if (!p.early_weights) {
      prefetch_weights<FMT, STEPS>(p);
    }
    feed_weights<FMT, STEPS, CAN_RES>(p, p, smem, bars, true, !p.early_weights, s, parity);
  } else if (!SMALL && warp >= kFirstCopier && copies) {
    griddep_wait();
    feed_activations<FMT, STEPS, CAN_RES>(p, smem, bars, warp - kFirstCopier, s, parity);
    if (p.world >= 1) finished_barrier();
  } else if (warp >= kFinisher) {
    // (reads scales and writes results in global memory: after the previous kernel)
    if (warp == kFinisher) start_activations<FMT, STEPS, CAN_RES>(p, p, smem, bars);
    else griddep_wait();
    if (!SMALL) finish_gemv<FMT, STEPS>(p, smem, bars, warp - kFinisher, copies ? 1 : kFinishers, s, parity);
    if (p.world >= 1) finished_barrier();
  } else {
    consume_gemv<FMT, NT, CAN_RES, STEPS, SMALL, false, XT>(p, smem, bars, s, parity, x_parity, true);
    if ((threadIdx.x & 31) == 0) trace_stamp(p.trace, TRACE_LAST_CONSUMED);
    if (p.world >= 1) {
      gather_copy(p);
      gather_signal(p, bars.abort_flag, 1u);
    }
  }
  if ((threadIdx.x & 31) == 0) trace_stamp(p.trace, TRACE_EXIT);
  // A wait that ran out leaves copies in flight towards this CTA's shared memory: let them land before the CTA's
  // memory is handed to the next one (bounded sleep, error path only).
  if (*bars.abort_flag) {
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
}

// Several independent GEMVs of one format and row count in one launch: `items` (device memory) are their launch
// parameters, all with the same ring shape (stages, stage bytes). Every CTA walks the GEMVs in order and the ring never
// drains between them: the copies of the next GEMV's weights are in flight while the last tiles of this one are
// consumed, which a sequence of launches cannot do (a CTA that holds the SM's shared memory must leave before the
// next kernel's CTA can come). With the all-gather epilogue each CTA sends a GEMV's rows to the peers as soon as it has
// finished them and goes on; the arrivals of all GEMVs are exchanged once, at the end. For GEMVs whose inputs do not
// depend on each other's outputs only (all activations are read after one wait for the previous kernel).
template <int FMT, int NT, bool CAN_RES, int STEPS, typename XT>
__global__ void __launch_bounds__(kThreads, 1) gemv_batch_kernel(const Params* __restrict__ items, int count) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t sums[kMaxStages + 1];   // and the resident activations' barrier
  __shared__ uint8_t exps[CAN_RES ? kResidentExps : 1];
  const bool copies = items[0].batch_copies != 0;
  const Bars bars = ring_setup(items[0], copies, smem, sums, exps);
  int s = 0;
  uint32_t parity = 0, x_parity = 0;
  const int warp = (int)(threadIdx.x >> 5);
  if (warp == kFeeder) {
    bool ok = true;
    for (int g = 0; g < count && ok; ++g)
      ok = feed_weights<FMT, STEPS, false>(items[g], items[g], smem, bars, g == 0, g == 0 && !items[0].early_weights, s, parity);
  } else if (warp >= kFinisher && !(copies && warp >= kFirstCopier)) {
    if (warp == kFinisher) start_activations<FMT, STEPS, false>(items[0], items[0], smem, bars);
    else griddep_wait();
    bool ok = true;
    for (int g = 0; g < count; ++g) {
      if (ok) ok = finish_gemv<FMT, STEPS>(items[g], smem, bars, warp - kFinisher, copies ? 1 : kFinishers, s, parity);
      if (items[g].world >= 1) finished_barrier();
    }
  } else if (warp >= kFirstCopier) {
    griddep_wait();
    bool ok = true;
    for (int g = 0; g < count; ++g) {
      if (ok) ok = feed_activations<FMT, STEPS, false>(items[g], smem, bars, warp - kFirstCopier, s, parity);
      if (items[g].world >= 1) finished_barrier();
    }
  } else {
    // (every warp passes every GEMV's barriers, also after a wait that ran out)
    for (int g = 0; g < count; ++g) {
      consume_gemv<FMT, NT, CAN_RES, STEPS, false, true, XT>(items[g], smem, bars, s, parity, x_parity, g == 0);
      if (items[g].world >= 1) gather_copy(items[g]);   // the CTA's rows of this GEMV go to the peers now
    }
    if ((threadIdx.x & 31) == 0) trace_stamp(items[0].trace, TRACE_LAST_CONSUMED);
    if (items[0].world >= 1) gather_signal(items[0], bars.abort_flag, (unsigned int)count);
  }
  if ((threadIdx.x & 31) == 0) trace_stamp(items[0].trace, TRACE_EXIT);
  // A wait that ran out leaves copies in flight towards this CTA's shared memory: let them land before the CTA's
  // memory is handed to the next one (bounded sleep, error path only).
  if (*bars.abort_flag) {
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
}

}  // namespace dg
