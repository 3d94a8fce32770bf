// Activation quantizers for B200 (sm_100a): BF16 rows to FP8 E4M3 with one scale per row, and to NVFP4 (E2M1 codes,
// one E4M3 scale per 16 values, scales in cuBLASLt's 128 x 4 tiled layout). The step just before a W8A8 / W4A4
// projection; they replace the reference's quantize_fp8_rows and quantize_nvfp4 (mma-rows/mma_rows_cuda/
// mma_rows.cu:15-140 kernels, :320-340 entry points; arithmetic in tile_parts.cuh:23-64, :301-331) bit for bit:
//
//   FP8 rows   scale = max(amax * fp32(1 / 448), 1e-12); q = E4M3(clamp(x / scale, +-448)), IEEE division, round to
//              nearest even. A NaN in a row makes its scale NaN (torch's amax).
//   NVFP4      per 16 values: s = E4M3(min((amax * fp32(1 / 6)) * g, 448)); d = max(e4m3(s) * (1 / g), 1e-30);
//              code = E2M1(x / d), nearest with ties to the even code, magnitudes above 6 to 6, the sign bit set for
//              every negative quotient, all codes 0 where e4m3(s) is not > 0.
//
// Machine mapping (not the reference's): a row of the FP8 quantizer is read from HBM once: one bulk copy (TMA, 1-D)
// brings it into shared memory, the CTA takes the maximum and quantizes from there, 16 output bytes per thread and
// store; rows that do not fit or are not 16-byte aligned are read twice through L2 instead. The NVFP4 quantizer gives a
// lane a block and converts with the hardware E2M1 / E4M3 conversions.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/decode_gemv_b200.h"

namespace {

constexpr float kRcp448 = 1.0f / 448.0f;   // a division by a constant is a product with its FP32 reciprocal in the
constexpr float kRcp6 = 1.0f / 6.0f;       // framework whose quantizers these reproduce
constexpr int kRowThreads = 256;
constexpr int kRowSmemLimit = 200 * 1024;
constexpr unsigned long long kCopyWaitNs = 2000000000ull;

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
// The larger of two values, NaN if either is (one instruction; BF16 pairs keep the maximum exactly).
__device__ __forceinline__ float nanmax(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint32_t amax2(uint32_t pair, uint32_t m) {   // per half: max(|pair|, m), NaN kept
  uint32_t r;
  asm("{\n\t.reg .b32 a;\n\tabs.bf16x2 a, %1;\n\tmax.NaN.bf16x2 %0, a, %2;\n\t}" : "=r"(r) : "r"(pair), "r"(m));
  return r;
}
__device__ __forceinline__ uint32_t amax8(const uint4& v, uint32_t m) {
  return amax2(v.w, amax2(v.z, amax2(v.y, amax2(v.x, m))));
}
__device__ __forceinline__ float amax_of(uint32_t m) { return nanmax(bf16_lo(m), bf16_hi(m)); }
// Two FP32 -> two E4M3 bytes (low byte = lo), round to nearest even, saturating.
__device__ __forceinline__ uint32_t e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float e4m3_value(uint32_t byte) {
  uint32_t h;
  asm("{\n\t.reg .b16 t;\n\tcvt.u16.u32 t, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, t;\n\t}" : "=r"(h) : "r"(byte & 0xffu));
  return __half2float(__ushort_as_half((unsigned short)(h & 0xffffu)));
}
// The clamp to +-448 that the quantizer's definition names is the saturating conversion's: every quotient beyond
// 448 (at most by a rounding of the scale) converts to 448 either way, NaN to NaN.
//
// x / d, correctly rounded, for many x over one d whose quotients stay within FP32's normal range (SAFE): with
// r = RN(1 / d) computed once, q0 = RN(x r), the exact residual e = x - d q0 (one FMA) and q = RN(q0 + e r) give the
// IEEE quotient (P. Markstein, Computation of elementary functions on the IBM RISC System/6000, 1990). A zero
// quotient keeps its own sign where that matters (KEEP_ZERO: the correction would turn -0 into +0). Quotients too
// small for an exact residual convert to zero whatever their last bits are. Otherwise the full division runs.
template <bool SAFE, bool KEEP_ZERO>
__device__ __forceinline__ float quotient(float x, float d, float r) {
  if constexpr (!SAFE) return __fdiv_rn(x, d);
  const float q0 = __fmul_rn(x, r);
  const float q1 = __fmaf_rn(__fmaf_rn(-d, q0, x), r, q0);
  return KEEP_ZERO && q0 == 0.f ? q0 : q1;
}
template <bool SAFE>
__device__ __forceinline__ uint32_t fp8_quad(uint32_t w0, uint32_t w1, float d, float r) {
  return e4m3x2(quotient<SAFE, true>(bf16_lo(w0), d, r), quotient<SAFE, true>(bf16_hi(w0), d, r)) |
         (e4m3x2(quotient<SAFE, true>(bf16_lo(w1), d, r), quotient<SAFE, true>(bf16_hi(w1), d, r)) << 16);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The second pass over a row: 16 (or 8) values a thread and store where the output allows it.
template <bool SAFE>
__device__ __forceinline__ void quantize_row(const __nv_bfloat16* xr, const uint4* row_smem, uint8_t* qr, int K, float d,
                                             int staged, bool aligned_in, int vector_out, int tid) {
  const float r = SAFE ? __frcp_rn(d) : 0.f;
  if (aligned_in) {
    const uint4* rv = staged ? row_smem : reinterpret_cast<const uint4*>(xr);
    if (vector_out && (K & 15) == 0) {   // 16 values -> one 16-byte store
      for (int i = tid; i < (K >> 4); i += kRowThreads) {
        const uint4 a = rv[2 * i], b = rv[2 * i + 1];
        reinterpret_cast<uint4*>(qr)[i] = make_uint4(fp8_quad<SAFE>(a.x, a.y, d, r), fp8_quad<SAFE>(a.z, a.w, d, r),
                                                     fp8_quad<SAFE>(b.x, b.y, d, r), fp8_quad<SAFE>(b.z, b.w, d, r));
      }
    } else if (vector_out) {             // 8 values -> one 8-byte store
      for (int i = tid; i < (K >> 3); i += kRowThreads) {
        const uint4 a = rv[i];
        reinterpret_cast<uint2*>(qr)[i] = make_uint2(fp8_quad<SAFE>(a.x, a.y, d, r), fp8_quad<SAFE>(a.z, a.w, d, r));
      }
    } else {
      for (int i = tid; i < (K >> 3); i += kRowThreads) {
        const uint4 a = rv[i];
        const uint32_t lo = fp8_quad<SAFE>(a.x, a.y, d, r), hi = fp8_quad<SAFE>(a.z, a.w, d, r);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          qr[8 * i + j] = (uint8_t)(lo >> (8 * j));
          qr[8 * i + 4 + j] = (uint8_t)(hi >> (8 * j));
        }
      }
    }
  } else {
    for (int k = tid; k < K; k += kRowThreads)
      qr[k] = (uint8_t)(e4m3x2(quotient<SAFE, true>(__bfloat162float(xr[k]), d, r), 0.f) & 0xffu);
  }
}

// Rows of up to 4 x 8 values per thread, held in registers between the two passes: `group` threads (a power of two of at
// least 32) to a row, blockDim.x / group rows to a CTA. A row's bytes are read once, all its loads in flight at once, with
// no trip through shared memory. Short rows are what it is for: a CTA and a bulk copy to each are bound by their latency
// (8192 x 1024: 14.5 us, now 6.0; 3.8 at copy bandwidth), and small batches, which a kernel's latency bounds (16 x 28672:
// 3.3 us, now 2.8; 1 x 4096: 1.65, now 1.35). From about 5000 values on in batches that fill the chip the bulk copy is the
// faster way (4096 x 28672: 54 us, at copy bandwidth; 96 here, with one CTA of 1024 threads waiting at its barrier).
constexpr int kHeld = 4;
__global__ void __launch_bounds__(1024) fp8_held_rows_kernel(const __nv_bfloat16* x, long long ldx, int M, int K,
                                                                uint8_t* __restrict__ q, long long ldq, float* __restrict__ scale,
                                                                int group) {
  __shared__ float part[32];
  const int tid = threadIdx.x, t = tid & (group - 1), warp = tid >> 5, warps = group >> 5;
  const int row = blockIdx.x * (blockDim.x / group) + tid / group;
  const bool in = row < M;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // x is the previous kernel's output
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
  uint4 v[kHeld];
  uint32_t m2 = 0u;
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    v[i] = in && t + i * group < (K >> 3) ? xr[t + i * group] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < kHeld; ++i) m2 = amax8(v[i], m2);
  float m = amax_of(m2);
#pragma unroll
  for (int o = 16; o; o >>= 1) m = nanmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (warps > 1) {
    if ((tid & 31) == 0) part[warp] = m;
    __syncthreads();
    const int lane = tid & 31;
    m = part[(warp & ~(warps - 1)) + (lane & (warps - 1))];
#pragma unroll
    for (int o = 16; o; o >>= 1) m = nanmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  if (!in) return;
  float sc = m * kRcp448;
  sc = sc < 1e-12f ? 1e-12f : sc;
  if (t == 0) scale[row] = sc;
  uint2* qr = reinterpret_cast<uint2*>(q + (size_t)row * ldq);
  const float r = sc <= 1e30f ? __frcp_rn(sc) : 0.f;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    if (t + i * group >= (K >> 3)) break;
    const uint4 a = v[i];
    qr[t + i * group] = sc <= 1e30f   // (see below)
                            ? make_uint2(fp8_quad<true>(a.x, a.y, sc, r), fp8_quad<true>(a.z, a.w, sc, r))
                            : make_uint2(fp8_quad<false>(a.x, a.y, sc, r), fp8_quad<false>(a.z, a.w, sc, r));
  }
}

// Other rows, one CTA each. `staged`: the row (K a multiple of 8, 16-byte aligned, within shared memory) arrives by one bulk copy.
__global__ void __launch_bounds__(kRowThreads) fp8_rows_kernel(const __nv_bfloat16* x, long long ldx, int K,
                                                               uint8_t* __restrict__ q, long long ldq,
                                                               float* __restrict__ scale, int staged, int vector_out) {
  extern __shared__ __align__(128) unsigned char row_smem[];
  __shared__ __align__(8) unsigned long long bar;
  __shared__ float part[kRowThreads / 32];
  __shared__ float row_scale;
  __shared__ int failed;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const __nv_bfloat16* xr = x + (size_t)row * ldx;
  uint8_t* qr = q + (size_t)row * ldq;
  const uint32_t bar_addr = (uint32_t)__cvta_generic_to_shared(&bar);
  if (tid == 0) {
    failed = 0;
    if (staged) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_addr) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
  }
  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // x is the previous kernel's output
  float m = 0.f;
  uint32_t m2 = 0u;   // running maximum of BF16 pairs
  if (staged) {
    if (tid == 0) {
      const uint32_t bytes = (uint32_t)K * 2u;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_addr), "r"(bytes) : "memory");
      asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(row_smem)),
                   "l"(xr), "r"(bytes), "r"(bar_addr)
                   : "memory");
    }
    // bounded wait for the copy (it cannot fail on valid arguments; the bound keeps a bad pointer from hanging)
    const unsigned long long start = global_ns();
    uint32_t ok = 0;
    for (uint32_t i = 1; !ok; ++i) {
      asm volatile(
          "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(bar_addr)
          : "memory");
      if (!ok && (i & 255u) == 0u && (failed || global_ns() - start > kCopyWaitNs)) {
        failed = 1;
        break;
      }
    }
    if (!ok) return;
    const uint4* rv = reinterpret_cast<const uint4*>(row_smem);
    for (int i = tid; i < (K >> 3); i += kRowThreads) m2 = amax8(rv[i], m2);
    m = amax_of(m2);
  } else if ((K & 7) == 0 && (ldx & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    const uint4* rv = reinterpret_cast<const uint4*>(xr);
    for (int i = tid; i < (K >> 3); i += kRowThreads) m2 = amax8(rv[i], m2);
    m = amax_of(m2);
  } else {
    for (int k = tid; k < K; k += kRowThreads) m = nanmax(m, fabsf(__bfloat162float(xr[k])));
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) m = nanmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) part[warp] = m;
  __syncthreads();
  if (tid == 0) {
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < kRowThreads / 32; ++w) a = nanmax(a, part[w]);
    const float sc = a * kRcp448;
    row_scale = sc < 1e-12f ? 1e-12f : sc;
    scale[row] = row_scale;
  }
  __syncthreads();
  const float sc = row_scale;
  const bool aligned_in = staged || ((K & 7) == 0 && (ldx & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0);
  // a finite scale bounds every quotient of the row by 448 (1 + a rounding): the short division; NaN or infinite
  // rows take the full one
  if (sc <= 1e30f)
    quantize_row<true>(xr, reinterpret_cast<const uint4*>(row_smem), qr, K, sc, staged, aligned_in, vector_out, tid);
  else
    quantize_row<false>(xr, reinterpret_cast<const uint4*>(row_smem), qr, K, sc, staged, aligned_in, vector_out, tid);
}

// Two quotients -> two E2M1 codes in one byte (low nibble = lo): every negative quotient's sign bit is set, also when it rounds to
// zero, and a negative zero's.
__device__ __forceinline__ uint32_t e2m1x2(float lo, float hi) {
  uint16_t r;
  asm("{\n\t.reg .b8 t;\n\tcvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n\tcvt.u16.u8 %0, t;\n\t}" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}

// Packed FP32 pairs (each half IEEE, round to nearest).
struct pair { unsigned long long v; };
__device__ __forceinline__ pair pack(float lo, float hi) {
  pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ pair mul2(pair a, pair b) {
  pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ pair fma2(pair a, pair b, pair c) {
  pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// A launch has at most 127 scales (an input scale times an E4M3 value each): their d and 1 / d, worked out once per CTA. d = 0: all
// codes are 0 (e4m3(s) is not > 0).
struct Scale { float d, r; };
__device__ __forceinline__ Scale scale_of(uint32_t byte, float g_rcp) {
  float d = e4m3_value(byte) * g_rcp;
  if (!(d > 0.f)) return {0.f, 0.f};
  d = d < 1e-30f ? 1e-30f : d;
  return {d, __frcp_rn(d)};
}

// Codes of 8 BF16 pairs. SHORT: no quotient can leave FP32's range, so they take the short division, two values at once. ZEROS: a
// negative zero quotient becomes +0 first (code 0, as a comparison with zero sees it). The short division does that by
// itself where no quotient underflows: the residual of -0 is +0, and so is its sum with it.
template <bool SHORT, bool ZEROS>
__device__ __forceinline__ void codes16(const uint32_t (&w)[8], const Scale& sc, uint32_t& lo, uint32_t& hi) {
  uint32_t byte[8];
  const pair r2 = pack(sc.r, sc.r), d2 = pack(-sc.d, -sc.d);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float a, b;
    if constexpr (SHORT) {
      const pair x = pack(bf16_lo(w[i]), bf16_hi(w[i])), q0 = mul2(x, r2), q1 = fma2(fma2(d2, q0, x), r2, q0);
      asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(q1.v));
    } else {
      a = __fdiv_rn(bf16_lo(w[i]), sc.d);
      b = __fdiv_rn(bf16_hi(w[i]), sc.d);
    }
    byte[i] = ZEROS ? e2m1x2(a + 0.f, b + 0.f) : e2m1x2(a, b);
  }
  lo = __byte_perm(__byte_perm(byte[0], byte[1], 0x0040), __byte_perm(byte[2], byte[3], 0x0040), 0x5410);
  hi = __byte_perm(__byte_perm(byte[4], byte[5], 0x0040), __byte_perm(byte[6], byte[7], 0x0040), 0x5410);
}

// 16 values (8 BF16 pairs) -> scale byte (returned) and 8 code bytes (lo, hi).
__device__ __forceinline__ uint32_t nvfp4_block(const uint32_t (&w)[8], float g, const Scale* scales, uint32_t& lo, uint32_t& hi) {
  uint32_t m = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = amax2(w[i], m);
  const float amax = amax_of(m);
  float bs = (amax * kRcp6) * g;
  bs = bs > 448.f ? 448.f : bs;
  const uint32_t sbits = e4m3x2(bs, 0.f) & 0xffu;
  const Scale sc = scales[sbits & 0x7fu];
  lo = hi = 0u;
  if (sc.d == 0.f) return sbits;
  // Below 1e8 no quotient leaves FP32's range; BF16's smallest value, 2^-133, over less than 2^17 is not yet rounded to zero.
  if (amax < 1e8f && sc.d < 131072.f) codes16<true, false>(w, sc, lo, hi);
  else if (amax < 1e8f) codes16<true, true>(w, sc, lo, hi);
  else codes16<false, true>(w, sc, lo, hi);
  return sbits;
}

// A CTA quantizes 32 rows x 512 values of a 128-row tile of the scales: warp w the rows 8 i + w, 32 + 8 i + w, 64 + 8 i + w
// and 96 + 8 i + w (i: which quarter), whose scale words lie side by side in the tiled layout. A lane takes one block of a
// row: a warp reads 1024 and writes 256 consecutive bytes at a time, two rows' loads in flight at once, and the scale bytes
// meet in shared memory and leave as 128 consecutive bytes per tile. (With four blocks to a thread a warp's load touched 32
// lines.) The arithmetic bounds it, more than the memory (an integer or conversion instruction takes a scheduler two clocks):
// the quotients are in packed pairs and the scales' reciprocals in a table. 4096 x 8192: 22.3 us with four blocks to a thread, 18.6
// without the table and with a + 0 for every quotient, 17.0 now (13.1 at copy bandwidth, 0.77 of it); 512 x 4096: 4.2 and 3.2; 16 x 28672: 5.0,
// 1.95 and 1.8. Five CTAs per SM (48 registers): 16.3, but 1024 x 8192 7.2 instead of 6.5.
constexpr int kQuantCols = 512, kQuantRows = 32;
__global__ void __launch_bounds__(256) nvfp4_kernel(const __nv_bfloat16* x, long long ldx, int M, int K,
                                                    float g, float g_rcp, uint8_t* __restrict__ codes,
                                                    uint8_t* __restrict__ scales, int quads, int col_tiles, int wide_scales) {
  __shared__ __align__(16) unsigned char tile[kQuantCols / 64 * 128];   // [quad][row % 8][row / 32][block % 4]
  __shared__ Scale known[128];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row_block = blockIdx.x / col_tiles, col_tile = blockIdx.x - row_block * col_tiles;
  const int tile_row = row_block >> 2, eight = row_block & 3;
  const int row0 = tile_row * 128 + eight * 8 + warp, k = col_tile * kQuantCols + lane * 16;
  if (tid < kQuantCols / 64 * 8) reinterpret_cast<uint4*>(tile)[tid] = make_uint4(0u, 0u, 0u, 0u);   // padding rows and blocks
  if (tid >= 128) known[tid - 128] = scale_of((uint32_t)tid - 128u, g_rcp);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint4 v[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + 32 * i;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * ldx + k);
    const bool in = row < M && k < K;
    v[i][0] = in ? src[0] : make_uint4(0u, 0u, 0u, 0u);
    v[i][1] = in ? src[1] : make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + 32 * i;
    if (row < M && k < K) {
      const uint32_t w[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
      uint32_t lo, hi;
      const uint32_t scale = nvfp4_block(w, g, known, lo, hi);
      *reinterpret_cast<uint2*>(codes + (size_t)row * (K >> 1) + (k >> 1)) = make_uint2(lo, hi);
      tile[(lane >> 2) * 128 + warp * 16 + i * 4 + (lane & 3)] = (unsigned char)scale;
    }
  }
  __syncthreads();
  const int quad = col_tile * (kQuantCols / 64) + (tid >> 3);
  if (tid < kQuantCols / 64 * 8 && quad < quads) {
    const uint4 s = reinterpret_cast<const uint4*>(tile)[tid];
    uint8_t* dst = scales + ((size_t)tile_row * quads + quad) * 512 + (eight * 8 + (tid & 7)) * 16;
    if (wide_scales) {
      *reinterpret_cast<uint4*>(dst) = s;
    } else {
      uint32_t* d32 = reinterpret_cast<uint32_t*>(dst);
      d32[0] = s.x; d32[1] = s.y; d32[2] = s.z; d32[3] = s.w;
    }
  }
}

bool aligned(const void* p, uintptr_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }

template <typename... Args>
cudaError_t launch_pdl(void (*kernel)(Args...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&config, kernel, args...);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

extern "C" {

int dg_enqueue_quantize_fp8_rows(const void* x, long long ldx, int M, int K, uint8_t* q, long long ldq, float* scale,
                                 void* stream) {
  if (M < 1 || K < 1 || !x || !q || !scale || ldx < K || ldq < K || !aligned(x, 2) || !aligned(scale, 4))
    return (int)cudaErrorInvalidValue;
  const size_t row_bytes = (size_t)K * 2;
  const int staged = K % 8 == 0 && ldx % 8 == 0 && aligned(x, 16) && row_bytes <= (size_t)kRowSmemLimit;
  const int vector_out = K % 16 == 0 ? (ldq % 16 == 0 && aligned(q, 16)) : (ldq % 8 == 0 && aligned(q, 8));
  if (K % 8 == 0 && (K <= 4096 || (M <= 256 && K <= 1024 * 8 * kHeld)) && ldx % 8 == 0 && aligned(x, 16) && ldq % 8 == 0 && aligned(q, 8)) {
    // threads to a row: enough to hold it; while the batch leaves SMs idle, up to one 16-byte load each
    int group = 32;
    while (group * 8 * kHeld < K || (group * 8 < K && group < 1024 && (long long)M * group < 32 * 1024)) group *= 2;
    const int threads = group < 256 ? 256 : group, rows = threads / group;
    return (int)launch_pdl(fp8_held_rows_kernel, dim3((unsigned)((M + rows - 1) / rows)), dim3(threads), 0,
                           static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x), ldx, M, K, q, ldq, scale,
                           group);
  }
  const size_t smem = staged ? row_bytes : 0;
  if (smem > 48 * 1024) {
    // opt in above the default limit; per device, not a stream operation (costs nothing after the first call)
    static thread_local int opted[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!opted[dev]) {
      const cudaError_t e =
          cudaFuncSetAttribute(fp8_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmemLimit);
      if (e != cudaSuccess) return (int)e;
      opted[dev] = 1;
    }
  }
  return (int)launch_pdl(fp8_rows_kernel, dim3((unsigned)M), dim3(kRowThreads), smem, static_cast<cudaStream_t>(stream),
                         static_cast<const __nv_bfloat16*>(x), ldx, K, q, ldq, scale, staged, vector_out);
}

int dg_enqueue_quantize_nvfp4(const void* x, long long ldx, int M, int K, float input_scale, float input_rcp,
                              uint8_t* codes, uint8_t* blocked_scales, void* stream) {
  if (M < 1 || K < 16 || K % 16 || !x || !codes || !blocked_scales || ldx < K || ldx % 8 || !aligned(x, 16) ||
      !aligned(codes, 8) || !aligned(blocked_scales, 4) || !(input_scale > 0.f))
    return (int)cudaErrorInvalidValue;
  const int quads = (K / 16 + 3) / 4;
  const int col_tiles = (K + kQuantCols - 1) / kQuantCols;
  const long long ctas = ((long long)M + 127) / 128 * (128 / kQuantRows) * col_tiles;
  return (int)launch_pdl(nvfp4_kernel, dim3((unsigned)ctas), dim3(256), 0, static_cast<cudaStream_t>(stream),
                         static_cast<const __nv_bfloat16*>(x), ldx, M, K, input_scale, input_rcp, codes, blocked_scales, quads, col_tiles,
                         (int)aligned(blocked_scales, 16));
}

}  // extern "C"
