// The arithmetic of the decode GEMVs: one consumer warp, one chunk of K, tiles of 16 weight rows times 8 or 16
// activation rows on mma.m16n8k16 with FP32 accumulators.
//
// What bounds it. A call streams its weights once (HBM) and multiplies each by 1..16 activations. On the FMA pipe that
// product is the limit from about 4 rows on (16 rows: one FP32 FMA per 4-bit weight and row takes 202 us where HBM
// takes 40, at 57344 x 8192); on the tensor cores it is not: mma.sync sustains about 1000 multiply-adds per clock and
// SM on a B200, a stream of NVFP4 codes at full HBM rate needs 330 (8 columns) to 660 (16 columns). What is left per
// weight is its decode in registers (one conversion per two E4M3 / E2M1 codes, NVFP4: one packed product with the block
// scale more), the same for every row count. The weights come from shared memory straight into the fragments, so the
// tcgen05 form, which reads its operands from shared or tensor memory, would have to write every decoded 16-bit weight
// back first: 4 bytes of traffic per half byte streamed, for a rate that is not needed.
//
// K order. A chunk is 64 bytes of a weight row (128 for BF16: two pieces of 64). Lane (g, t) = (lane / 4, lane % 4) supplies the weights of rows g and
// g + 8 at bytes 16 t .. 16 t + 15 of the chunk (MXFP8: bytes 8 t .. 8 t + 7 of each 32-byte block) and, as the second
// operand, the activations at the same K of activation row g: the k index inside an mma is only a name, so both sides
// keep their natural order in memory and no shuffles are needed.
//
// Precision. Products of two 16-bit operands are exact. The tensor core adds the 16 products of a step to the
// accumulator with a wider alignment but truncates where an FMA rounds, so the chains are kept short: at most four
// steps (64 products), then rounded FP32 additions into the running sums, of which there are few. Measured against FP64
// the error of a sum is that of chains of FP32 FMAs.
//
// Row invariance. A column of an mma depends on that column's activations alone, and chunks, chains and the order of
// their sums are functions of K and the format. Which of the two ways below a chunk of an activation row goes depends on
// that row's own values in that chunk.
//
// Activations. BF16 weights multiply BF16 activations as they are. Decoded E4M3 and E2M1 x E4M3 weights are FP16 values
// (at most 6 significant bits, 2^-10 .. 2688), so FP16 activations are used as they are too. BF16 activations of these
// formats become FP16 times a power of two, exactly; it comes off in the FP32 FMA. The power is 2^7 for a chunk of a row
// whose magnitudes lie in [2^-24, 2^8) or are zero, the one that fits for any other chunk within 32 binades. A chunk that
// spans more (or holds infinities or NaNs) stays BF16: its products are made with the weights converted to BF16, which is
// exact too and takes about twice as long.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

namespace dg {

// ---------------------------------------------------------------------------------------------------------------
// Shared-memory loads by 32-bit shared-space address. Volatile keeps them behind the barrier waits.
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts_f32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void sts_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts_u8(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Two FP32 values in one 64-bit register pair, the operand form of the packed fma.rn.f32x2 / mul.rn.f32x2.
struct pk2 { unsigned long long v; };
__device__ __forceinline__ pk2 pack2(float lo, float hi) {
  pk2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(pk2 a, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ pk2 ffma2(pk2 a, pk2 b, pk2 c) {   // (a.lo * b.lo + c.lo, a.hi * b.hi + c.hi), each IEEE RN
  pk2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ pk2 fadd2(pk2 a, pk2 b) {
  pk2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ pk2 fmul2(pk2 a, pk2 b) {
  pk2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}

// ---------------------------------------------------------------------------------------------------------------
// Decoding. All exact. The conversions take their packed source from a 16-bit (E4M3 pair) or 8-bit (E2M1 pair)
// register; unpacking the word in PTX lets the assembler select the sub-word instead of shifting it out first.
__device__ __forceinline__ void decode_e4m3_h(uint32_t a, uint32_t b, uint32_t (&h)[4]) {   // 8 E4M3 -> 4 FP16 pairs
  asm("{\n\t.reg .b16 lo, hi;\n\t"
      "mov.b32 {lo, hi}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, lo;\n\t"
      "cvt.rn.f16x2.e4m3x2 %1, hi;\n\t}"
      : "=r"(h[0]), "=r"(h[1]) : "r"(a));
  asm("{\n\t.reg .b16 lo, hi;\n\t"
      "mov.b32 {lo, hi}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, lo;\n\t"
      "cvt.rn.f16x2.e4m3x2 %1, hi;\n\t}"
      : "=r"(h[2]), "=r"(h[3]) : "r"(b));
}
__device__ __forceinline__ void decode_e2m1_h(uint32_t a, uint32_t (&h)[4]) {               // 8 E2M1 -> 4 FP16 pairs
  asm("{\n\t.reg .b8 c0, c1, c2, c3;\n\t"
      "mov.b32 {c0, c1, c2, c3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, c0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, c1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, c2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, c3;\n\t}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]) : "r"(a));
}
__device__ __forceinline__ uint32_t e4m3x2_to_half2(uint32_t v) {   // low 16 bits: two E4M3 -> two FP16
  uint32_t h;
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, lo;\n\t}" : "=r"(h) : "r"(v));
  return h;
}
__device__ __forceinline__ uint32_t mul_half2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// Two E8M0 exponent bytes (low 16 bits) as FP32 2^(e-127), each in both halves of a packed pair; e = 0 is the FP32
// subnormal 2^-127 and e = 255 is NaN, as the reference decodes them (decode_gemv.cu:275-278): BF16 holds all of these.
__device__ __forceinline__ void e8m0x2_to_f32(uint32_t v, pk2& first, pk2& second) {
  uint32_t h;
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tcvt.rn.bf16x2.ue8m0x2 %0, lo;\n\t}" : "=r"(h) : "r"(v));
  const float a = __uint_as_float(h << 16), b = __uint_as_float(h & 0xffff0000u);
  first = pack2(a, a);
  second = pack2(b, b);
}
// ---------------------------------------------------------------------------------------------------------------
// d (+)= A B for one k16 step: a[0], a[2] the lane's two pairs of row g, a[1], a[3] those of row g + 8; b0, b1 its two
// pairs of activation row g. FIRST starts a chain (the addend is zero).
template <bool BF, bool FIRST>
__device__ __forceinline__ void mma_step(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  if constexpr (BF && FIRST)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  else if constexpr (BF)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else if constexpr (FIRST)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------------------------------------------------------
// BF16 activations as FP16. FP16 holds BF16's eight bits over 32 binades, [2^-17, 2^15) (the lower ones as subnormals): a
// chunk of an activation row whose values lie within 32 binades is multiplied by the power of two that takes them there,
// 2^(141 - e), e being a biased exponent: the usual 2^7 (e = kWindowExp) for zeros and magnitudes of [2^-24, 2^8), else that
// of the chunk's largest magnitude (from kExpLow on: below it the power would leave FP32's range, and everything down to
// BF16's subnormals fits under 2^121).
constexpr uint32_t kWindowExp = 134, kExpLow = 20, kExpInf = 255, kExpSpan = 31;
constexpr uint32_t kWindowLow = (kWindowExp - kExpSpan) << 7, kOutside = 0xe000e000u;
constexpr float kWindowScale = 128.0f, kWindowUnscale = 1.0f / 128.0f;
// Has a bit of kOutside set where one of a pair is not in the usual window: (|v| - 2^-24) as 15-bit patterns lies within 32
// binades there. (Zeros set one too: chunk_range looks closer.) v * 2 drops the upper half's sign and puts the lower half's
// where it does no harm.
__device__ __forceinline__ uint32_t window_bits(uint32_t v) { return v * 2u - 2u * (kWindowLow << 16 | kWindowLow); }
__device__ __forceinline__ float exp_scale(uint32_t e) { return __uint_as_float((268u - e) << 23); }      // 2^(141 - e)
__device__ __forceinline__ float exp_unscale(uint32_t e) { return __uint_as_float((e - 14u) << 23); }     // 2^(e - 141)

// Range of NB pairs: the largest magnitude's 15-bit pattern in the upper half; in the lower 0xffff less (the pattern of the
// smallest magnitude that is not zero, less one), 0 where all are zeros. The ranges of two parts join as their larger halves.
template <int NB>
__device__ __forceinline__ uint32_t chunk_range(const uint32_t (&v)[NB]) {
  uint32_t hi[NB], lo[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    hi[i] = v[i] & 0x7fff7fffu;
    lo[i] = hi[i] + 0x7fff7fffu;              // (zero: the largest of signed halves; else the smaller the lower)
  }
#pragma unroll
  for (int n = NB / 2; n > 0; n /= 2)         // (a chain would cost its latency)
#pragma unroll
    for (int i = 0; i < n; ++i) {
      hi[i] = __vmaxu2(hi[i], hi[i + n]);
      lo[i] = __vmins2(lo[i], lo[i + n]);
    }
  const uint32_t top = max(hi[0] & 0xffffu, hi[0] >> 16), low = ~(lo[0] ^ 0x80008000u);
  return top << 16 | max(low & 0xffffu, low >> 16);
}
// The chunk's exponent e from the ranges of the four lanes that hold it; kWide: its values span more than FP16 holds, or are
// not all finite.
constexpr uint32_t kWide = 0;
__device__ __forceinline__ uint32_t chunk_exp(uint32_t range) {
  range = __vmaxu2(range, __shfl_xor_sync(0xffffffffu, range, 1));
  range = __vmaxu2(range, __shfl_xor_sync(0xffffffffu, range, 2));
  const uint32_t top = range >> 16, smallest = 0x10000u - (range & 0xffffu);
  const uint32_t e = top >> 7 <= kWindowExp && smallest >= kWindowLow ? kWindowExp : max(top >> 7, kExpLow);
  return e < kExpInf && (e <= kExpSpan || smallest >= (e - kExpSpan) << 7) ? e : kWide;
}

__device__ __forceinline__ uint32_t scaled_half2(uint32_t v, float s) {   // two BF16 times s as two FP16
  float lo, hi;
  unpack2(fmul2(pack2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)), pack2(s, s)), lo, hi);
  const __half2 t = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&t);
}
// A pair that fitted the usual window, from FP16 times 2^7 back to BF16.
__device__ __forceinline__ uint32_t window_back(uint32_t h) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  const __nv_bfloat162 t = __floats2bfloat162_rn(f.x * kWindowUnscale, f.y * kWindowUnscale);
  return *reinterpret_cast<const uint32_t*>(&t);
}
// A pair of decoded weights (FP16 with at most 6 significant bits) as BF16: exact.
__device__ __forceinline__ uint32_t half2_to_bf162(uint32_t h) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  const __nv_bfloat162 t = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&t);
}

}  // namespace dg
