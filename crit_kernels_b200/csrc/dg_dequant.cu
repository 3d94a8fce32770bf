// NVFP4 dequantizers for B200 (sm_100a): the matrix's values [N][K] as BF16 / FP16, or as FP8 E4M3 in units of a
// per-row factor. The "dequantize" half of the reference's dequantize-then-matmul path.
//
// Replaces the Triton kernels of the reference package decode-gemv (torch-ext/decode_gemv/triton_gemv.py:156-176
// `_decode_kernel` / `decode`, :179-200 `_decode_fp8_kernel` / `decode_fp8`). Contract, as the reference's test pins
// it (tests/test_decode_gemv.py:131-140): value = e2m1(code) * scale (exact in FP32) times the row's factor, one FP32
// product, rounded once to the output type; the FP8 form clamps to +-448 before rounding to nearest even.
//
// Pure streaming, HBM-bound and write-dominated: per value 0.5 B of codes + 1/16 B of scales in, 2 B (or 1 B) out.
// A lane writes one 16-byte vector per step: 8 values from one 32-bit word of codes for the 16-bit types, 16 values
// (one scale block) from two words for FP8, so a warp reads 128 (256) consecutive bytes and writes 512 consecutive
// bytes per step; four steps are loaded before any is converted.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <type_traits>

#include "../../include/decode_gemv_b200.h"
#include "dg_kernel.cuh"

namespace {

enum : int { DQ_BF16 = 1, DQ_F16 = 2, DQ_E4M3 = 3 };
constexpr int kThreads = 256;
constexpr int kBatch = 4;   // 16-byte output units a thread has in flight in a large matrix

__device__ __forceinline__ float e4m3_to_f32(uint32_t byte) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)byte, __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

// 8 codes (word c, element 2i in the low nibble of byte i) -> 8 FP32 values: (e2m1 * scale) * factor.
__device__ __forceinline__ void values8(uint32_t c, float scale, float factor, float (&v)[8]) {
  uint32_t h[4];
  dg::decode_e2m1_h(c, h);                                 // (element 2q, element 2q + 1) of byte q
  const dg::pk2 s2 = dg::pack2(scale, scale), f2 = dg::pack2(factor, factor);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 w = __half22float2(*reinterpret_cast<const __half2*>(&h[q]));
    dg::unpack2(dg::fmul2(dg::fmul2(dg::pack2(w.x, w.y), s2), f2), v[2 * q], v[2 * q + 1]);
  }
}

template <int OUT>
__device__ __forceinline__ uint32_t round2(float lo, float hi) {   // two values of a 16-bit type in one word
  if constexpr (OUT == DQ_BF16) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&t);
  } else {
    const __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&t);
  }
}
// Four values as E4M3 bytes; the saturating conversion gives +-448 beyond +-448, as the reference's clamp before its
// rounding.
__device__ __forceinline__ uint32_t round4_e4m3(float a, float b, float c, float d) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}

// A lane's unit is 16 output bytes: one word of codes (8 values) for the 16-bit types, two words (16 values, one
// scale block) for FP8. `unit` counts such units from the start of the matrix.
template <int OUT> struct Unit { static constexpr int WORDS = OUT == DQ_E4M3 ? 2 : 1; };

// The matrix is one run of units, BATCH x kThreads to a CTA, whatever its rows: the rows of codes, scales and values follow
// each other without gaps. As many CTAs as that takes: a CTA that is done makes room for the next, so that loads and stores
// of different CTAs overlap all the time (eight persistent CTAs per SM, walking whole rows, took 33.5 us for 8192 x 8192 to
// BF16; this 30.7, the rate of a device-to-device copy of as many bytes; stores alone take 24.5; 28672 x 8192: 105.7 and 92.2).
// BATCH is kBatch where that makes a CTA for every SM, else one unit per thread: a small matrix is bound by a CTA's latency and by
// the SMs without one (256 x 512 to BF16 2.03 us with four, 1.52 with one, and 1.74 with a CTA per row; 1024 x 1024 to FP8 2.84,
// 2.37 and 2.65; from a CTA per SM on both are the same).
template <int OUT, int BATCH>
__global__ void __launch_bounds__(kThreads)
    dequantize_kernel(const uint32_t* codes, const uint8_t* scales, const float* factor, uint4* __restrict__ out, long long total, int units) {
  constexpr int WORDS = Unit<OUT>::WORDS;
  const long long first = (long long)blockIdx.x * (kThreads * BATCH);
  const int count = (int)min((long long)(kThreads * BATCH), total - first);
  // row and place within the row of the CTA's first unit (units: per row)
  const long long row0 = total <= 0xffffffffll ? (long long)((uint32_t)first / (uint32_t)units) : first / units;
  const int place0 = (int)(first - row0 * units);
  codes += first * WORDS;
  scales += (first * WORDS) >> 1;                           // (first is even)
  factor += row0;
  out += first;
  // This kernel may start while the previous one of the stream still runs (its CTAs are then in place when that one ends): what the
  // previous kernel writes is read behind the wait. It does not let the next kernel start before it has ended itself: its output is
  // a weight matrix, and a GEMV that has been told of static weights reads those before its own wait. us as an ordinary launch and
  // so: 8192 x 8192 to BF16, eager calls 30.8 and 28.8, 1024 x 1024 in a graph 2.05 and 1.70; to FP8, 4414 x 1216 in a graph 3.16 and
  // 2.53, 3000 x 4096 4.70 and 4.27 (with the next kernel let in at the start 4.30 and 4.97: its CTAs take the places of CTAs still to come).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t c[BATCH][WORDS] = {}, sb[BATCH] = {};
  float f[BATCH] = {};
#pragma unroll
  for (int b = 0; b < BATCH; ++b) {
    const int u = b * kThreads + threadIdx.x;
    if (u < count) {
      if constexpr (WORDS == 2) {
        const uint2 two = reinterpret_cast<const uint2*>(codes)[u];
        c[b][0] = two.x;
        c[b][1] = two.y;
        sb[b] = scales[u];                          // the unit is one scale block
      } else {
        c[b][0] = codes[u];
        sb[b] = scales[u >> 1];                   // one scale per 16 values = per two words
      }
      f[b] = factor[(uint32_t)(place0 + u) / (uint32_t)units];
    }
  }
#pragma unroll
  for (int b = 0; b < BATCH; ++b) {
    const int u = b * kThreads + threadIdx.x;
    if (u < count) {
      const float scale = e4m3_to_f32(sb[b]);
      float v[8];
      uint4 o;
      values8(c[b][0], scale, f[b], v);
      if constexpr (WORDS == 2) {
        o.x = round4_e4m3(v[0], v[1], v[2], v[3]);
        o.y = round4_e4m3(v[4], v[5], v[6], v[7]);
        values8(c[b][1], scale, f[b], v);
        o.z = round4_e4m3(v[0], v[1], v[2], v[3]);
        o.w = round4_e4m3(v[4], v[5], v[6], v[7]);
      } else {
        o.x = round2<OUT>(v[0], v[1]);
        o.y = round2<OUT>(v[2], v[3]);
        o.z = round2<OUT>(v[4], v[5]);
        o.w = round2<OUT>(v[6], v[7]);
      }
      out[u] = o;
    }
  }
}

// SM count of the current device (0: not a device this library runs on), looked up once per device.
int sm_count() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int sms = cache[dev].load(std::memory_order_relaxed);
  if (sms == 0) {
    int major = 0, count = 0;
    const bool ok = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) == cudaSuccess &&
                    major == 10 &&
                    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && count > 0;
    sms = ok ? count : -1;
    cache[dev].store(sms, std::memory_order_relaxed);
  }
  return sms > 0 ? sms : 0;
}

bool aligned(const void* ptr, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(ptr) % bytes == 0; }

}  // namespace

extern "C" DG_API int dg_enqueue_dequantize(const uint8_t* codes, const uint8_t* scales, const float* factor, void* out,
                                     int out_kind, int N, int K, void* stream) {
  if (N < 1 || K < 16 || K % 16 || out_kind < DQ_BF16 || out_kind > DQ_E4M3) return (int)cudaErrorInvalidValue;
  if (!codes || !scales || !factor || !out || !aligned(codes, 16) || !aligned(out, 16) || !aligned(factor, 4))
    return (int)cudaErrorInvalidValue;
  const int sms = sm_count();
  if (sms < 1) return (int)cudaErrorInvalidDevice;
  const int units = K / (out_kind == DQ_E4M3 ? 16 : 8);      // 16-byte output vectors per row
  const long long total = (long long)N * units;
  auto launch = [&](auto out_type) {
    constexpr int OUT = decltype(out_type)::value;
    const bool batched = total >= (long long)sms * kThreads * kBatch;
    const int run = kThreads * (batched ? kBatch : 1);
    const dim3 grid((unsigned)((total + run - 1) / run));
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = dim3(kThreads);
    config.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, batched ? dequantize_kernel<OUT, kBatch> : dequantize_kernel<OUT, 1>, reinterpret_cast<const uint32_t*>(codes),
                              scales, factor, static_cast<uint4*>(out), total, units);
  };
  const cudaError_t e = out_kind == DQ_BF16  ? launch(std::integral_constant<int, DQ_BF16>())
                        : out_kind == DQ_F16 ? launch(std::integral_constant<int, DQ_F16>())
                                             : launch(std::integral_constant<int, DQ_E4M3>());
  return (int)(e != cudaSuccess ? e : cudaGetLastError());
}
