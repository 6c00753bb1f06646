// rint(v / s) for the quantizers, bit for bit what an IEEE division followed by round-half-to-even
// gives, without a division per element.
//
// The quantizers read their input once and should be HBM-bound: at 6.5 TB/s an SM receives eight to
// nine 16-bit elements per clock, so it has about fifteen instruction slots for each, and an IEEE
// division with its conversions takes more than that.  So t = v * (1 / s) decides whenever it
// can: with r = rn(1 / s), t = rn(v r) lies within |t| 2^-23 (1 + 2^-24) of v / s and rn(v / s) within
// another |t| 2^-24, so if t is farther than |t| 2^-22 from every half-integer, t and rn(v / s) round
// to the same integer.
//
// Otherwise h, the half-integer next to t, decides: e = v - h s is exact in one FMA (|e| is at most
// |v| 2^-21 and a multiple of the last bit of h s), v / s = h + e / s, and rn(v / s) is h itself - a tie,
// to the even integer - exactly when |e| is at most s times half the spacing of floats on e's side
// of h.  16-bit weights do hit half-integers: with 8-bit mantissas a third of all groups of 128 N(0, 1)
// values have a value (2 k + 1) / 14 of their maximum.  (With a division there instead of the FMA,
// 24576 x 4096 bf16 weights to group-128 nibbles took 86 us; with the FMA 75.)
#pragma once
#include "internal.cuh"

namespace b200q {

// 1.5 * 2^23: adding it to |t| < 2^22 rounds to an integer, ties to even, and leaves that
// integer in the low bits of the sum's mantissa.
constexpr float kRoundMagic = 12582912.0f;

// What a thread knows about its divisor.  `usable`: every |v| of the row or group is at most `peak`
// and |v r| then stays below `most` + 0.49, so no quotient needs the clamp (false for a zero or
// infinite divisor).
struct Divisor {
  float s, r;
  bool usable;
};
__device__ __forceinline__ Divisor make_divisor(float s, float peak, float most) {
  Divisor d;
  d.s = s;
  d.r = __frcp_rn(s);
  d.usable = __fmul_rn(peak, d.r) < most + 0.49f;
  return d;
}

// Two fp32 operations per instruction.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// rint(rn(v / s)) where t, within |t| 2^-22 of it, is next to a half-integer; off = t - rint(t).
__device__ __forceinline__ float round_at_half(float v, float s, float t, float off) {
  const float h = (t - off) + copysignf(0.5f, off);
  const float e = fmaf(-h, s, v);
  // half the spacing of floats at h, away from zero; towards zero it is half of that below |h| = 1/2
  float half_ulp = __uint_as_float((__float_as_uint(h) & 0x7F800000u) - (24u << 23));
  if (fabsf(h) == 0.5f && e * h < 0.0f) half_ulp *= 0.5f;
  // (on the boundary rn() goes to h, whose last mantissa bit is 0)
  return fabsf(e) <= s * half_ulp ? rintf(h) : h + copysignf(0.5f, e);
}

// bits[i]: rint(v[i] / s) + offset in the low mantissa bits, for |v / s| < kMost + 1/2 (kMost a power
// of two less one).  `exact(v)` supplies rint(v / s) + offset, clamped, for elements that are not finite
// and for divisors that are not `usable`.
template <int kMost, typename Exact>
__device__ __forceinline__ void round_quotients8(const float (&v)[8], const Divisor& d, float offset,
                                                 uint32_t (&bits)[8], Exact exact) {
  constexpr float kNear = 0.5f - (kMost + 1) * 2.384185791015625e-7f;    // 1/2 - |t| 2^-22 at the largest |t|
  const float magic = kRoundMagic + offset;
  const uint64_t r2 = pack_f32x2(d.r, d.r), magic2 = pack_f32x2(magic, magic), back2 = pack_f32x2(-magic, -magic);
  const uint64_t minus2 = pack_f32x2(-1.0f, -1.0f);
  bool sure = d.usable;
  float t[8], off[8];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const uint64_t t2 = mul_f32x2(pack_f32x2(v[i], v[i + 1]), r2);
    const uint64_t u2 = add_f32x2(t2, magic2);
    const uint64_t o2 = fma_f32x2(add_f32x2(u2, back2), minus2, t2);     // t - rint(t), exact
    float u0, u1;
    unpack_f32x2(u2, u0, u1);
    unpack_f32x2(t2, t[i], t[i + 1]);
    unpack_f32x2(o2, off[i], off[i + 1]);
    bits[i] = __float_as_uint(u0);
    bits[i + 1] = __float_as_uint(u1);
    sure = sure && fabsf(off[i]) < kNear && fabsf(off[i + 1]) < kNear;   // false for NaN
  }
  if (!sure) {
    bool odd = !d.usable;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (!(fabsf(off[i]) < kNear)) {
        bits[i] = __float_as_uint(round_at_half(v[i], d.s, t[i], off[i]) + magic);
        odd = odd || !(fabsf(off[i]) <= 0.5f);
      }
    }
    if (odd) {
#pragma unroll
      for (int i = 0; i < 8; ++i) bits[i] = exact(v[i]);
    }
  }
}

// The low bytes of four words, in order.
__device__ __forceinline__ uint32_t pack_low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return prmt(prmt(a, b, 0x0040), prmt(c, d, 0x0040), 0x5410);
}

// Eight 16-byte aligned consecutive elements (one load for 16-bit types, two for fp32): as floats,
// and their largest |value| / value / -value with NaN ignored, as fmaxf does.
template <typename T>
struct Vec8;
template <>
struct Vec8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    a = __ldg(reinterpret_cast<const float4*>(p));
    b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  }
  __device__ __forceinline__ void zero() { a = b = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  __device__ __forceinline__ float max_abs() const {
    return fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                 fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
  }
  __device__ __forceinline__ void range(float& neg_lo, float& hi) const {    // max(-min, 0), max(max, 0)
    hi = fmaxf(fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w))), 0.0f);
    neg_lo = fmaxf(-fminf(fminf(fminf(a.x, a.y), fminf(a.z, a.w)), fminf(fminf(b.x, b.y), fminf(b.z, b.w))), 0.0f);
  }
};

__device__ __forceinline__ float low_float(__half2 h) { return __low2float(h); }
__device__ __forceinline__ float high_float(__half2 h) { return __high2float(h); }
__device__ __forceinline__ float low_float(__nv_bfloat162 h) { return __low2float(h); }
__device__ __forceinline__ float high_float(__nv_bfloat162 h) { return __high2float(h); }

template <typename T, typename T2>
struct Vec8Bits16 {
  uint4 v;
  __device__ __forceinline__ void load(const T* p) { v = __ldg(reinterpret_cast<const uint4*>(p)); }
  __device__ __forceinline__ void zero() { v = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ T2 pair(uint32_t w) const { return *reinterpret_cast<const T2*>(&w); }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = low_float(pair(w[i]));
      f[2 * i + 1] = high_float(pair(w[i]));
    }
  }
  __device__ __forceinline__ float max_abs() const {
    const T2 m = __hmax2(__hmax2(__habs2(pair(v.x)), __habs2(pair(v.y))), __hmax2(__habs2(pair(v.z)), __habs2(pair(v.w))));
    return fmaxf(low_float(m), high_float(m));
  }
  __device__ __forceinline__ void range(float& neg_lo, float& hi) const {
    const T2 h = __hmax2(__hmax2(pair(v.x), pair(v.y)), __hmax2(pair(v.z), pair(v.w)));
    const T2 l = __hmin2(__hmin2(pair(v.x), pair(v.y)), __hmin2(pair(v.z), pair(v.w)));
    hi = fmaxf(fmaxf(low_float(h), high_float(h)), 0.0f);
    neg_lo = fmaxf(-fminf(low_float(l), high_float(l)), 0.0f);
  }
};
template <>
struct Vec8<__half> : Vec8Bits16<__half, __half2> {};
template <>
struct Vec8<__nv_bfloat16> : Vec8Bits16<__nv_bfloat16, __nv_bfloat162> {};

// ---------------------------------------------------------------- rows -> int8
// Per-row symmetric int8, for weights (fp16 or fp32 scales: engine/kernels/w8a16_linear.py:43-47,
// engine/quantization/int8.py:19-20) and activations (engine/kernels/w8a8_linear.py:43-44).
enum RowScale { kWeightF16 = B200Q_W8_SCALE_F16, kWeightF32 = B200Q_W8_SCALE_F32, kActivation = 2 };

// NaN: 0 for weights (torch's CPU conversion), -127 for activations (what the clamp gives).  Rare, and
// not inlined: eight copies in each kernel would crowd its loop out of the instruction cache.
template <bool kNanIsZero>
__device__ __noinline__ uint32_t exact_int8(float v, float s) {
  const float q = rintf(__fdiv_rn(v, s));
  if (kNanIsZero && q != q) return 0u;
  return static_cast<uint32_t>(static_cast<int>(fminf(fmaxf(q, -127.0f), 127.0f)));
}

// One block of kThreads per row of whole 16-byte vectors (K % 8 == 0): kHeld vectors of a thread
// stay in registers between the maximum and the rounding; a longer row reads the rest again (from
// L2).  Few threads per row, because what a row costs beyond its elements (the scale's divisions, the
// block's reduction) is paid by each of them.
template <typename T, int kMode, int kThreads>
__global__ void __launch_bounds__(kThreads) rows_to_int8_kernel(const T* __restrict__ x, int64_t ldx, int K,
                                                                int8_t* __restrict__ q, int64_t ldq,
                                                                void* __restrict__ scales) {
  constexpr int kHeld = sizeof(T) == 4 ? 4 : 8;
  constexpr int kWarps = kThreads / 32;
  const int64_t row_no = blockIdx.x;
  const T* row = x + row_no * ldx;
  const int vecs = K / 8;
  Vec8<T> held[kHeld];
#pragma unroll
  for (int h = 0; h < kHeld; ++h) {
    const int v = static_cast<int>(threadIdx.x) + h * kThreads;
    if (v < vecs) held[h].load(row + v * 8); else held[h].zero();
  }
  float peak = 0.0f;
#pragma unroll
  for (int h = 0; h < kHeld; ++h) peak = fmaxf(peak, held[h].max_abs());
  for (int v = static_cast<int>(threadIdx.x) + kHeld * kThreads; v < vecs; v += kThreads) {
    Vec8<T> more;
    more.load(row + v * 8);
    peak = fmaxf(peak, more.max_abs());
  }
  // non-negative floats order like their bits
  peak = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(peak)));
  if (kWarps > 1) {
    __shared__ float warp_peak[kWarps];
    if ((threadIdx.x & 31) == 0) warp_peak[threadIdx.x >> 5] = peak;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; ++w) peak = fmaxf(peak, warp_peak[w]);
  }
  float s;
  if (kMode == kWeightF16) {
    const __half sh = __float2half_rn(__fdiv_rn(fmaxf(peak, 1e-8f), 127.0f));
    if (threadIdx.x == 0) reinterpret_cast<__half*>(scales)[row_no] = sh;
    s = __half2float(sh);                    // may be 0: then every quotient takes the division
  } else if (kMode == kWeightF32) {
    s = __fdiv_rn(fmaxf(peak, 1.1920928955078125e-07f), 127.0f);
    if (threadIdx.x == 0) reinterpret_cast<float*>(scales)[row_no] = s;
  } else {
    s = fmaxf(peak, 1e-8f) * (1.0f / 127.0f);   // tensor / scalar on the reference's device
    if (threadIdx.x == 0) reinterpret_cast<float*>(scales)[row_no] = s;
  }
  const Divisor d = make_divisor(s, peak, 127.0f);
  auto exact = [s](float value) { return exact_int8<kMode != kActivation>(value, s); };
  uint2* out = reinterpret_cast<uint2*>(q + row_no * ldq);
  auto emit = [&](int v, const Vec8<T>& in) {
    float f[8];
    uint32_t b[8];
    in.get(f);
    round_quotients8<127>(f, d, 0.0f, b, exact);
    out[v] = make_uint2(pack_low_bytes(b[0], b[1], b[2], b[3]), pack_low_bytes(b[4], b[5], b[6], b[7]));
  };
#pragma unroll
  for (int h = 0; h < kHeld; ++h) {
    const int v = static_cast<int>(threadIdx.x) + h * kThreads;
    if (v < vecs) emit(v, held[h]);
  }
  for (int v = static_cast<int>(threadIdx.x) + kHeld * kThreads; v < vecs; v += kThreads) {
    Vec8<T> more;
    more.load(row + v * 8);
    emit(v, more);
  }
}

// True when the vector kernel takes these rows (and was launched); a grid of many rows uses as few
// threads per row as hold it in registers, a short one spreads each row over a whole block.
template <typename T, int kMode>
bool launch_rows_to_int8(const T* x, int64_t ldx, int rows, int K, int8_t* q, int64_t ldq, void* scales,
                         cudaStream_t stream) {
  if (K % 8 || reinterpret_cast<uintptr_t>(x) % 16 || ldx * sizeof(T) % 16 || ldq % 8 ||
      reinterpret_cast<uintptr_t>(q) % 8)
    return false;
  const int need = (K / 8 + (sizeof(T) == 4 ? 4 : 8) - 1) / (sizeof(T) == 4 ? 4 : 8);   // threads that hold the row
  if (rows < 64 || need > 128)
    rows_to_int8_kernel<T, kMode, 256><<<rows, 256, 0, stream>>>(x, ldx, K, q, ldq, scales);
  else if (need > 64)
    rows_to_int8_kernel<T, kMode, 128><<<rows, 128, 0, stream>>>(x, ldx, K, q, ldq, scales);
  else if (need > 32)
    rows_to_int8_kernel<T, kMode, 64><<<rows, 64, 0, stream>>>(x, ldx, K, q, ldq, scales);
  else
    rows_to_int8_kernel<T, kMode, 32><<<rows, 32, 0, stream>>>(x, ldx, K, q, ldq, scales);
  return true;
}

}  // namespace b200q
