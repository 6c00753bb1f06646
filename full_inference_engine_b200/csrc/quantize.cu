// Weight quantizers and the 4-bit dequantizer.  One-time (install/load) work, HBM-bound,
// bit-exact against the reference's torch arithmetic (IEEE fp32 division, round-half-to-even).
// Group-128 4-bit weights and int8 weights with 16-byte aligned rows take the vector kernels; the
// others (small groups, odd widths, unaligned views) the element-wise ones.
#include "round_div.cuh"

namespace b200q {

template <typename T>
__device__ __forceinline__ float load_as_float(const T* p, int64_t i);
template <>
__device__ __forceinline__ float load_as_float<float>(const float* p, int64_t i) {
  return p[i];
}
template <>
__device__ __forceinline__ float load_as_float<__half>(const __half* p, int64_t i) {
  return __half2float(p[i]);
}
template <>
__device__ __forceinline__ float load_as_float<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) {
  return __bfloat162float(p[i]);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// clamp that maps NaN to 0 (torch's NaN -> int8 conversion yields 0 on the
// reference's CPU path; an all-zero row divides 0 by a zero fp16 scale).
__device__ __forceinline__ float clamp_nan0(float v, float lo, float hi) {
  if (v != v) return 0.0f;
  return fminf(fmaxf(v, lo), hi);
}

// ------------------------------------------------------------------ W8
// engine/kernels/w8a16_linear.py:43-47 (mode 0) and engine/quantization/int8.py:19-20 (mode 1)
template <typename T>
__global__ void __launch_bounds__(256) quantize_w8_kernel(const T* __restrict__ w, int64_t ldw,
                                                          int N, int K, int mode,
                                                          int8_t* __restrict__ q,
                                                          void* __restrict__ scales) {
  __shared__ float red[8];
  __shared__ float s_div;
  const int n = blockIdx.x;
  const T* row = w + static_cast<int64_t>(n) * ldw;
  float m = 0.0f;
  for (int k = threadIdx.x; k < K; k += blockDim.x) m = fmaxf(m, fabsf(load_as_float(row, k)));
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float mm = red[0];
    for (int i = 1; i < (blockDim.x >> 5); ++i) mm = fmaxf(mm, red[i]);
    if (mode == B200Q_W8_SCALE_F16) {
      float s32 = __fdiv_rn(fmaxf(mm, 1e-8f), 127.0f);
      __half sh = __float2half_rn(s32);
      reinterpret_cast<__half*>(scales)[n] = sh;
      s_div = __half2float(sh);
    } else {
      float s32 = __fdiv_rn(fmaxf(mm, 1.1920928955078125e-07f), 127.0f);
      reinterpret_cast<float*>(scales)[n] = s32;
      s_div = s32;
    }
  }
  __syncthreads();
  const float s = s_div;
  int8_t* qrow = q + static_cast<int64_t>(n) * K;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    float v = rintf(__fdiv_rn(load_as_float(row, k), s));
    qrow[k] = static_cast<int8_t>(static_cast<int>(clamp_nan0(v, -127.0f, 127.0f)));
  }
}

// ------------------------------------------------------------------ W4
// Group-128 rows of 16-byte vectors: sixteen threads hold a group (eight elements each) in registers
// from its maximum to its nibbles, so the weights are read once; a warp takes four pairs of groups, all
// loads issued before the first is used.  The four maxima of a half-warp are reduced together (each
// exchange halves the number of values a lane still carries), which leaves group p's in lanes 4p..4p+3:
// each lane then computes ONE scale and its reciprocal, and the group's sixteen threads fetch it by
// shuffle.  Split-half layout: the eight threads with inputs 0..63 get the other eight's nibbles by
// shuffle and write eight bytes each.  24576 x 4096: bf16 235 -> 75 us and fp16 234 -> 58 us (bound by
// instruction issue), fp32 236 -> 69 us (6.6 TB/s),
// against a block per row that read the weights twice and divided element by element.
__device__ __forceinline__ float max_of_four_groups(const float (&m)[4], int l16) {
  const bool b3 = (l16 & 8) != 0, b2 = (l16 & 4) != 0;
  const float a0 = fmaxf(b3 ? m[2] : m[0], __shfl_xor_sync(0xffffffffu, b3 ? m[0] : m[2], 8));
  const float a1 = fmaxf(b3 ? m[3] : m[1], __shfl_xor_sync(0xffffffffu, b3 ? m[1] : m[3], 8));
  float c = fmaxf(b2 ? a1 : a0, __shfl_xor_sync(0xffffffffu, b2 ? a0 : a1, 4));
  c = fmaxf(c, __shfl_xor_sync(0xffffffffu, c, 2));
  return fmaxf(c, __shfl_xor_sync(0xffffffffu, c, 1));
}

// What round_quotients8 asks for where the reciprocal does not serve (not inlined: rare).
__device__ __noinline__ uint32_t exact_nibble(float v, float s) {
  return static_cast<uint32_t>(static_cast<int>(clamp_nan0(rintf(__fdiv_rn(v, s)), -7.0f, 7.0f)) + 8);
}
__device__ __noinline__ uint32_t exact_magic(float v, float s, float zero) {
  const float q = rintf(__fdiv_rn(v, s));
  // NaN: the nibble 0 whatever the zero-point
  return __float_as_uint(kRoundMagic + (q != q ? -zero : fminf(fmaxf(q, -15.0f), 15.0f)));
}

template <typename T, bool kAsym>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 5) quantize_w4_g128_kernel(const T* __restrict__ w, int64_t ldw, int total,
                                                               int groups, uint8_t* __restrict__ packed,
                                                               __half* __restrict__ scales,
                                                               __half* __restrict__ zeros) {
  constexpr int kPer = 4;
  const int l16 = threadIdx.x & 15;
  const int g0 = (static_cast<int>(blockIdx.x) * 8 + static_cast<int>(threadIdx.x >> 5)) * (2 * kPer) +
                 ((threadIdx.x >> 4) & 1);                 // this half-warp's groups: g0, g0 + 2, g0 + 4, g0 + 6
  const bool dense = ldw == static_cast<int64_t>(groups) * 128;     // the groups follow one another
  Vec8<T> x[kPer];
#pragma unroll
  for (int p = 0; p < kPer; ++p) {
    const int gi = g0 + 2 * p;
    int64_t at = static_cast<int64_t>(gi) * 128;
    if (!dense) {
      const int n = gi / groups;
      at = n * ldw + (gi - n * groups) * 128;
    }
    if (gi < total) x[p].load(w + at + l16 * 8); else x[p].zero();
  }
  const int mine = g0 + 2 * (l16 >> 2);                    // the group whose scale this lane computes
  Divisor d;
  float zp = 0.0f;
  if (!kAsym) {
    float m[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) m[p] = x[p].max_abs();
    const float peak = max_of_four_groups(m, l16);
    d = make_divisor(__fdiv_rn(fmaxf(peak, 1e-8f), 7.0f), peak, 7.0f);
  } else {
    float lo[kPer], hi[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) x[p].range(lo[p], hi[p]);
    const float neg_lo = max_of_four_groups(lo, l16), top = max_of_four_groups(hi, l16);
    d = make_divisor(fmaxf(__fdiv_rn(top + neg_lo, 15.0f), 1e-8f), fmaxf(neg_lo, top), 15.0f);
    zp = clamp_nan0(rintf(__fdiv_rn(neg_lo, d.s)), 0.0f, 15.0f);
  }
  if ((l16 & 3) == 0 && mine < total) {
    scales[mine] = __float2half_rn(d.s);
    if (kAsym) zeros[mine] = __float2half_rn(zp);
  }
#pragma unroll
  for (int p = 0; p < kPer; ++p) {
    const int gi = g0 + 2 * p;
    const int from = (threadIdx.x & 16) + 4 * p;
    Divisor dp;
    dp.s = __shfl_sync(0xffffffffu, d.s, from);
    dp.r = __shfl_sync(0xffffffffu, d.r, from);
    dp.usable = __shfl_sync(0xffffffffu, d.usable ? 1 : 0, from) != 0;
    float f[8];
    uint32_t b[8];
    x[p].get(f);
    if (!kAsym) {
      round_quotients8<7>(f, dp, 8.0f, b, [&](float value) { return exact_nibble(value, dp.s); });
      const uint32_t q0 = pack_low_bytes(b[0], b[1], b[2], b[3]), q1 = pack_low_bytes(b[4], b[5], b[6], b[7]);
      const uint32_t h0 = __shfl_xor_sync(0xffffffffu, q0, 8), h1 = __shfl_xor_sync(0xffffffffu, q1, 8);
      if (gi < total && l16 < 8)
        *reinterpret_cast<uint2*>(packed + static_cast<int64_t>(gi) * 64 + l16 * 8) =
            make_uint2(q0 | (h0 << 4), q1 | (h1 << 4));
    } else {
      const float z = __shfl_sync(0xffffffffu, zp, from);
      round_quotients8<15>(f, dp, 0.0f, b, [&](float value) { return exact_magic(value, dp.s, z); });
      int v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = min(max(static_cast<int>(b[i]) - (__float_as_int(kRoundMagic) - static_cast<int>(z)), 0), 15);
      // positions 0..7 hold inputs 0,2,4,6,1,3,5,7
      const int word = v[0] + 16 * v[2] + 256 * v[4] + 4096 * v[6] + 65536 * (v[1] + 16 * v[3] + 256 * v[5] + 4096 * v[7]);
      if (gi < total) reinterpret_cast<uint32_t*>(packed)[static_cast<int64_t>(gi) * 16 + l16] = static_cast<uint32_t>(word);
    }
  }
}

// Any group size and alignment: one block per row.  Per (row, group) scale (and zero-point) into shared memory, then pack.
// REF:  engine/kernels/w4a16_format.py:32-50.
template <typename T>
__global__ void __launch_bounds__(256) quantize_w4_kernel(const T* __restrict__ w, int64_t ldw,
                                                          int N, int K, int group, int layout,
                                                          uint8_t* __restrict__ packed,
                                                          __half* __restrict__ scales,
                                                          __half* __restrict__ zeros) {
  extern __shared__ float sm[];  // [groups] scale32, then [groups] zero (ASYM)
  const int groups = K / group;
  float* s_scale = sm;
  float* s_zero = sm + groups;
  const int n = blockIdx.x;
  const T* row = w + static_cast<int64_t>(n) * ldw;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int g = warp; g < groups; g += nwarps) {
    const T* gp = row + static_cast<int64_t>(g) * group;
    if (layout == B200Q_W4_REF_SPLIT_HALF_SYM) {
      float m = 0.0f;
      for (int j = lane; j < group; j += 32) m = fmaxf(m, fabsf(load_as_float(gp, j)));
      m = warp_max(m);
      if (lane == 0) {
        float s32 = __fdiv_rn(fmaxf(m, 1e-8f), 7.0f);
        s_scale[g] = s32;
        scales[static_cast<int64_t>(n) * groups + g] = __float2half_rn(s32);
      }
    } else {
      float lo = 0.0f, hi = 0.0f;
      for (int j = lane; j < group; j += 32) {
        float v = load_as_float(gp, j);
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
      }
      lo = warp_min(lo);
      hi = warp_max(hi);
      if (lane == 0) {
        float s32 = fmaxf(__fdiv_rn(hi - lo, 15.0f), 1e-8f);
        float zp = clamp_nan0(rintf(__fdiv_rn(-lo, s32)), 0.0f, 15.0f);
        s_scale[g] = s32;
        s_zero[g] = zp;
        scales[static_cast<int64_t>(n) * groups + g] = __float2half_rn(s32);
        zeros[static_cast<int64_t>(n) * groups + g] = __float2half_rn(zp);
      }
    }
  }
  __syncthreads();
  if (layout == B200Q_W4_REF_SPLIT_HALF_SYM) {
    const int half = group >> 1;
    uint8_t* prow = packed + static_cast<int64_t>(n) * (K >> 1);
    for (int idx = threadIdx.x; idx < (K >> 1); idx += blockDim.x) {
      const int g = idx / half, j = idx - g * half;
      const float s = s_scale[g];
      const T* gp = row + static_cast<int64_t>(g) * group;
      float a = clamp_nan0(rintf(__fdiv_rn(load_as_float(gp, j), s)), -7.0f, 7.0f) + 8.0f;
      float b = clamp_nan0(rintf(__fdiv_rn(load_as_float(gp, j + half), s)), -7.0f, 7.0f) + 8.0f;
      prow[idx] = static_cast<uint8_t>(static_cast<int>(a) | (static_cast<int>(b) << 4));
    }
  } else {
    uint32_t* prow = reinterpret_cast<uint32_t*>(packed) + static_cast<int64_t>(n) * (K >> 3);
    for (int idx = threadIdx.x; idx < (K >> 3); idx += blockDim.x) {
      const int k0 = idx << 3;
      const int g = k0 / group;
      const float s = s_scale[g], zp = s_zero[g];
      uint32_t word = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float v = clamp_nan0(rintf(__fdiv_rn(load_as_float(row, k0 + i), s)) + zp, 0.0f, 15.0f);
        // input i of the word sits at nibble position (i & 1) * 4 + (i >> 1): positions
        // 0..7 hold inputs 0,2,4,6,1,3,5,7
        word |= static_cast<uint32_t>(static_cast<int>(v)) << (4 * ((i & 1) * 4 + (i >> 1)));
      }
      prow[idx] = word;
    }
  }
}

// ------------------------------------------------------------------ dequant
// out[n,k] = fp16(nibble - zero) * fp16(scale), product in fp16.
// REF: engine/kernels/w4a16_format.py:53-69, engine/kernels/w4a16_linear.py:211-242.
// One thread per 32-bit packed word (8 weights).
__global__ void __launch_bounds__(256) dequant_w4_kernel(const uint32_t* __restrict__ packed,
                                                         const __half* __restrict__ scales,
                                                         const __half* __restrict__ zeros,
                                                         int layout, int N, int K, int group,
                                                         __half* __restrict__ out, int64_t ldo) {
  const int words_per_row = K >> 3;
  const int64_t total = static_cast<int64_t>(N) * words_per_row;
  const int groups = K / group;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int n = static_cast<int>(t / words_per_row);
    const int wi = static_cast<int>(t - static_cast<int64_t>(n) * words_per_row);
    const uint32_t w = packed[t];
    __half* orow = out + static_cast<int64_t>(n) * ldo;
    if (layout == B200Q_W4_REF_SPLIT_HALF_SYM) {
      const int half = group >> 1;
      const int byte0 = wi << 2;               // first packed byte of this word in the row
      const int g = byte0 / half;
      const int j = byte0 - g * half;
      const __half2 s = __half2half2(scales[static_cast<int64_t>(n) * groups + g]);
      W4Quad q = dequant_w4_word_splithalf(w, __float2half2_rn(1032.0f), __float2half2_rn(-72.0f), s);
      __half2* lo = reinterpret_cast<__half2*>(orow + static_cast<int64_t>(g) * group + j);
      __half2* hi = reinterpret_cast<__half2*>(orow + static_cast<int64_t>(g) * group + half + j);
      lo[0] = q.lo01;
      lo[1] = q.lo23;
      hi[0] = q.hi01;
      hi[1] = q.hi23;
    } else {
      const int k0 = wi << 3;
      const int g = k0 / group;
      const float zp = __half2float(zeros[static_cast<int64_t>(n) * groups + g]);
      const __half2 s = __half2half2(scales[static_cast<int64_t>(n) * groups + g]);
      W4Oct o = dequant_w4_word_seq(w, __float2half2_rn(1024.0f + zp),
                                    __float2half2_rn(-(64.0f + zp)), s);
      __half2* dst = reinterpret_cast<__half2*>(orow + k0);
      dst[0] = o.k01;
      dst[1] = o.k23;
      dst[2] = o.k45;
      dst[3] = o.k67;
    }
  }
}

// Group-128 rows with 16-byte aligned output rows: a thread takes eight packed bytes and writes two
// 16-byte pieces (split-half: inputs 8j.. of either half of the group; zero-point layout: two
// words of eight consecutive inputs).  24576 x 4096: 72 -> 44 us (5.8 TB/s) split-half, 77 -> 56 us
// zero-points, against one word per thread with 4-byte stores.
template <bool kAsym>
__global__ void __launch_bounds__(256) dequant_w4_g128_kernel(const uint2* __restrict__ packed,
                                                              const __half* __restrict__ scales,
                                                              const __half* __restrict__ zeros, int64_t total,
                                                              int pieces, __half* __restrict__ out, int64_t ldo) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int n = static_cast<int>(t / pieces);
  const int c = static_cast<int>(t - static_cast<int64_t>(n) * pieces);    // eight-byte piece of the row: group c / 8
  const uint2 v = __ldg(packed + t);
  const __half2 s = __half2half2(__ldg(scales + (t >> 3)));
  __half* orow = out + static_cast<int64_t>(n) * ldo;
  uint4 a, b;
  __half* at;
  if (!kAsym) {
    const __half2 bias_lo = __float2half2_rn(1032.0f), nbias_hi = __float2half2_rn(-72.0f);
    const W4Quad p = dequant_w4_word_splithalf(v.x, bias_lo, nbias_hi, s);
    const W4Quad q = dequant_w4_word_splithalf(v.y, bias_lo, nbias_hi, s);
    a = make_uint4(as_u32(p.lo01), as_u32(p.lo23), as_u32(q.lo01), as_u32(q.lo23));
    b = make_uint4(as_u32(p.hi01), as_u32(p.hi23), as_u32(q.hi01), as_u32(q.hi23));
    at = orow + (c >> 3) * 128 + (c & 7) * 8;
  } else {
    const float zp = __half2float(__ldg(zeros + (t >> 3)));
    const __half2 bias_lo = __float2half2_rn(1024.0f + zp), nbias_hi = __float2half2_rn(-(64.0f + zp));
    const W4Oct p = dequant_w4_word_seq(v.x, bias_lo, nbias_hi, s);
    const W4Oct q = dequant_w4_word_seq(v.y, bias_lo, nbias_hi, s);
    a = make_uint4(as_u32(p.k01), as_u32(p.k23), as_u32(p.k45), as_u32(p.k67));
    b = make_uint4(as_u32(q.k01), as_u32(q.k23), as_u32(q.k45), as_u32(q.k67));
    at = orow + c * 16;
  }
  *reinterpret_cast<uint4*>(at) = a;
  *reinterpret_cast<uint4*>(at + (kAsym ? 8 : 64)) = b;
}

// Scalar variant for groups whose half is not a multiple of 4 bytes (REF layout only).
__global__ void __launch_bounds__(256) dequant_w4_ref_bytes_kernel(
    const uint8_t* __restrict__ packed, const __half* __restrict__ scales, int N, int K, int group,
    __half* __restrict__ out, int64_t ldo) {
  const int bytes_per_row = K >> 1;
  const int half = group >> 1;
  const int groups = K / group;
  const int64_t total = static_cast<int64_t>(N) * bytes_per_row;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int n = static_cast<int>(t / bytes_per_row);
    const int bi = static_cast<int>(t - static_cast<int64_t>(n) * bytes_per_row);
    const int g = bi / half, j = bi - g * half;
    const uint32_t b = packed[t];
    const __half s = scales[static_cast<int64_t>(n) * groups + g];
    __half* orow = out + static_cast<int64_t>(n) * ldo + static_cast<int64_t>(g) * group;
    orow[j] = __hmul(__int2half_rn(static_cast<int>(b & 15u) - 8), s);
    orow[j + half] = __hmul(__int2half_rn(static_cast<int>(b >> 4) - 8), s);
  }
}

// ------------------------------------------------------------------ host launchers
static bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

template <typename T>
static void launch_quantize_w8_typed(const T* w, int64_t ldw, int N, int K, int mode, int8_t* q, void* scales,
                                     cudaStream_t stream) {
  const bool done = mode == B200Q_W8_SCALE_F16 ? launch_rows_to_int8<T, kWeightF16>(w, ldw, N, K, q, K, scales, stream)
                                               : launch_rows_to_int8<T, kWeightF32>(w, ldw, N, K, q, K, scales, stream);
  if (!done) quantize_w8_kernel<T><<<N, 256, 0, stream>>>(w, ldw, N, K, mode, q, scales);
}

int launch_quantize_w8(const void* w, int w_dtype, int64_t ldw, int N, int K, int mode, int8_t* q,
                       void* scales, cudaStream_t stream) {
  switch (w_dtype) {
    case B200Q_F32:
      launch_quantize_w8_typed(static_cast<const float*>(w), ldw, N, K, mode, q, scales, stream);
      break;
    case B200Q_F16:
      launch_quantize_w8_typed(static_cast<const __half*>(w), ldw, N, K, mode, q, scales, stream);
      break;
    case B200Q_BF16:
      launch_quantize_w8_typed(static_cast<const __nv_bfloat16*>(w), ldw, N, K, mode, q, scales, stream);
      break;
    default:
      return B200Q_ERR_INVALID;
  }
  return note_launch();
}

template <typename T>
static int launch_quantize_w4_typed(const T* w, int64_t ldw, int N, int K, int group, int layout, uint8_t* packed,
                                    __half* scales, __half* zeros, cudaStream_t stream) {
  const int groups = K / group;
  const int64_t total = static_cast<int64_t>(N) * groups;
  if (group == 128 && total < (1ll << 30) && aligned16(w) && ldw * sizeof(T) % 16 == 0 &&
      reinterpret_cast<uintptr_t>(packed) % 8 == 0) {
    constexpr int kGroupsPerBlock = 8 * 2 * 4;
    const int blocks = static_cast<int>((total + kGroupsPerBlock - 1) / kGroupsPerBlock);
    if (layout == B200Q_W4_ASYM_ZP_INT32)
      quantize_w4_g128_kernel<T, true><<<blocks, 256, 0, stream>>>(w, ldw, static_cast<int>(total), groups, packed,
                                                                  scales, zeros);
    else
      quantize_w4_g128_kernel<T, false><<<blocks, 256, 0, stream>>>(w, ldw, static_cast<int>(total), groups, packed,
                                                                   scales, zeros);
    return note_launch();
  }
  const size_t smem = sizeof(float) * 2 * static_cast<size_t>(groups);
  if (smem > 48 * 1024) return B200Q_ERR_UNSUPPORTED;
  quantize_w4_kernel<T><<<N, 256, smem, stream>>>(w, ldw, N, K, group, layout, packed, scales, zeros);
  return note_launch();
}

int launch_quantize_w4(const void* w, int w_dtype, int64_t ldw, int N, int K, int group,
                       int layout, void* packed, void* scales, void* zeros, cudaStream_t stream) {
  auto p = static_cast<uint8_t*>(packed);
  auto s = static_cast<__half*>(scales);
  auto z = static_cast<__half*>(zeros);
  switch (w_dtype) {
    case B200Q_F32:
      return launch_quantize_w4_typed(static_cast<const float*>(w), ldw, N, K, group, layout, p, s, z, stream);
    case B200Q_F16:
      return launch_quantize_w4_typed(static_cast<const __half*>(w), ldw, N, K, group, layout, p, s, z, stream);
    case B200Q_BF16:
      return launch_quantize_w4_typed(static_cast<const __nv_bfloat16*>(w), ldw, N, K, group, layout, p, s, z, stream);
    default:
      return B200Q_ERR_INVALID;
  }
}

int launch_dequant_w4(const void* packed, const void* scales, const void* zeros, int layout,
                      int N, int K, int group, void* out, int64_t ldo, cudaStream_t stream) {
  const bool word_path =
      (layout == B200Q_W4_ASYM_ZP_INT32) ? (group % 8 == 0) : ((group >> 1) % 4 == 0);
  const bool aligned = (reinterpret_cast<uintptr_t>(out) % 4 == 0) && (ldo % 2 == 0) &&
                       (reinterpret_cast<uintptr_t>(packed) % 4 == 0);
  const int64_t pieces = static_cast<int64_t>(N) * (K >> 4);       // of eight packed bytes
  if (group == 128 && aligned16(out) && ldo % 8 == 0 && reinterpret_cast<uintptr_t>(packed) % 8 == 0 &&
      pieces < (1ll << 38)) {
    const unsigned blocks = static_cast<unsigned>((pieces + 255) / 256);
    if (layout == B200Q_W4_ASYM_ZP_INT32)
      dequant_w4_g128_kernel<true><<<blocks, 256, 0, stream>>>(
          static_cast<const uint2*>(packed), static_cast<const __half*>(scales), static_cast<const __half*>(zeros),
          pieces, K >> 4, static_cast<__half*>(out), ldo);
    else
      dequant_w4_g128_kernel<false><<<blocks, 256, 0, stream>>>(
          static_cast<const uint2*>(packed), static_cast<const __half*>(scales), nullptr, pieces, K >> 4,
          static_cast<__half*>(out), ldo);
  } else if (word_path && aligned) {
    const int64_t total = static_cast<int64_t>(N) * (K >> 3);
    int blocks = static_cast<int>((total + 255) / 256);
    if (blocks > 148 * 32) blocks = 148 * 32;
    if (blocks < 1) blocks = 1;
    dequant_w4_kernel<<<blocks, 256, 0, stream>>>(
        static_cast<const uint32_t*>(packed), static_cast<const __half*>(scales),
        static_cast<const __half*>(zeros), layout, N, K, group, static_cast<__half*>(out), ldo);
  } else {
    if (layout != B200Q_W4_REF_SPLIT_HALF_SYM) return B200Q_ERR_UNSUPPORTED;
    const int64_t total = static_cast<int64_t>(N) * (K >> 1);
    int blocks = static_cast<int>((total + 255) / 256);
    if (blocks > 148 * 32) blocks = 148 * 32;
    if (blocks < 1) blocks = 1;
    dequant_w4_ref_bytes_kernel<<<blocks, 256, 0, stream>>>(
        static_cast<const uint8_t*>(packed), static_cast<const __half*>(scales), N, K, group,
        static_cast<__half*>(out), ldo);
  }
  return note_launch();
}

}  // namespace b200q
