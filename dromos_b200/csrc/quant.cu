// Load-time conversions of the kernel ABI: lx_quantize_weight, lx_dequantize_weight, lx_quantize_w8 and the per-token
// activation quantizer lx_quantize_act. Every rounding is to nearest, ties to even, saturating; weight quantizers
// divide with IEEE division, the FP4 activation quantizer multiplies by the block's reciprocal (the ABI's rules:
// lernex/dromos engine/cuda/kernels.h:479-493, 513-523).
#include <algorithm>

#include "launch.cuh"

namespace b200 {
namespace {

constexpr int kBlock = 256;

// Nearest e2m1 code (0, .5, 1, 1.5, 2, 3, 4, 6 with a sign bit): the code is how many midpoints lie below |x|, a
// value on a midpoint goes to the even neighbour, magnitudes saturate at 6, and a zero result carries no sign.
__device__ __forceinline__ uint32_t e2m1_encode(float x) {
  const float a = fminf(fabsf(x), 6.0f);
  uint32_t code = (a > 0.25f) + (a >= 0.75f) + (a > 1.25f) + (a >= 1.75f) + (a > 2.5f) + (a >= 3.5f) + (a > 5.0f);
  return code | ((x < 0.0f && code) ? 8u : 0u);
}

// ---- weights ----------------------------------------------------------------------------------------------------------
// All of these are bound by HBM as long as a lane moves 16 bytes of bf16 per access with several accesses in flight; with
// one 2-byte value per lane they were bound by the count of loads (figures beside launch_rows below).
constexpr int kInFlight = 4;  // 16-byte words of a row a lane has in flight
constexpr int kRowWarps = kBlock / 32;

// The largest magnitude of eight packed bf16 values and `m` (packed too), NaN ignored as fmaxf does.
__device__ __forceinline__ uint32_t max_abs2(uint32_t m, const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) asm("max.bf16x2 %0, %0, %1;" : "+r"(m) : "r"(w[j] & 0x7fff7fffu));
  return m;
}
__device__ __forceinline__ float max_of2(uint32_t m) { return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)); }

// One warp per row: the row's absmax, then its values. kFp8: e4m3 with scale absmax / 448; else int8, absmax / 127.
// WORDS > 0: rows of whole 16-byte words (cols % 8 == 0, w on 16 and q on 8 bytes), so many of them in flight per lane.
template <bool kFp8, int WORDS>
__global__ void __launch_bounds__(kBlock) quantize_rows_kernel(const uint16_t* __restrict__ w, uint8_t* __restrict__ q,
                                                               float* __restrict__ scale, int64_t rows, int cols) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kRowWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const uint16_t* src = w + row * cols;
  const uint4* src8 = reinterpret_cast<const uint4*>(src);
  const int words = cols / 8;
  float amax = 0.0f;
  if constexpr (WORDS > 0) {
    uint32_t m = 0;
    for (int c0 = lane; c0 < words; c0 += 32 * WORDS) {
      uint4 v[WORDS];
#pragma unroll
      for (int i = 0; i < WORDS; ++i) v[i] = c0 + 32 * i < words ? __ldg(src8 + c0 + 32 * i) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < WORDS; ++i) m = max_abs2(m, v[i]);
    }
    amax = max_of2(m);
  } else {
    for (int c = lane; c < cols; c += 32) amax = fmaxf(amax, fabsf(bf16_bits_to_f32(src[c])));
  }
  amax = warp_max(amax);
  constexpr float qmax = kFp8 ? 448.0f : 127.0f;
  const float s = amax > 0.0f ? __fdiv_rn(amax, qmax) : 1.0f;
  if (lane == 0) scale[row] = s;
  uint8_t* dst = q + row * cols;
  auto code = [&](uint32_t bits) -> uint32_t {
    const float v = __fdiv_rn(bf16_bits_to_f32(bits), s);
    if constexpr (kFp8) return e4m3_encode(fminf(fmaxf(v, -448.0f), 448.0f)) & 0xffu;
    else return static_cast<uint32_t>(static_cast<int>(fminf(fmaxf(rintf(v), -127.0f), 127.0f))) & 0xffu;
  };
  if constexpr (WORDS > 0) {
    for (int c0 = lane; c0 < words; c0 += 32 * WORDS) {
      uint4 v[WORDS];
#pragma unroll
      for (int i = 0; i < WORDS; ++i) v[i] = c0 + 32 * i < words ? __ldg(src8 + c0 + 32 * i) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < WORDS; ++i) {
        if (c0 + 32 * i >= words) break;
        const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        uint32_t o[2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
          o[h] = code(u[2 * h] & 0xffffu) | (code(u[2 * h] >> 16) << 8) | (code(u[2 * h + 1] & 0xffffu) << 16) | (code(u[2 * h + 1] >> 16) << 24);
        reinterpret_cast<uint2*>(dst)[c0 + 32 * i] = make_uint2(o[0], o[1]);
      }
    }
  } else {
    for (int c = lane; c < cols; c += 32) dst[c] = static_cast<uint8_t>(code(src[c]));
  }
}

// max |w| of the whole matrix, as the bit pattern of a non-negative float (which orders like the value). VEC: w on 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(kBlock) absmax_kernel(const uint16_t* __restrict__ w, int64_t n, unsigned long long* out) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x, step = static_cast<int64_t>(gridDim.x) * kBlock;
  float m = 0.0f;
  if constexpr (VEC) {  // n is whole blocks of 16 values
    const uint4* w8 = reinterpret_cast<const uint4*>(w);
    uint32_t m2 = 0;
    for (int64_t i = i0; i < n / 8; i += step * kInFlight) {
      uint4 v[kInFlight];
#pragma unroll
      for (int j = 0; j < kInFlight; ++j) v[j] = i + j * step < n / 8 ? __ldg(w8 + i + j * step) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < kInFlight; ++j) m2 = max_abs2(m2, v[j]);
    }
    m = max_of2(m2);
  } else {
    for (int64_t i = i0; i < n; i += step) m = fmaxf(m, fabsf(bf16_bits_to_f32(w[i])));
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<unsigned int*>(out), __float_as_uint(m));
}

// Eight e2m1 codes of eight values, e2m1_encode's: the conversion rounds and saturates alike, but keeps the sign of a value
// that rounds to zero.
__device__ __forceinline__ uint32_t e2m1_encode8(const float (&v)[8]) {
  uint32_t c;
  asm("{ .reg .b8 b0, b1, b2, b3; cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1; cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5; cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7; mov.b32 %0, {b0, b1, b2, b3}; }"
      : "=r"(c)
      : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  const uint32_t nonzero = (c | (c >> 1) | (c >> 2)) & 0x11111111u;
  return c & (nonzero * 8u | 0x77777777u);
}

// One thread per 16-value block: the block's e4m3 scale (absmax / (6 * global)), then its codes, w / (scale * global).
// VEC: w on 16 and q on 8 bytes.
template <bool VEC>
__global__ void __launch_bounds__(kBlock) quantize_nvfp4_kernel(const uint16_t* __restrict__ w, uint8_t* __restrict__ q,
                                                                uint8_t* __restrict__ scale, float global, int64_t rows,
                                                                int cols) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t per_row = cols / 16;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (i >= rows * per_row) return;
  const uint16_t* src = w + i * 16;
  float v[16], amax = 0.0f;
  if constexpr (VEC) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(src)), b = __ldg(reinterpret_cast<const uint4*>(src) + 1);
    const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) v[2 * j] = __uint_as_float(u[j] << 16), v[2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = bf16_bits_to_f32(src[j]);
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(v[j]));
  const uint32_t sb = e4m3_encode(__fdiv_rn(amax, 6.0f * global));
  scale[i] = static_cast<uint8_t>(sb);
  const float eff = e4m3_to_f32(sb) * global;
  uint8_t* dst = q + i * 8;
  uint32_t o[2] = {0, 0};
  if (eff > 0.0f) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float r[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) r[j] = __fdiv_rn(v[8 * h + j], eff);
      o[h] = e2m1_encode8(r);
    }
  }
  if constexpr (VEC) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
  } else {
#pragma unroll
    for (int p = 0; p < 8; ++p) dst[p] = static_cast<uint8_t>(o[p >> 2] >> (8 * (p & 3)));
  }
}

// out[n, k] = bf16(element * row factor). WORDS > 0 (cols % 8 == 0, out on 16, the elements on 8 bytes, NVFP4's on 4): eight values per
// lane and word, a warp takes WORDS words of 32 lanes of one row, the pieces of a row one after the other; 0: one thread per element.
template <int F, int WORDS>
__global__ void __launch_bounds__(kBlock) dequantize_kernel(const uint8_t* __restrict__ data, const uint8_t* __restrict__ scale,
                                                            float global, uint16_t* __restrict__ out, int64_t rows, int cols, unsigned pieces) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  if constexpr (WORDS > 0) {
    const unsigned group = blockIdx.x / pieces, piece = blockIdx.x - group * pieces;
    const int64_t row = static_cast<int64_t>(group) * kRowWarps + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int words = cols / 8, c0 = static_cast<int>(piece) * 32 * WORDS + static_cast<int>(threadIdx.x & 31);
    uint4* dst = reinterpret_cast<uint4*>(out + row * cols);
    float rf = 1.0f;
    if constexpr (F != LX_W_NVFP4) rf = reinterpret_cast<const float*>(scale)[row];
    uint2 e[WORDS];
    uint32_t sb[WORDS];
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
      const int c = c0 + 32 * i;
      if (c >= words) continue;
      if constexpr (F == LX_W_NVFP4) {
        e[i].x = __ldg(reinterpret_cast<const uint32_t*>(data + row * (cols / 2)) + c);
        sb[i] = __ldg(scale + row * (cols / 16) + c / 2);
      } else {
        e[i] = __ldg(reinterpret_cast<const uint2*>(data + row * cols) + c);
      }
    }
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
      const int c = c0 + 32 * i;
      if (c >= words) continue;
      float v[8];
      if constexpr (F == LX_W_NVFP4) {
        const float f = e4m3_to_f32(sb[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = e2m1_to_f32((e[i].x >> (4 * j)) & 15u) * f * global;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t word = j < 4 ? e[i].x : e[i].y;
          if constexpr (F == LX_W_INT8)  // 2^23 + 128 + the value, as bits: the conversion instructions are a quarter as fast
            v[j] = (__uint_as_float(__byte_perm(word ^ 0x80808080u, 0x4b000000u, 0x7440 + (j & 3))) - 8388736.0f) * rf;
          else v[j] = e4m3_to_f32((word >> (8 * (j & 3))) & 0xffu) * rf;
        }
      }
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = (f32_to_bf16_bits(v[2 * j]) & 0xffffu) | (f32_to_bf16_bits(v[2 * j + 1]) << 16);
      dst[c] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    return;
  }
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (i >= rows * cols) return;
  const int64_t n = i / cols, k = i % cols;
  float v;
  if constexpr (F == LX_W_INT8) {
    v = static_cast<float>(reinterpret_cast<const int8_t*>(data)[i]) * reinterpret_cast<const float*>(scale)[n];
  } else if constexpr (F == LX_W_FP8) {
    v = e4m3_to_f32(data[i]) * reinterpret_cast<const float*>(scale)[n];
  } else {
    const uint32_t byte = data[n * (cols / 2) + k / 2];
    v = e2m1_to_f32((k & 1) ? byte >> 4 : byte & 15u) * e4m3_to_f32(scale[n * (cols / 16) + k / 16]) * global;
  }
  out[i] = static_cast<uint16_t>(f32_to_bf16_bits(v));
}

// One CTA per activation row: absmax, then the row's values in the math's number type.
__global__ void __launch_bounds__(kBlock) quantize_act_kernel(const void* __restrict__ x, int x_dtype, int ld_x, int math,
                                                              uint8_t* __restrict__ q, int ld_q, float* __restrict__ scale,
                                                              uint8_t* __restrict__ block_scale, int ld_bs, int K) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  __shared__ float part[kBlock / 32];
  const int m = blockIdx.x;
  const int64_t base = static_cast<int64_t>(m) * ld_x;
  float a = 0.0f;
  for (int k = threadIdx.x; k < K; k += kBlock) a = fmaxf(a, fabsf(load_f32(x, x_dtype, base + k)));
  a = warp_max(a);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = a;
  __syncthreads();
  a = 0.0f;
  for (int i = 0; i < kBlock / 32; ++i) a = fmaxf(a, part[i]);
  uint8_t* qr = q + static_cast<int64_t>(m) * ld_q;
  if (math == LX_MATH_INT8 || math == LX_MATH_FP8) {
    const float qmax = math == LX_MATH_INT8 ? 127.0f : 448.0f;
    const float inv = a > 0.0f ? __fdiv_rn(qmax, a) : 0.0f;
    for (int k = threadIdx.x; k < K; k += kBlock) {
      const float v = load_f32(x, x_dtype, base + k) * inv;
      if (math == LX_MATH_INT8)
        qr[k] = static_cast<uint8_t>(static_cast<int8_t>(static_cast<int>(fminf(fmaxf(rintf(v), -127.0f), 127.0f))));
      else
        qr[k] = static_cast<uint8_t>(e4m3_encode(v));
    }
    if (threadIdx.x == 0) scale[m] = a > 0.0f ? __fdiv_rn(a, qmax) : 1.0f;
    return;
  }
  const float g = a > 0.0f ? __fdiv_rn(a, 2688.0f) : 1.0f;
  if (threadIdx.x == 0) scale[m] = g;
  uint8_t* bs = block_scale + static_cast<int64_t>(m) * ld_bs;
  for (int b = threadIdx.x; b < K / 16; b += kBlock) {
    float v[16], amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] = load_f32(x, x_dtype, base + 16 * b + j);
      amax = fmaxf(amax, fabsf(v[j]));
    }
    const uint32_t s8 = e4m3_encode(__fdiv_rn(amax, 6.0f * g));
    bs[b] = static_cast<uint8_t>(s8);
    const float d = e4m3_to_f32(s8) * g;
    const float r = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      uint32_t lo = 0, hi = 0;
      if (d > 0.0f) {
        lo = e2m1_encode(v[2 * p] * r);
        hi = e2m1_encode(v[2 * p + 1] * r);
      }
      qr[8 * b + p] = static_cast<uint8_t>(lo | (hi << 4));
    }
  }
}

unsigned blocks_for(int64_t n, int per_block) { return static_cast<unsigned>((n + per_block - 1) / per_block); }

// 14336 x 4096, quantized and expanded again (a loader's pass; 352 / 264 MB): INT8 272 -> 104 us, FP8 265 -> 77, NVFP4 365 -> 112
// with the copy of its maximum to the host. (INT8's quantizer is left with an IEEE division and a rounding per value.) Rows shorter
// than a word per lane go value by value (FP8 50000 x 64: 10.1 us, by words 13.4), rows of one word with one in flight (FP8 100000 x 256:
// 26.0 us, with four 31.5, value by value 28.1).
template <bool kFp8>
int launch_rows(const void* w, uint8_t* q, float* scale, int64_t rows, int cols, cudaStream_t s) {
  const bool vec = cols % 8 == 0 && cols >= 256 && aligned(w, 16) && aligned(q, 8);
  return launch_kernel(!vec ? quantize_rows_kernel<kFp8, 0> : cols <= 256 ? quantize_rows_kernel<kFp8, 1> : quantize_rows_kernel<kFp8, kInFlight>, dim3(blocks_for(rows, kRowWarps)), dim3(kBlock), 0, s,
                       static_cast<const uint16_t*>(w), q, scale, rows, cols);
}

template <int F, int WORDS>
int launch_dequantize_words(const lx_weight& w, float global, uint16_t* out, int64_t rows, int cols, cudaStream_t s) {
  const unsigned pieces = WORDS ? blocks_for(cols, 256 * std::max(1, WORDS)) : 1;
  const unsigned grid = WORDS ? blocks_for(rows, kRowWarps) * pieces : blocks_for(rows * cols, kBlock);
  return launch_kernel(dequantize_kernel<F, WORDS>, dim3(grid), dim3(kBlock), 0, s, static_cast<const uint8_t*>(w.data), static_cast<const uint8_t*>(w.scale), global, out, rows, cols, pieces);
}

// A row's values are spread over as many warps as they fill, four words a lane (14336 x 4096: FP8 27.6 us, one warp per row 30.3, one
// thread per value 169); where that is fewer than four blocks per SM, or a row is no longer than one word a lane, one word a lane. (One warp per
// row leaves few wide rows to few SMs: FP8 64 x 16384 11.1 us, 1 x 65536 32; now 1.7 and 1.2; one thread per value 3.2 and 1.2.
// 100000 x 256 with one word a lane 14, with four 15.6.)
template <int F>
int launch_dequantize(const lx_weight& w, float global, uint16_t* out, int64_t rows, int cols, cudaStream_t s) {
  if (cols % 8 != 0 || !aligned(out, 16) || !aligned(w.data, F == LX_W_NVFP4 ? 4 : 8)) return launch_dequantize_words<F, 0>(w, global, out, rows, cols, s);
  const bool few = static_cast<int64_t>(blocks_for(rows, kRowWarps)) * blocks_for(cols, 256 * kInFlight) < 148 * 4;
  if (few || cols <= 256) return launch_dequantize_words<F, 1>(w, global, out, rows, cols, s);
  return launch_dequantize_words<F, kInFlight>(w, global, out, rows, cols, s);
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" int lx_quantize_w8(const void* w, int8_t* q, float* scale, int64_t rows, int cols, void* stream) {
  if (rows <= 0) return kOk;
  if (cols <= 0 || !w || !q || !scale) return kInvalid;
  return launch_rows<false>(w, reinterpret_cast<uint8_t*>(q), scale, rows, cols, static_cast<cudaStream_t>(stream));
}

extern "C" int lx_quantize_weight(const void* w, lx_weight* out, int64_t rows, int cols, void* stream) {
  if (!out || !w) return kInvalid;
  if (rows <= 0) return kOk;
  if (cols <= 0) return kInvalid;
  auto s = static_cast<cudaStream_t>(stream);
  auto* data = static_cast<uint8_t*>(const_cast<void*>(out->data));
  auto* scale = const_cast<void*>(out->scale);
  const auto* src = static_cast<const uint16_t*>(w);
  switch (out->type) {
    case LX_W_BF16X: {
      if (!data) return kInvalid;
      const int64_t bytes = lx_bf16x_bytes(w, rows, cols, stream);
      if (bytes < 0) return static_cast<int>(-bytes);
      return lx_bf16x_encode(w, rows, cols, data, bytes, stream);
    }
    case LX_W_INT8:
      if (!data || !scale) return kInvalid;
      return lx_quantize_w8(w, reinterpret_cast<int8_t*>(data), static_cast<float*>(scale), rows, cols, stream);
    case LX_W_FP8:
      if (!data || !scale) return kInvalid;
      return launch_rows<true>(w, data, static_cast<float*>(scale), rows, cols, s);
    case LX_W_NVFP4: {
      if (!data || !scale || cols % 16 != 0) return kInvalid;
      // The global scale is max|w| / (448 * 6); it is a host field of lx_weight, so this load-time call reads the
      // maximum back (it synchronizes the stream).
      ResultWord word(s);
      if (word.status) return word.status;
      const int64_t n = rows * cols;
      const bool vec = aligned(w, 16);
      if (int e = launch_kernel(vec ? absmax_kernel<true> : absmax_kernel<false>, dim3(std::min<unsigned>(blocks_for(n, kBlock), 148 * 8)), dim3(kBlock), 0, s,
                                src, n, word.dev))
        return e;
      unsigned long long value = 0;
      if (int e = word.read(&value)) return e;
      const auto bits = static_cast<unsigned int>(value);
      float amax;
      memcpy(&amax, &bits, sizeof(amax));
      const float global = amax / 2688.0f;
      out->global = global;
      return launch_kernel(vec && aligned(data, 8) ? quantize_nvfp4_kernel<true> : quantize_nvfp4_kernel<false>, dim3(blocks_for(rows * (cols / 16), kBlock)),
                           dim3(kBlock), 0, s, src, data, static_cast<uint8_t*>(scale), global, rows, cols);
    }
    default:
      return kInvalid;  // BF16: nothing to quantize
  }
}

extern "C" int lx_dequantize_weight(const lx_weight* w, void* out, int64_t rows, int cols, void* stream) {
  if (!w || !w->data || !out) return kInvalid;
  if (rows <= 0) return kOk;
  if (cols <= 0) return kInvalid;
  if (w->type < LX_W_BF16 || w->type > LX_W_BF16X) return kInvalid;
  if (w->type != LX_W_BF16 && w->type != LX_W_BF16X && !w->scale) return kInvalid;
  if (w->type == LX_W_NVFP4 && cols % 16 != 0) return kInvalid;
  auto s = static_cast<cudaStream_t>(stream);
  if (w->type == LX_W_BF16X) return lx_bf16x_decode(w->data, rows, cols, out, stream);
  if (w->type == LX_W_BF16)
    return static_cast<int>(cudaMemcpyAsync(out, w->data, 2 * rows * cols, cudaMemcpyDeviceToDevice, s));
  auto* o = static_cast<uint16_t*>(out);
  switch (w->type) {
    case LX_W_INT8: return launch_dequantize<LX_W_INT8>(*w, 1.0f, o, rows, cols, s);
    case LX_W_FP8: return launch_dequantize<LX_W_FP8>(*w, 1.0f, o, rows, cols, s);
    default: return launch_dequantize<LX_W_NVFP4>(*w, w->global, o, rows, cols, s);
  }
}

extern "C" int lx_quantize_act(const void* x, lx_dtype x_dtype, int ld_x, lx_math math, void* q, int ld_q, float* scale,
                               void* block_scale, int ld_bs, int M, int K, void* stream) {
  if (M <= 0) return kOk;
  if (!x || !q || !scale || K <= 0 || !valid_dtype(x_dtype) || (M > 1 && ld_x < K)) return kInvalid;
  if (math != LX_MATH_INT8 && math != LX_MATH_FP8 && math != LX_MATH_FP4) return kInvalid;
  if (math == LX_MATH_FP4) {
    if (K % 16 != 0 || !block_scale || (M > 1 && (ld_q < K / 2 || ld_bs < K / 16))) return kInvalid;
  } else if (M > 1 && ld_q < K) {
    return kInvalid;
  }
  return launch_kernel(quantize_act_kernel, dim3(M), dim3(kBlock), 0, static_cast<cudaStream_t>(stream), x,
                       static_cast<int>(x_dtype), ld_x, static_cast<int>(math), static_cast<uint8_t*>(q), ld_q, scale,
                       static_cast<uint8_t*>(block_scale), ld_bs, K);
}
