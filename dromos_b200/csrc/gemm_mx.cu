// lx_gemm_w on NVFP4 weights: y[m, n] = sum_k x[m, k] * w[n, k], up to 64 activation rows per pass, with the weights
// multiplied as they are stored (tcgen05.mma kind::mxf4nvf4, block scales of 16 values applied by the tensor core).
//
// Why digits. No instruction multiplies e2m1 x e4m3-block-scale weights by wider activations, and expanding the weights to
// f16 in registers was what bound the kernels before this one: eight converter warps, ~27 instructions per 16 values, 72 us
// for 28672 x 8192 at 16 rows where the bytes take 20. So it is the activations that are taken apart, once per call, into
// what the instruction multiplies: every block of 16 values gets the power of two of its largest magnitude as its scale and
// seven digits in base 13, 24 bits below that magnitude. (e2m1 holds 0, 1, 2, 3, 4, 6, 8, 12 halves with a sign: every residue
// of 13. Base 8, whose digits need only -4..4, gives 21 bits from seven columns, and nine columns of it leave no room for 64
// rows in tensor memory.) A digit is a column of its own (column j * Mp + m is digit j of row m), summed on its own in f32 and
// put together in the epilogue, least first.
//
// Remainders. A bf16 value within 2^-16 of its block's largest comes out of the digits exactly. What they leave of smaller ones is
// kept too where it can be told in a result: as digits under a scale of its own, and its stage of 256 values of K is multiplied a
// second time from these, into the same accumulators. The operands are then exact down to 2^-33 of the row's largest magnitude and
// rounded at 2^-41 of it below (an f16 row under one power of two: 2^-31 and 2^-39), so that an output whose weights are zero
// wherever the row has its outliers is as exact as any other. It is dropped where all that is left of 2048 values together is
// below 2^-24 (K <= 512; in proportion to K beyond, as f32 sums of so many products) of what as many values add up to that have the
// geometric mean of the smaller of every two neighbours: the sums were cut off by more, for every output that is not made of a few of
// the smallest values alone, be half of the weights zero and half of the values a thousand times the others. (N(0, 1) rows
// and products of SwiGLU hardly ever need a second stage; one outlier channel of 3000 needs one stage of 16; an outlier of 256 and more in
// every block all of them. Kept always, SwiGLU rows took twice as long: 28672 x 8192, 64 rows 138 us.) Which stages go
// again, only the values say: the preparation leaves a bit per row and stage, and a chunk's stage goes again if any of its rows has
// one. A row without them adds zeros, so its bits do not depend on the rows beside it.
//
// What a product costs: an instruction covers 128 weight rows x 64 values of K (four times kind::f16's) for half a cycle per
// column; up to 64 rows are 448 columns in two instructions of four and three digits. A launch takes up to 1024 rows in
// chunks of at most 64, the chunks of a weight panel next to each other so that its later readers find it in L2.
//
// Measured (replayed graphs; before: the f16 expansion): 28672 x 8192, 16 / 32 / 48 / 64 rows 70.7 / 72.1 / 74.2 / 80.3 -> 36.1 / 47.4
// / 64.7 / 78.5 us; 14336 x 4096, 64 / 100 / 500 / 1000 rows 26.8 / 49.5 / 205 / 406 -> 25.4 / 43.6 / 136 / 248. At
// 64 rows it is the 60 KB of digits that every SM fetches from L2 per 12 KB of weights. Error against 64 bits, N(0, 1) rows: 4e-8 at
// every K (f16: 9e-8 at K = 512, 2.3e-6 at 8192); with an outlier of 2^6 .. 2^20 in every block, outputs whose weights are zero there:
// 5e-8 .. 7.5e-7 at K = 8192 (f16: 2.3e-6; seven base-8 digits alone, as this kernel began: 4e-6 .. 0.4).
//   * The block scales go to tensor memory with tcgen05.st. Written to shared memory for tcgen05.cp they needed the proxy fence,
//     which waits for the thread's scale loads in flight: 84 us. With the activations' scales by tcgen05.cp: 57 us (copies
//     and products of one pipe wait for each other).
//   * As many stages of activations in flight as of weights: with four, 16 rows took 50 us.
//
// Roles (one CTA per SM, tiles of R <= 128 weight rows dealt evenly, as in gemm_tc.cu): warps 0-3 epilogue (lane = weight
// row); warps 4-7 bring the block scales: each thread loads its weight row's 16 bytes per stage straight from memory, kAhead
// stages ahead (a tile copy of 16 bytes per row costs the copy engine as much as one of 128), the four warps exchange rows
// through shared memory, and every warp writes all of them to its quarter of tensor memory, the activations' beside them;
// warp 8 weights, warp 10 activations (one thread each, bulk copies, no multicast); warp 9 issues.
//
// Weights and their scales stream before the dependency wait, as in gemm_tc.cu. Every wait is bounded; a role that gives up
// leaves its loop, the producers wait (bounded) for their copies in flight, and the CTA frees its tensor memory.
#include "tc.cuh"

namespace b200 {
namespace {

constexpr int kMxStageK = 256;                  // values of K per stage: 128 bytes per weight row, four products
constexpr int kMxDigits = 7;
constexpr int kMxBase = 13;
constexpr int kMxUnit = 23;                     // a block's values are whole numbers of 2^(e - kMxUnit), e the exponent of its largest
constexpr int kMxThreads = 11 * 32;
constexpr int kMxScaleBytes = 2 * 128 * 16;     // shared memory in which the scale warps exchange rows, for each stage of a slot: two of 128 rows x 16 bytes
constexpr int kAhead = 8;                       // stages whose weight scales a thread has in flight

// How a chunk's rows lie in accumulator columns and in the workspace. An instruction has at most 256 columns, in whole 16s. A stage's
// activations are its digits and, from sf_off on, its block scales: as they go to tensor memory, those of whole 128 columns per product (64
// values of K), or (compact, what small chunks take) those of sf_rows rows, a word each.
struct MxLayout {
  int Mp = 0;                // accumulator columns per digit
  int cols0 = 0, cols1 = 0;  // columns of a step's first instruction and of its second (0: one takes all digits)
  int sf_off = 0, sf_rows = 0, x_bytes = 0;
  static constexpr __host__ __device__ int compact_rows(bool two_atoms) { return two_atoms ? 32 : 16; }  // as many as chunks of the same kernel can have
  MxLayout() = default;
  explicit MxLayout(int rows, int compact_as = 0) {
    auto whole = [](int c) { return (c + 15) / 16 * 16; };
    Mp = (rows + 7) / 8 * 8;
    cols0 = whole(kMxDigits * Mp);
    if (cols0 > 256) cols0 = 4 * Mp, cols1 = whole((kMxDigits - 4) * Mp);  // four digits, then the rest
    sf_off = (cols0 + cols1) * (kMxStageK / 2);
    sf_rows = compact_as;
    x_bytes = sf_off + (compact_as ? 16 * compact_as : 4 * ((cols0 + 127) / 128) * 512);
  }
};

struct MxParams {
  const void* x;            // the activations themselves, for rows with infinities
  int x_bf16, ld_x;
  const uint8_t* w;         // e2m1 [N, K / 2]
  const uint8_t* scale;     // e4m3 [N, K / 16]
  float global;
  int N, K, M;
  int chunks, chunk_rows;   // the activation rows are multiplied in chunks of at most 64
  int64_t chunk_bytes;      // a chunk's prepared activations
  int R, box_bytes;         // weight rows per tile; shared memory of a stage's box (1024-aligned)
  MxLayout lay[2];          // the chunks' and the last one's, which may have fewer rows
  int sf0, sf_turns;        // where in tensor memory the scales begin, and for how many slots in turn (4, 2 or 1)
  const uint8_t* xprep;
  int64_t remainders;       // from a stage's digits to those of its remainders
  const uint8_t* again;     // [chunks][groups][64]: bit b of byte (c, g, m): row m of chunk c has remainders in stage 8 g + b
  int groups;
  const float* row_scale;   // per activation row: what its sums are multiplied by
  int buffers;              // accumulators (2 where they fit)
  int SW, SX;
  const void* bias;
  int bias_dtype;
  void* y;
  int y_dtype, ld_y;
  float alpha, beta;
  int* status;
};

// ---- activations -----------------------------------------------------------------------------------------------------------
// bf16 bits of value k of a row (f32 rows are rounded first, as lx_gemm_w does).
template <bool XBF>
__device__ __forceinline__ uint32_t bf16_at(const void* x, int64_t i) {
  if constexpr (XBF) return static_cast<const uint16_t*>(x)[i];
  else return f32_to_bf16_bits(static_cast<const float*>(x)[i]) & 0xffffu;
}
// Eight values as packed bf16.
template <bool XBF>
__device__ __forceinline__ uint4 bf16x8_at(const void* x, int64_t i, bool vec) {
  if (vec) {
    if constexpr (XBF) return *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + i);
    const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(x) + i), b = *reinterpret_cast<const float4*>(static_cast<const float*>(x) + i + 4);
    auto pack = [](float lo, float hi) { return (f32_to_bf16_bits(lo) & 0xffffu) | (f32_to_bf16_bits(hi) << 16); };
    return make_uint4(pack(a.x, a.y), pack(a.z, a.w), pack(b.x, b.y), pack(b.z, b.w));
  }
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = bf16_at<XBF>(x, i + 2 * j) | (bf16_at<XBF>(x, i + 2 * j + 1) << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint32_t max_magnitude(uint32_t m, const uint4& v) {  // bf16 magnitudes order as integers, NaN above all
  const uint32_t t = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
  return max(m, max(t & 0xffffu, t >> 16));
}
// Digits come in pairs: for a residue u of 169, the e2m1 codes (the digit's half) of its two base-13 digits, the lower one in bits
// 0-3, and in bit 8 what the pair carries. Residue r of 13 is the digit r, or r - 13 where e2m1 has that: 0 1 2 3 4 -8 6 -6 8 -4 -3 -2 -1.
__device__ __forceinline__ uint32_t digit_pair(uint32_t u) {
  constexpr uint64_t kCodes = 0x9abc6d5e43210ull;
  auto code_of = [&](uint32_t r) { return static_cast<uint32_t>(kCodes >> (4 * r)) & 15u; };
  const uint32_t lo = code_of(u % kMxBase), next = u / kMxBase + (lo >> 3);  // 0..13
  const uint32_t hi = next == kMxBase ? 0u : code_of(next);
  return lo | hi << 4 | (next == kMxBase ? 256u : hi >> 3 << 8);
}
// The seven digits of q, |q| < 1.246 * 2^24, as codes into bits 4 i .. 4 i + 3 of w[0..6], most significant first. (Three steps of a pair
// from a table in shared memory; six of a digit are twice the instructions, and the preparation is bound by them.)
__device__ __forceinline__ void put_digits(int q, int i, const uint16_t* pairs, uint32_t (&w)[kMxDigits]) {
  constexpr uint32_t kPair = kMxBase * kMxBase, kBias = kPair << 18;  // keeps what is divided positive
#pragma unroll
  for (int j = kMxDigits - 1; j > 0; j -= 2) {
    const uint32_t u = static_cast<uint32_t>(q) + kBias, t = u / kPair, c = pairs[u - t * kPair];
    w[j] |= (c & 15u) << (4 * i);
    w[j - 1] |= (c >> 4 & 15u) << (4 * i);
    q = static_cast<int>(t - kBias / kPair + (c >> 8));
  }
  w[0] |= static_cast<uint32_t>(q < 0 ? 8 - q : q) << (4 * i);  // -4..4 is left
}
// 2^e as ue4m3, e in -9..8.
__device__ __forceinline__ uint32_t ue4m3_pow2(int e) { return e >= -6 ? static_cast<uint32_t>(e + 7) << 3 : 1u << (e + 9); }
// 2^e as f32, e in -149..127.
__device__ __forceinline__ float exp2_of(int e) { return __uint_as_float(e >= -126 ? static_cast<uint32_t>(e + 127) << 23 : 1u << (e + 149)); }

// Block (piece, row): 256 threads, each 8 values (half a scale block) of an activation row; every block finds the row's largest
// magnitude again (a few KB, from L2), which saves a second kernel. (With 32 values per thread the seven digits of each were
// ~1400 instructions in a row: at 16 rows the preparation took as long as an eighth of the product.) A warp's values are one
// stage's, a block's eight stages': their bits are one byte of `again`. A block without remainders gets the scale zero there, which
// makes whatever its digits are zero.
// A row with a NaN has NaN outputs; one with infinities has no digits, and -0 as its scale: the epilogue adds its infinities up.
constexpr int kPrepThreads = 256;  // (at most 40 registers each: a block fits beside the product's CTA and starts under its end. With 48,
                                   // and 140 in the product, it did not: 14336 x 4096 at 32 rows 23 us instead of 19)
template <bool XBF>
__global__ void __launch_bounds__(kPrepThreads, 6) mx_prep_kernel(const void* __restrict__ x, int ld_x, int K, int chunks, int chunk_rows, int64_t chunk_bytes,
                                                               const MxLayout lay, const MxLayout lay_last, uint8_t* __restrict__ out, int64_t remainders,
                                                               uint8_t* __restrict__ again, float* __restrict__ row_scale) {
  pdl_trigger();
  __shared__ uint32_t part[kPrepThreads / 32], stages_again;
  __shared__ unsigned long long all_squares;
  __shared__ int all_exponents, all_pairs, all_count;
  __shared__ uint16_t pairs[kMxBase * kMxBase];
  if (threadIdx.x < kMxBase * kMxBase) pairs[threadIdx.x] = static_cast<uint16_t>(digit_pair(threadIdx.x));
  pdl_wait();  // the kernel before this one may still be reading the workspace
  const int row_id = blockIdx.y, chunk = row_id / chunk_rows, m = row_id - chunk * chunk_rows, tid = threadIdx.x;
  const int64_t row = static_cast<int64_t>(row_id) * ld_x;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ld_x % (XBF ? 8 : 4) == 0;
  const int k0 = (blockIdx.x * kPrepThreads + tid) * 8;
  const uint4 v = k0 < K ? bf16x8_at<XBF>(x, row + k0, vec) : make_uint4(0, 0, 0, 0);
  uint32_t top = 0;
#pragma unroll 4
  for (int k = 8 * tid; k < K; k += 8 * kPrepThreads) top = max_magnitude(top, bf16x8_at<XBF>(x, row + k, vec));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  if ((tid & 31) == 0) part[tid >> 5] = top;
  if (tid == 0) stages_again = 0, all_squares = 0, all_exponents = all_pairs = all_count = 0;
  uint32_t block_top = max_magnitude(0, v);
  block_top = max(block_top, __shfl_xor_sync(0xffffffffu, block_top, 1));
  __syncthreads();
  top = 0;
#pragma unroll
  for (int i = 0; i < kPrepThreads / 32; ++i) top = max(top, part[i]);
  const bool finite = top < 0x7f80u;
  const int e_row = max(static_cast<int>(top >> 7), 30) - 127;
  if (blockIdx.x == 0 && tid == 0)
    row_scale[row_id] = finite ? exp2_of(e_row - 7 - kMxUnit) : __uint_as_float(top == 0x7f80u ? 0x80000000u : 0x7fc00000u);
  // The block's exponent; one less for a largest value below 1.25 * 2^e, which the digits still hold. 2^-9 is the least scale.
  const int e = max(max(static_cast<int>(block_top + 96) >> 7, 2) - 128, e_row - 17);
  // 2^(kMxUnit - e) in two factors: the whole can be beyond f32
  const int half = (kMxUnit - e) / 2;
  const float f0 = exp2_of(half), f1 = exp2_of(kMxUnit - e - half), to_least = exp2_of(e - e_row + 17);
  const uint32_t keep = finite ? ~0u : 0u, words[4] = {v.x & keep, v.y & keep, v.z & keep, v.w & keep};
  uint32_t w[kMxDigits] = {};
  bool some = false;
  auto value_of = [&](int i) { return bf16_bits_to_f32((words[i / 2] >> (16 * (i & 1))) & 0xffffu) * f0 * f1; };
  auto rest_of = [&](float t) { return __float2int_rn((t - rintf(t)) * to_least); };  // what the digits leave, in units of the least scale: up to 2^16
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float t = value_of(i);
    some |= rest_of(t) != 0;
    put_digits(__float2int_rn(t), i, pairs, w);
  }
  uint32_t with_rest = __ballot_sync(0xffffffffu, some);
  if (with_rest && (tid & 31) == 0) atomicOr(&stages_again, 1u << (tid >> 5));
  __syncthreads();
  uint32_t stages = stages_again;
  if (stages) {
    // Can the remainders of these 2048 values be told in a result (see above)? Sums of whole numbers: the order does not matter.
    unsigned long long squares = 0;
    int exponents = 0, pairs_of = 0, count = 0;  // of the smaller of each two neighbours (not zero), those pairs, all values
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t rest = static_cast<uint32_t>(abs(rest_of(value_of(i))));
      squares += static_cast<unsigned long long>(rest) * rest;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t a = words[i] & 0x7fffu, b = words[i] >> 16 & 0x7fffu, least = a && b ? min(a, b) : a | b;
      if (least) exponents += static_cast<int>(least >> 7), ++pairs_of;
      count += (a != 0) + (b != 0);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      squares += __shfl_xor_sync(0xffffffffu, squares, o);
      exponents += __shfl_xor_sync(0xffffffffu, exponents, o);
      pairs_of += __shfl_xor_sync(0xffffffffu, pairs_of, o);
      count += __shfl_xor_sync(0xffffffffu, count, o);
    }
    if ((tid & 31) == 0) {
      atomicAdd(&all_squares, squares);
      atomicAdd(&all_exponents, exponents);
      atomicAdd(&all_pairs, pairs_of);
      atomicAdd(&all_count, count);
    }
    __syncthreads();
    const float typical = static_cast<float>(all_exponents) / static_cast<float>(all_pairs) - static_cast<float>(127 + e_row - 40);  // log2, in units of the least scale
    const float long_row = fmaxf(1.0f, static_cast<float>(K) * 0x1p-9f);
    if (static_cast<float>(all_squares) <= static_cast<float>(all_count) * exp2f(2.0f * typical) * (0x1p-48f * long_row * long_row)) with_rest = stages = 0;
  }
  if (tid == 0) again[(static_cast<int64_t>(chunk) * gridDim.x + blockIdx.x) * kMaxRows + m] = static_cast<uint8_t>(stages);
  if (k0 >= K) return;
  const bool last = chunk + 1 == chunks;
  const int Mp = last ? lay_last.Mp : lay.Mp, NC = last ? lay_last.cols0 + lay_last.cols1 : lay.cols0 + lay.cols1;
  uint8_t* stage = out + chunk * chunk_bytes + static_cast<size_t>(k0 / kMxStageK) * (last ? lay_last.x_bytes : lay.x_bytes);
  const int kb = (k0 % kMxStageK) / 2;
#pragma unroll
  for (int j = 0; j < kMxDigits; ++j) *reinterpret_cast<uint32_t*>(stage + block_offset(NC, kb & ~15, j * Mp + m) + (kb & 15)) = w[j];
  const bool block_rest = (with_rest >> (tid & 30) & 3u) != 0;  // this thread's eight values' or its neighbour's
  int zeros = 0;
  if (with_rest) {
    // Under the largest scale that keeps them whole: few columns get few more bits, and their sums stay exact. (Under the least
    // scale every product cut off the sums of the digits above: 2.5e-6 at K = 4096 with an outlier in every block, now 6e-8.)
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) bits |= static_cast<uint32_t>(rest_of(value_of(i)));
    bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
    if (block_rest) {
      zeros = __ffs(static_cast<int>(bits)) - 1;
      uint32_t d[kMxDigits] = {};
#pragma unroll
      for (int i = 0; i < 8; ++i) put_digits(rest_of(value_of(i)) >> zeros, i, pairs, d);
#pragma unroll
      for (int j = 0; j < kMxDigits; ++j) *reinterpret_cast<uint32_t*>(stage + remainders + block_offset(NC, kb & ~15, j * Mp + m) + (kb & 15)) = d[j];
    }
  }
  if (k0 % 16 != 0) return;
  const uint8_t sf = static_cast<uint8_t>(finite ? ue4m3_pow2(e - e_row + 8) : 0x38u), sf_rest = static_cast<uint8_t>(block_rest ? ue4m3_pow2(zeros - 9) : 0u);
  uint8_t* sfs = stage + (last ? lay_last.sf_off : lay.sf_off) + (k0 % 64) / 16;
  const int product = (k0 % kMxStageK) / 64;
  if (lay.sf_rows) {  // once for all digits of the row
    const int at = product * (4 * lay.sf_rows) + 4 * m;
    sfs[at] = sf;
    sfs[remainders + at] = sf_rest;
    return;
  }
  // 128 columns are 32 lanes of 16 bytes, a column's 4 bytes at word column / 32
  const int cols0 = lay.cols0, atoms = (cols0 + 127) / 128;
  sfs += product * (atoms * 512);
#pragma unroll
  for (int j = 0; j < kMxDigits; ++j) {
    const int c = j * Mp + m;
    if (c >= cols0) break;
    const int at = (c >> 7) * 512 + (c & 31) * 16 + ((c >> 5) & 3) * 4;
    sfs[at] = sf;
    sfs[remainders + at] = sf_rest;
  }
}

// ---- instructions ------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
               "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
// All of `threads` threads meet at a named barrier; true for each if p was for all.
__device__ __forceinline__ bool named_bar_and(int id, int threads, bool p) {
  uint32_t r;
  asm volatile(
      "{ .reg .pred a, b; setp.ne.u32 a, %1, 0; barrier.cta.red.and.pred b, %2, %3, a; selp.u32 %0, 1, 0, b; }"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(p)), "r"(id), "r"(threads)
      : "memory");
  return r != 0;
}
// The first stage after s whose bit is set in `again`; n if there is none.
__device__ __forceinline__ int again_after(const uint8_t* again, int n, int s) {
#pragma unroll 1
  for (++s; s < n; s = (s | 7) + 1) {
    const uint32_t b = static_cast<uint32_t>(again[s >> 3]) >> (s & 7);
    if (b) return s + __ffs(static_cast<int>(b)) - 1;
  }
  return n;
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mx_umma(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                        uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; .reg .b64 da, db; setp.ne.u32 p, %8, 0; mov.b64 da, {%1, %2}; mov.b64 db, {%3, %4};\n"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %5, [%6], [%7], p; }" ::"r"(d_tmem),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}

// What a row with infinities gives under a weight row: the sum of the infinities' products, an infinity or NaN as IEEE has it (the
// finite values next to them do not count). No one's hot path: one thread, all of K.
__device__ __noinline__ float infinite_sum(const void* x, int x_bf16, const uint8_t* w, const uint8_t* scale, int K) {
  float sum = 0.0f;
  for (int k = 0; k < K; ++k) {
    const uint32_t bits = x_bf16 ? bf16_at<true>(x, k) : bf16_at<false>(x, k);
    if ((bits & 0x7fffu) == 0x7f80u) sum += bf16_bits_to_f32(bits) * (e2m1_to_f32(w[k >> 1] >> (4 * (k & 1)) & 15u) * e4m3_to_f32(scale[k >> 4]));
  }
  return sum;
}

// ---- the product -------------------------------------------------------------------------------------------------------------
// ATOMS: 128-column pieces of a step's activation scales; TWO: two instructions per step.
// SUB: stages per slot of the rings. What bounds a product of few rows is neither copies nor products but what every role does once per
// slot (waits, commits, the meeting of the scale warps and their store to tensor memory: ~650 ns, where the copies of a stage take 370
// and its products 200), so up to 32 rows, where two or more slots of twice the size fit, a slot holds two stages: 28672 x 8192, 1 / 8 / 16 /
// 24 / 32 rows 42.4 / 43.4 / 44.7 / 48.0 / 50.3 -> 34.0 / 34.9 / 36.1 / 44.3 / 47.4 us; 14336 x 4096 and 4096 x 4096, 16 rows 17.7 / 16.5 ->
// 15.6 / 14.3. (Beyond, where a step is two instructions, a slot of two stages would take more than half of the shared memory.)
// COMPACT: the activations' scales come once per row, and the last chunk may have fewer rows (see mx_cut).
// Tensor memory columns of a stage's scales: 4 products x 4 columns of the weights', then 4 x 4 per piece of the activations'.
template <int ATOMS, bool TWO, int SUB, bool COMPACT>
__global__ void __launch_bounds__(kMxThreads, 1) tc_mx_kernel(const __grid_constant__ CUtensorMap wmap, const MxParams P) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int kSfCols = 16 + 16 * ATOMS;
  const int SW = P.SW, SX = P.SX, x_slot = P.lay[0].x_bytes, box_bytes = P.box_bytes;
  // The tensor core reads 128 rows from every box, whatever R is: behind the boxes come the scales and the activations.
  uint8_t* const sring = smem + static_cast<size_t>(SW) * SUB * box_bytes;
  uint8_t* const xring = sring + SUB * kMxScaleBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(xring + static_cast<size_t>(SX) * SUB * x_slot);
  const uint32_t bar0 = smem_u32(bars);
  auto w_full = [&](int s) { return bar0 + 8u * s; };                       // weights landed
  auto w_empty = [&](int s) { return bar0 + 8u * (SW + s); };               // products done
  auto x_full = [&](int s) { return bar0 + 8u * (2 * SW + s); };
  auto x_empty = [&](int s) { return bar0 + 8u * (2 * SW + SX + s); };
  auto s_full = [&](int b) { return bar0 + 8u * (2 * SW + 2 * SX + b); };       // scales b are in tensor memory
  auto s_empty = [&](int b) { return bar0 + 8u * (2 * SW + 2 * SX + 4 + b); };  // and their products are done
  auto d_full = [&](int b) { return bar0 + 8u * (2 * SW + 2 * SX + 8 + b); };   // accumulator b is complete
  auto d_empty = [&](int b) { return bar0 + 8u * (2 * SW + 2 * SX + 10 + b); };  // and has been read
  const uint32_t a_full = bar0 + 8u * (2 * SW + 2 * SX + 12);                    // `again` is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SW + 2 * SX + 13);
  // [chunks][groups]: the stages that a chunk multiplies again, from the preparation's bits per row
  uint8_t* const again = reinterpret_cast<uint8_t*>(tmem_slot + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_stages = P.K / kMxStageK;
  // a tile is a panel of weight rows times a chunk; the chunks of a panel are neighbours, so that its later readers find it in L2
  const int chunks = P.chunks;
  const int n_tiles = (P.N + P.R - 1) / P.R * chunks;
  const int tile_begin = static_cast<int>(static_cast<int64_t>(n_tiles) * blockIdx.x / gridDim.x);
  const int tile_end = static_cast<int>(static_cast<int64_t>(n_tiles) * (blockIdx.x + 1) / gridDim.x);
  const int groups = P.groups;
  // slot(s, second, rest) for each of a chunk's stages in turn (second: the other stage of a slot, n_stages if there is none), then for
  // those that go again; false as soon as one gives up
  auto all_slots = [&](int chunk, auto&& slot) __attribute__((always_inline)) {
    for (int s = 0; s < n_stages; s += SUB)
      if (!slot(s, SUB == 2 ? s + 1 : n_stages, false)) return false;
    if (!tc_wait(a_full, 0, P.status)) return false;
    const uint8_t* bits = again + chunk * groups;
    for (int s = again_after(bits, n_stages, -1); s < n_stages;) {
      const int second = SUB == 2 ? again_after(bits, n_stages, s) : n_stages;
      if (!slot(s, second, true)) return false;
      s = again_after(bits, n_stages, SUB == 2 ? second : s);
    }
    return true;
  };

  if (tid == 0) {
    mbar_init(a_full, 128);
    for (int s = 0; s < SW; ++s) {
      mbar_init(w_full(s), 1);
      mbar_init(w_empty(s), 1);
    }
    for (int s = 0; s < SX; ++s) {
      mbar_init(x_full(s), 1);
      mbar_init(x_empty(s), 1);
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(s_full(b), 4);
      mbar_init(s_empty(b), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(d_full(b), 1);
      mbar_init(d_empty(b), 4);
    }
    mbar_init_fence();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(tmem_slot), kTmemColumns);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 8) {
    // ================================ weights ================================
    pdl_trigger();
    if (lane == 0) {  // static: no wait
      asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
      Ring w;
      bool ok = true, wrapped = false;
      int issued = 0;
      for (int tile = tile_begin; tile < tile_end && ok; ++tile) {
        const int row = tile / chunks * P.R, chunk = tile % chunks;
        auto slot = [&](int s, int second, bool) __attribute__((always_inline)) {
          if (wrapped && !tc_wait(w_empty(w.slot), w.lap ^ 1u, P.status)) return false;
          const bool both = SUB == 2 && second < n_stages;
          const uint32_t dst = smem_u32(smem) + static_cast<uint32_t>(w.slot) * SUB * box_bytes;
          mbar_arrive_expect_tx(w_full(w.slot), (both ? 2 : 1) * P.R * 128);
          tile_g2s(dst, &wmap, s * 32, row, w_full(w.slot));
          if (both) tile_g2s(dst + box_bytes, &wmap, second * 32, row, w_full(w.slot));
          ++issued;
          w.advance(SW);
          wrapped |= w.slot == 0;
          return true;
        };
        ok = all_slots(chunk, slot);
      }
      if (!ok)  // the copies in flight land before the CTA leaves
        for (int i = max(0, issued - SW); i < issued; ++i) tc_wait(w_full(i % SW), (i / SW) & 1, P.status);
    }
  } else if (warp == 10) {
    // ================================ activations ================================
    if (lane == 0) {
      pdl_wait();  // prepared by the kernel before this one
      Ring x;
      bool ok = true, wrapped = false;
      int i = 0, chunk = tile_begin % chunks;
      for (int tile = tile_begin; tile < tile_end && ok; ++tile) {
        const uint8_t* src = P.xprep + chunk * P.chunk_bytes;
        const int x_bytes = P.lay[COMPACT && chunk + 1 == chunks].x_bytes;
        auto slot = [&](int s, int second, bool rest) __attribute__((always_inline)) {
          if (wrapped && !tc_wait(x_empty(x.slot), x.lap ^ 1u, P.status)) return false;
          const bool both = SUB == 2 && second < n_stages;
          const uint32_t dst = smem_u32(xring) + static_cast<uint32_t>(x.slot) * SUB * x_slot;
          const uint8_t* from = src + (rest ? P.remainders : 0);
          mbar_arrive_expect_tx(x_full(x.slot), (both ? 2 : 1) * x_bytes);
          bulk_g2s(dst, from + static_cast<size_t>(s) * x_bytes, x_bytes, x_full(x.slot));
          if (both) bulk_g2s(dst + x_slot, from + static_cast<size_t>(second) * x_bytes, x_bytes, x_full(x.slot));
          ++i;
          x.advance(SX);
          wrapped |= x.slot == 0;
          return true;
        };
        ok = all_slots(chunk, slot);
        if (++chunk == chunks) chunk = 0;
      }
      if (!ok)
        for (int j = max(0, i - SX); j < i; ++j) tc_wait(x_full(j % SX), (j / SX) & 1, P.status);
    }
  } else if (warp == 9) {
    // ================================ issuer ================================
    if (lane == 0) {
      // e2m1 x e2m1, ue4m3 scales, 128 rows
      const uint32_t idesc = (1u << 7) | (1u << 10) | (1u << 27);
      const uint32_t sbo = 128;
      const uint32_t a_hi = (1024u >> 4) | (1u << 14) | (2u << 29), b_hi = (sbo >> 4) | (1u << 14);
      const uint32_t a_lo0 = ((smem_u32(smem) & 0x3ffffu) >> 4) | (1u << 16);
      Ring w, x;
      bool ok = true;
      const uint32_t sf_mask = P.sf_turns - 1, sf_shift = P.sf_turns == 4 ? 2 : P.sf_turns == 2 ? 1 : 0;
      uint32_t i = 0;
      int chunk = tile_begin % chunks;
      for (int tile = tile_begin, t = 0; tile < tile_end && ok; ++tile, ++t) {
        const int buf = P.buffers == 2 ? t & 1 : 0, use = P.buffers == 2 ? t >> 1 : t;  // this accumulator's use-th use
        const MxLayout& L = P.lay[COMPACT && chunk + 1 == chunks];
        const uint32_t cols0 = L.cols0, cols1 = L.cols1, lbo = (cols0 + cols1) / 8 * 128;
        const uint32_t idesc0 = idesc | (cols0 >> 3 << 17), idesc1 = idesc | (cols1 >> 3 << 17);
        const uint32_t b_lo0 = ((smem_u32(xring) & 0x3ffffu) >> 4) | ((lbo >> 4) << 16);
        const uint32_t b_step = (2u * lbo) >> 4, b_second = cols0 / 8 * 128 >> 4;
        const uint32_t d_tmem = tmem_base + buf * (P.lay[0].cols0 + P.lay[0].cols1);
        if (use > 0 && !tc_wait(d_empty(buf), (use - 1) & 1, P.status)) break;
        tc_fence_after();
        auto slot = [&](int s, int second, bool rest) __attribute__((always_inline)) {
          const uint32_t turn = i & sf_mask;
          if (!tc_wait(x_full(x.slot), x.lap, P.status) || !tc_wait(w_full(w.slot), w.lap, P.status) || !tc_wait(s_full(turn), (i >> sf_shift) & 1, P.status)) {
            return false;
          }
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < SUB; ++h) {
            if (h > 0 && second >= n_stages) break;
            const uint32_t sfa = tmem_base + P.sf0 + (turn * SUB + h) * kSfCols, sfb = sfa + 16;
            const uint32_t x_at = ((static_cast<uint32_t>(x.slot) * SUB + h) * x_slot) >> 4;
            const uint32_t a_lo = a_lo0 + (((static_cast<uint32_t>(w.slot) * SUB + h) * box_bytes) >> 4), b_lo = b_lo0 + x_at;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint32_t adds = rest || (s | h | ks) ? 1u : 0u;
              mx_umma(d_tmem, a_lo + 2 * ks, a_hi, b_lo + ks * b_step, b_hi, idesc0, sfa + 4 * ks, sfb + 4 * ATOMS * ks, adds);
              if constexpr (TWO) mx_umma(d_tmem + cols0, a_lo + 2 * ks, a_hi, b_lo + ks * b_step + b_second, b_hi, idesc1, sfa + 4 * ks, sfb + 4 * ATOMS * ks, adds);
            }
          }
          umma_commit(w_empty(w.slot));
          umma_commit(x_empty(x.slot));
          umma_commit(s_empty(turn));
          w.advance(SW);
          x.advance(SX);
          ++i;
          return true;
        };
        ok = all_slots(chunk, slot);
        if (ok) umma_commit(d_full(buf));
        if (++chunk == chunks) chunk = 0;
      }
    }
  } else if (warp >= 4) {
    // ================================ weight scales ================================
    const int r = tid - 128;
    const int64_t pitch = P.K / 16;
    uint4 q[kAhead];
    auto scales_of = [&](int panel) -> const uint4* {  // this thread's row of a panel, null past the last
      const int n = panel * P.R + r;
      return r < P.R && n < P.N ? reinterpret_cast<const uint4*>(P.scale + n * pitch) : nullptr;
    };
    int panel = tile_begin / chunks, chunk = tile_begin % chunks;
    const uint4* scales = tile_begin < tile_end ? scales_of(panel) : nullptr;
#pragma unroll
    for (int i = 0; i < kAhead; ++i) q[i] = scales && i < n_stages ? __ldg(scales + i) : make_uint4(0, 0, 0, 0);
    // Lane l of each of the four warps holds rows l, 32 + l, 64 + l and 96 + l in tensor memory: every quarter has all 128 rows.
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + P.sf0;
    Ring w, x;
    bool ok = true;
    uint32_t count = 0;  // slots so far
    uint32_t x_rows[ATOMS] = {}, sf_off = 0;  // compact, the chunk's: the rows of columns lane, 32 + lane, ..., a byte each, and where their scales begin
    const uint32_t sf_mask = P.sf_turns - 1, sf_shift = P.sf_turns == 4 ? 2 : P.sf_turns == 2 ? 1 : 0;
    // One slot: this thread's scales of its stages to the tensor core (both: there is a second stage); `fetch` asks for the ones that
    // come later. (A warp whose wait gave up still comes to the meetings.)
    auto slot = [&](uint4 (&s)[SUB], bool both, auto&& fetch) __attribute__((always_inline)) {
      const uint32_t turn = count & sf_mask, use = count >> sf_shift;
      uint4* rows = reinterpret_cast<uint4*>(sring) + (count & 1) * SUB * 128;  // (two slots in turn: one meeting per slot is enough)
#pragma unroll
      for (int h = 0; h < SUB; ++h) {
        if (h > 0 && !both) break;
        if ((s[h].x | s[h].y | s[h].z | s[h].w) & 0x80808080u) {  // scales have no sign here: it goes to the block's values
          ok = ok && tc_wait(w_full(w.slot), w.lap, P.status);
          const uint32_t sc[4] = {s[h].x, s[h].y, s[h].z, s[h].w};
          uint8_t* box = smem + (static_cast<size_t>(w.slot) * SUB + h) * box_bytes + r * 128;
          for (int b = 0; b < 16 && ok && r < P.R; ++b)
            if (sc[b >> 2] >> (8 * (b & 3)) & 0x80u) {
              uint2* at = reinterpret_cast<uint2*>(box + (((b >> 1) ^ (r & 7)) << 4) + 8 * (b & 1));
              *at = make_uint2(at->x ^ 0x88888888u, at->y ^ 0x88888888u);
            }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads what this thread wrote
        }
        rows[h * 128 + r] = make_uint4(s[h].x & 0x7f7f7f7fu, s[h].y & 0x7f7f7f7fu, s[h].z & 0x7f7f7f7fu, s[h].w & 0x7f7f7f7fu);
      }
      fetch(s);
      __syncwarp();
      named_bar_sync(1, 128);
      uint32_t v[16], xv[ATOMS][16];
      auto read_rows = [&](int h) __attribute__((always_inline)) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 u = rows[h * 128 + 32 * c + lane];
          v[c] = u.x, v[4 + c] = u.y, v[8 + c] = u.z, v[12 + c] = u.w;
        }
      };
      auto read_x = [&](int h) __attribute__((always_inline)) {
        // The activations' scales lie behind their digits, as the four words of each lane and product or, compact, a word per product and row:
        // column c is a digit of row c % Mp, word q of a product is that of column 32 q + lane. (Words: the four products' of a row at once
        // would have to change places before they are stored.)
        const uint8_t* const xsf = xring + static_cast<size_t>(x.slot * SUB + h) * x_slot + (COMPACT ? sf_off : P.lay[0].sf_off);
#pragma unroll
        for (int q = 0; q < 4 * ATOMS; ++q) {
          if constexpr (COMPACT) {
            uint32_t row = x_rows[q / 4];
            asm volatile("" : "+r"(row));  // (taken out for each slot: the addresses of all words, kept, would take the next preparation's registers)
            const uint32_t* from = reinterpret_cast<const uint32_t*>(xsf + 4 * (row >> 8 * (q % 4) & 255u));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) xv[(4 * ATOMS * ks + q) / 16][(4 * ATOMS * ks + q) % 16] = from[ks * MxLayout::compact_rows(ATOMS == 2)];
          } else {
            const uint4 u = *reinterpret_cast<const uint4*>(xsf + 512 * q + 16 * lane);
            uint32_t* to = xv[q / 4] + 4 * (q % 4);
            to[0] = u.x, to[1] = u.y, to[2] = u.z, to[3] = u.w;
          }
        }
      };
      read_rows(0);
      ok = ok && tc_wait(x_full(x.slot), x.lap, P.status);
      read_x(0);  // before the wait for their place (the second stage's after: they would take more registers than there are)
      if (use > 0 && ok) ok = tc_wait(s_empty(turn), (use - 1) & 1, P.status);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < SUB; ++h) {
          if (h > 0 && !both) break;
          if (h > 0) read_rows(h), read_x(h);
          const uint32_t at = lane_addr + (turn * SUB + h) * kSfCols;
          tmem_st16(at, v);
#pragma unroll
          for (int a = 0; a < ATOMS; ++a) tmem_st16(at + 16 + 16 * a, xv[a]);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_full(turn));
      }
      x.advance(SX);
      w.advance(SW);
      ++count;
    };
    for (int tile = tile_begin; tile < tile_end; ++tile) {
      const bool turns = chunk + 1 == chunks;
      const uint4* const scales_next = tile + 1 >= tile_end ? nullptr : turns ? scales_of(panel + 1) : scales;
      const uint8_t* const bits = again + chunk * groups;
      if constexpr (COMPACT) {
        const MxLayout& L = P.lay[chunk + 1 == chunks];
        sf_off = L.sf_off;
#pragma unroll
        for (int q = 0, m = lane; q < 4 * ATOMS; ++q, m += 32) {
          while (m >= L.Mp) m -= L.Mp;
          x_rows[q / 4] = q % 4 ? x_rows[q / 4] | static_cast<uint32_t>(m) << 8 * (q % 4) : static_cast<uint32_t>(m);
        }
      }
      for (int s0 = 0; s0 < n_stages; s0 += kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; i += SUB) {
          if (s0 + i >= n_stages) break;
          uint4 now[SUB];
#pragma unroll
          for (int h = 0; h < SUB; ++h) now[h] = q[i + h];
          slot(now, SUB == 2 && s0 + i + 1 < n_stages, [&](uint4 (&)[SUB]) {  // stage s0 + i + kAhead, or stage i of the next tile
#pragma unroll
            for (int h = 0; h < SUB; ++h) {
              const bool here = s0 + i + h + kAhead < n_stages;
              const uint4* from = here ? scales : scales_next;
              if (from && (here || i + h < n_stages)) q[i + h] = __ldg(from + (here ? s0 + i + h + kAhead : i + h));
            }
          });
        }
      }
      if (!named_bar_and(1, 128, tc_wait(a_full, 0, P.status))) break;  // all four warps leave together
      // the stages that go again next: their scales are asked for a slot ahead
      auto scales_at = [&](int a) { return a < n_stages && scales ? __ldg(scales + a) : make_uint4(0, 0, 0, 0); };
      int a = again_after(bits, n_stages, -1), second = SUB == 2 ? again_after(bits, n_stages, a) : n_stages;
      uint4 ahead[SUB];
      ahead[0] = scales_at(a);
      if constexpr (SUB == 2) ahead[1] = scales_at(second);
      while (a < n_stages) {
        uint4 now[SUB];
#pragma unroll
        for (int h = 0; h < SUB; ++h) now[h] = ahead[h];
        const bool both = SUB == 2 && second < n_stages;
        a = again_after(bits, n_stages, SUB == 2 ? second : a);
        second = SUB == 2 ? again_after(bits, n_stages, a) : n_stages;
        slot(now, both, [&](uint4 (&)[SUB]) {
          ahead[0] = scales_at(a);
          if constexpr (SUB == 2) ahead[1] = scales_at(second);
        });
      }
      scales = scales_next;
      panel += turns, chunk = turns ? 0 : chunk + 1;
    }
  } else {
    // ================================ epilogue ================================
    const int r = tid;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    pdl_wait();  // y and the activation scales come from earlier kernels
    for (int i = tid; i < chunks * groups; i += 128) {
      const uint4* rows64 = reinterpret_cast<const uint4*>(P.again + static_cast<int64_t>(i) * kMaxRows);
      const int rows = min(P.chunk_rows, P.M - i / groups * P.chunk_rows);
      uint32_t any = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 u = rows64[q];
        const uint32_t four[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int z = 0; z < 4; ++z) {
          const int left = rows - 16 * q - 4 * z;  // rows among these four
          any |= left >= 4 ? four[z] : left > 0 ? four[z] & ((1u << (8 * left)) - 1u) : 0u;
        }
      }
      any |= any >> 16;
      again[i] = static_cast<uint8_t>(any | (any >> 8));
    }
    mbar_arrive(a_full);
    for (int tile = tile_begin, t = 0; tile < tile_end; ++tile, ++t) {
      const int buf = P.buffers == 2 ? t & 1 : 0, use = P.buffers == 2 ? t >> 1 : t;
      const int panel = tile / chunks, chunk = tile - panel * chunks, m0 = chunk * P.chunk_rows, rows = min(P.chunk_rows, P.M - m0);
      const int Mp = P.lay[COMPACT && chunk + 1 == chunks].Mp;
      const int n = panel * P.R + r;
      const bool live = r < P.R && n < P.N;
      const float inv_lo = lane < rows ? P.row_scale[m0 + lane] : 0.0f, inv_hi = 32 + lane < rows ? P.row_scale[m0 + 32 + lane] : 0.0f;
      const float bias = live && P.bias ? load_f32(P.bias, P.bias_dtype, n) : 0.0f;
      if (!tc_wait(d_full(buf), use & 1, P.status)) break;
      tc_fence_after();
      const uint32_t d_addr = lane_addr + buf * (P.lay[0].cols0 + P.lay[0].cols1);
      for (int c = 0; c < rows; c += 8) {
        uint32_t raw[kMxDigits][8];
#pragma unroll
        for (int j = 0; j < kMxDigits; ++j) tmem_ld8(d_addr + j * Mp + c, raw[j]);
        float old[8] = {};  // with beta: all eight asked for before the first is stored (see gemm_tc.cu)
        if (P.beta != 0.0f && live) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (c + i < rows) old[i] = load_f32(P.y, P.y_dtype, static_cast<int64_t>(m0 + c + i) * P.ld_y + n);
        }
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float inv = __shfl_sync(0xffffffffu, c < 32 ? inv_lo : inv_hi, (c + i) & 31);
          if (!live || c + i >= rows) continue;
          float sum = __uint_as_float(raw[kMxDigits - 1][i]), power = 1.0f;  // least first: the first digit's sum is rounded once
#pragma unroll
          for (int j = kMxDigits - 2; j >= 0; --j) {
            power *= kMxBase;
            sum = fmaf(__uint_as_float(raw[j][i]), power, sum);
          }
          float out = P.alpha * (P.global * (sum * inv) + bias);
          const int64_t at = static_cast<int64_t>(m0 + c + i) * P.ld_y + n;
          if (P.beta != 0.0f) out = fmaf(P.beta, old[i], out);
          store_from_f32(P.y, P.y_dtype, at, out);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d_empty(buf));
      // Rows with infinities: what is stored is all but their sum (NaN already if a scale is). (Left out of the stores above instead,
      // by a test of every output, they cost 1000 rows of 14336 x 4096 12 of 267 us.)
      auto infinite = [&](float inv) { return __ballot_sync(0xffffffffu, __float_as_uint(inv) == 0x80000000u); };
      uint64_t left = infinite(inv_lo) | static_cast<uint64_t>(infinite(inv_hi)) << 32;
      for (; left; left &= left - 1) {
        if (!live) continue;
        const int64_t m = m0 + __ffsll(static_cast<long long>(left)) - 1, n64 = n, at = m * P.ld_y + n;
        const float sum = infinite_sum(static_cast<const uint8_t*>(P.x) + m * P.ld_x * (P.x_bf16 ? 2 : 4), P.x_bf16, P.w + n64 * (P.K / 2), P.scale + n64 * (P.K / 16), P.K);
        store_from_f32(P.y, P.y_dtype, at, load_f32(P.y, P.y_dtype, at) + P.alpha * (P.global * sum));
      }
    }
  }
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem_base, kTmemColumns);
}

}  // namespace

// The most rows one launch takes (more come in launches of as many): bounds the workspace.
constexpr int kMxMaxRows = 1024;

// The fewest chunks of at most `most` rows that hold M, all of the same size (a multiple of 8) but the last.
constexpr int kMxChunkMost[] = {kMaxRows, 32, 16};
static int mx_chunk_rows(int M, int most) {
  const int chunks = (M + most - 1) / most;
  return ((M + chunks - 1) / chunks + 7) / 8 * 8;
}
// What a stage of a tile takes with so many activation rows, in tens of ns (28672 x 8192, two tiles per SM).
static int mx_stage_cost(int rows) { return rows <= 16 ? 49 : rows <= 24 ? 61 : rows <= 32 ? 66 : 88 + (rows - 40) * 11 / 10; }

// How P.M <= kMxMaxRows rows lie in the workspace when they go in chunks of at most `most`; returns the bytes. Rows that are split further
// than into chunks of 64 have their block scales there once, not for each of their digits, and a last chunk of fewer rows takes the room of
// those only: so no split takes more than the chunks of 64 do (which split, N decides, and who asks for the size has no N to give).
// Whole chunks keep the scales as they go to tensor memory: 28672 x 8192, 16 / 64 rows 36.0 / 78.0 us, compact 37.1 / 80.0.
static int64_t mx_cut(MxParams& P, int most) {
  const int stages = (P.K + kMxStageK - 1) / kMxStageK, whole = mx_chunk_rows(P.M, kMaxRows);
  P.chunk_rows = mx_chunk_rows(P.M, most);
  P.chunks = (P.M + P.chunk_rows - 1) / P.chunk_rows;
  P.lay[0] = P.lay[1] = MxLayout(P.chunk_rows);
  if (P.chunk_rows < whole) {
    const int as = MxLayout::compact_rows(P.lay[0].cols0 > 128);
    P.lay[0] = MxLayout(P.chunk_rows, as), P.lay[1] = MxLayout(P.M - (P.chunks - 1) * P.chunk_rows, as);
  }
  P.chunk_bytes = static_cast<int64_t>(stages) * P.lay[0].x_bytes;
  P.remainders = (P.chunks - 1) * P.chunk_bytes + static_cast<int64_t>(stages) * P.lay[1].x_bytes;
  P.groups = (stages + 7) / 8;
  return 2 * P.remainders + static_cast<int64_t>(P.chunks) * P.groups * kMaxRows + 4 * P.M + 256;
}

int64_t mx_workspace_bytes(int M, int K) {
  int64_t need = 0;
  MxParams P{};
  P.K = K;
  for (int rows : {std::min(M, kMxMaxRows), M % kMxMaxRows})  // a launch of the most rows, and the last one
    for (int most : kMxChunkMost) {                           // (which of them N decides)
      if (rows == 0) continue;
      P.M = rows;
      need = std::max(need, mx_cut(P, most));
    }
  return need;
}

// Everything about a launch that follows from the sizes (P.M, P.N, P.K) and the number of SMs. *sub: stages per slot, *smem: dynamic
// shared memory. even_rows: the weight rows per tile that deal N out evenly over the SMs.
static int mx_plan(MxParams& P, int sms, int even_rows, int* sub, size_t* smem) {
  constexpr int kMostFlags = 8192;  // of a chunk's groups, in shared memory: a split does not take room from the rings for more
  // Chunks of up to 64 rows, or of 32 or 16 where the busiest SM is done sooner with more, shorter tiles: a weight of few rows
  // leaves most SMs without a tile otherwise. (A row's bits do not depend on its chunk.) Replayed graphs, chunks of 64 and as the rule has it:
  // 4096 x 4096 at 64 rows 25.3 and 17.3 us, 1000 x 2048 at 64 rows 16.3 and 12.2, 293 x 2048 at 525 rows 21.6 and 15.1.
  auto turns_of = [&](int R, int chunk) { return (static_cast<int64_t>((P.N + R - 1) / R) * ((P.M + chunk - 1) / chunk) + sms - 1) / sms; };
  int64_t least = -1;
  int best = kMaxRows;
  for (int most : kMxChunkMost) {
    mx_cut(P, most);
    const int64_t cost = std::min(turns_of(kBM, P.chunk_rows), turns_of(even_rows, P.chunk_rows)) * mx_stage_cost(P.chunk_rows);
    if (least >= 0 && (cost >= least || P.chunks * P.groups > kMostFlags)) continue;
    least = cost, best = most;
  }
  mx_cut(P, best);
  const MxLayout& L = P.lay[0];
  // A tile takes as long with 128 weight rows as with fewer (its steps do), so what counts is the busiest SM's tiles; rows dealt
  // evenly where that is the same.
  P.R = turns_of(kBM, P.chunk_rows) < turns_of(even_rows, P.chunk_rows) ? kBM : even_rows;
  P.box_bytes = (P.R + 7) / 8 * 1024;
  // tensor memory from its end: the scales, then the accumulators, more than one of each where they fit
  const int cols = L.cols0 + L.cols1;
  const int sf_cols = 16 + 16 * ((L.cols0 + 127) / 128);
  *sub = L.cols1 ? 1 : 2;  // see the kernel
  P.sf_turns = cols + 4 * *sub * sf_cols <= kTmemColumns ? 4 : cols + 2 * *sub * sf_cols <= kTmemColumns ? 2 : 1;
  P.sf0 = kTmemColumns - P.sf_turns * *sub * sf_cols;
  P.buffers = 2 * cols <= P.sf0 ? 2 : 1;
  // A ring of as many stages of activations as of weights: a block of them, the same for every SM, travels as long as the weights
  // do. Where that is fewer than four, the weights keep six.
  const int tail = std::max(1024, 448 + P.chunks * P.groups);  // barriers, and the stages that go again
  const int room = 224 * 1024 - *sub * kMxScaleBytes - tail, box = *sub * P.box_bytes, block = *sub * L.x_bytes;
  const int even = room / (box + block);
  P.SX = *sub == 2 ? std::max(2, std::min(6, even)) : even >= 4 ? std::min(8, even) : std::max(2, std::min(4, (room - 6 * P.box_bytes) / L.x_bytes));
  P.SW = std::min(12, (room - P.SX * block) / box);
  if (P.SW < 2) return kNotSupported;
  *smem = std::max<size_t>(static_cast<size_t>(P.SW) * box + *sub * kMxScaleBytes + static_cast<size_t>(P.SX) * block + tail, 120 * 1024);
  return kOk;
}

int mx_plan_numbers(int M, int N, int K, int sms, int even_rows, int32_t* out) {
  MxParams P{};
  P.M = M, P.N = N, P.K = K;
  int sub = 0;
  size_t smem = 0;
  if (int e = mx_plan(P, sms, even_rows, &sub, &smem)) return e;
  const int64_t bytes = 2 * P.remainders + static_cast<int64_t>(P.chunks) * P.groups * kMaxRows + 4 * P.M;
  const int32_t v[] = {P.chunk_rows, P.chunks,  P.lay[0].cols0, P.lay[0].cols1, P.lay[0].x_bytes, P.lay[1].cols0, P.lay[1].x_bytes, sub, P.R,
                       P.SW,         P.SX,      P.sf_turns,     P.sf0,          P.buffers,        static_cast<int32_t>(smem), static_cast<int32_t>(bytes)};
  std::copy(v, v + 16, out);
  return kOk;
}

template <int ATOMS, bool TWO, bool COMPACT>
static int launch_mx(const MxParams& P, const CUtensorMap& wmap, size_t smem, int sms, cudaStream_t stream) {
  constexpr auto kernel = tc_mx_kernel<ATOMS, TWO, TWO ? 1 : 2, COMPACT>;
  if (int e = allow_big_smem<300 + ATOMS * 4 + TWO * 2 + COMPACT>(kernel)) return e;
  const int tiles = (P.N + P.R - 1) / P.R * P.chunks;
  return launch_kernel(kernel, dim3(std::min(tiles, sms)), dim3(kMxThreads), smem, stream, wmap, P);
}

// K % 256 == 0; weights, scales and workspace (mx_workspace_bytes) on 16 bytes.
int mx_product(const void* x, int x_dtype, int ld_x, const lx_weight& w, const void* bias, int bias_dtype, void* y, int y_dtype, int ld_y,
               int M, int N, int K, float alpha, float beta, void* workspace, int even_rows, cudaStream_t stream) {
  if (K % kMxStageK != 0) return kNotSupported;
  const bool x_bf16 = x_dtype == LX_BF16;
  const int sms = sm_count();
  if (!sms) return kInvalid;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  MxParams P{};
  P.x_bf16 = x_bf16, P.ld_x = ld_x;
  P.w = static_cast<const uint8_t*>(w.data);
  P.scale = static_cast<const uint8_t*>(w.scale);
  P.global = w.global;
  P.N = N, P.K = K;
  P.bias = bias, P.bias_dtype = bias_dtype;
  P.y_dtype = y_dtype, P.ld_y = ld_y;
  P.alpha = alpha, P.beta = beta;
  P.status = status_word();
  P.xprep = ws;
  for (int first = 0; first < M; first += kMxMaxRows) {
    P.M = std::min(kMxMaxRows, M - first);
    int sub = 0;
    size_t smem = 0;
    if (int e = mx_plan(P, sms, even_rows, &sub, &smem)) return e;
    uint8_t* again = ws + 2 * P.remainders;
    P.again = again;
    float* row_scale = reinterpret_cast<float*>(again + static_cast<int64_t>(P.chunks) * P.groups * kMaxRows);
    P.row_scale = row_scale;
    P.y = static_cast<uint8_t*>(y) + static_cast<int64_t>(first) * ld_y * (y_dtype == LX_BF16 ? 2 : 4);
    const void* xrow = static_cast<const uint8_t*>(x) + static_cast<int64_t>(first) * ld_x * (x_bf16 ? 2 : 4);
    P.x = xrow;
    alignas(64) CUtensorMap wmap;
    if (int e = make_tile_map(&wmap, w.data, K / 2, N, 128, P.R, 4, true)) return e;
    if (int e = launch_kernel(x_bf16 ? mx_prep_kernel<true> : mx_prep_kernel<false>, dim3(P.groups, P.M), dim3(kPrepThreads), 0, stream, xrow, ld_x, K,
                              P.chunks, P.chunk_rows, P.chunk_bytes, P.lay[0], P.lay[1], ws, P.remainders, again, row_scale))
      return e;
    const int e = P.lay[0].cols0 <= 128 ? (P.lay[0].sf_rows ? launch_mx<1, false, true>(P, wmap, smem, sms, stream) : launch_mx<1, false, false>(P, wmap, smem, sms, stream))
                  : P.lay[0].cols1      ? launch_mx<2, true, false>(P, wmap, smem, sms, stream)
                  : P.lay[0].sf_rows    ? launch_mx<2, false, true>(P, wmap, smem, sms, stream)
                                        : launch_mx<2, false, false>(P, wmap, smem, sms, stream);
    if (e) return e;
  }
  return kOk;
}

}  // namespace b200
