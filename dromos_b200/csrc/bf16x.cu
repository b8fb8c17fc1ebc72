// The lossless bf16 encoding LX_W_BF16X: size query, encoder and decoder (the ABI of lernex/dromos
// engine/cuda/kernels.h:574-583; the layout is documented in engine/cuda/bf16x.cuh:13-28 and restated in stream.cuh).
//
// Encoding a row: per 128 values the largest exponent is the block's base; a value keeps sign|mantissa in one byte and
// base - exponent as a 4-bit code; a value more than 15 binades below its base is a patch (position << 8 | exponent),
// listed in ascending position in the row's header slots, or in an overflow record after all rows when the row has
// more patches than slots. Rows are independent except for where their overflow records land, which is fixed by
// a prefix sum over the rows' record sizes in row order, so the bytes never depend on scheduling.
#include <algorithm>

#include "launch.cuh"

namespace b200 {
namespace {

constexpr int kBlock = 256;
constexpr int kWarpsPerBlock = kBlock / 32;
// Iterations of 256 values a warp keeps in flight. What bounds these kernels is HBM once a lane's loads are 16 bytes and
// several are in flight: with 2-byte loads, one 128-value block at a time, sizing, encoding and decoding 14336 x 4096 took
// 390 us in all, 6.3 x the time its bytes take; with both 153; with sizing and encoding in one pass (lx_b200_bf16x_encode_sized) 102, of which
// ~76 are the matrix read once and written once and the records once each way, the rest a round trip to the host (the size is a
// host number) and launches.
constexpr int kInFlight = 4;

__host__ __device__ inline int64_t record_bytes(int64_t patches) { return (4 * (patches + 2) + 7) / 8 * 8; }

// The eight values of a row from k0 on, packed as they lie in memory, zero past K. VEC: rows of whole 16-byte words.
template <bool VEC>
__device__ __forceinline__ uint4 load8(const uint16_t* __restrict__ src, int k0, int K) {
  if constexpr (VEC) return k0 < K ? __ldg(reinterpret_cast<const uint4*>(src + k0)) : make_uint4(0, 0, 0, 0);
  uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (k0 + j < K) w[j >> 1] |= static_cast<uint32_t>(__ldg(src + k0 + j)) << (16 * (j & 1));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// A lane's eight values against the block of 128 its half of the warp holds (16 lanes x 8 values): the block's base, and
// which of the lane's values are patches. Exponents stay where they are in the bf16 words (bits 7..14 of each half).
constexpr uint32_t kExpBits = 0x7f807f80u;
__device__ __forceinline__ uint32_t block_base(const uint4& v) {
  const uint32_t m = __vmaxu2(__vmaxu2(v.x & kExpBits, v.y & kExpBits), __vmaxu2(v.z & kExpBits, v.w & kExpBits));
  uint32_t base = max(m & 0xffffu, m >> 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) base = max(base, __shfl_xor_sync(0xffffffffu, base, o));
  return base;  // exponent << 7
}
__device__ __forceinline__ uint32_t patch_mask(const uint4& v, uint32_t base, int live) {
  const uint32_t lo = __vminu2(__vminu2(v.x & kExpBits, v.y & kExpBits), __vminu2(v.z & kExpBits, v.w & kExpBits));
  if (min(lo & 0xffffu, lo >> 16) + (15u << 7) >= base) return 0;
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t mask = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t e = (w[j >> 1] >> (16 * (j & 1))) & 0x7f80u;
    if (j < live && e + (15u << 7) < base) mask |= 1u << j;
  }
  return mask;
}

// One warp per row: *area += bytes of the row's overflow record, for rows with more patches than slots. (A sum of whole
// numbers: the order in which rows add does not matter.)
template <bool VEC>
__global__ void __launch_bounds__(kBlock) count_kernel(const uint16_t* __restrict__ w, int64_t rows, int K, unsigned long long* __restrict__ area) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const uint16_t* src = w + row * K;
  int n = 0;
  for (int k_base = 0; k_base < K; k_base += 256 * kInFlight) {
    uint4 v[kInFlight];
#pragma unroll
    for (int i = 0; i < kInFlight; ++i) v[i] = load8<VEC>(src, k_base + 256 * i + 8 * lane, K);
#pragma unroll
    for (int i = 0; i < kInFlight; ++i) n += __popc(patch_mask(v[i], block_base(v[i]), K - (k_base + 256 * i + 8 * lane)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0 && n > x16::patch_slots(K)) atomicAdd(area, static_cast<unsigned long long>(record_bytes(n)));
}

// Where a lane's patches go in its row's list: after those of the lanes below it. Returns the warp's count.
__device__ __forceinline__ int place_patches(uint32_t mask, int lane, int& before) {
  const int n = __popc(mask);
  int upto = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  before = upto - n;
  return __shfl_sync(0xffffffffu, upto, 31);
}

// One warp per row: writes the row's record, patches in its own slots. A row that has more patches than slots is left with
// 0x80000000 | its patches in slot 0 and adds its record's bytes to *area; the two kernels below finish such rows. So the
// common matrix is read once, and nothing but *area has to be known before.
// A lane holds eight consecutive values: eight sign|mantissa bytes, and one word of codes (byte j holds value j low and
// value 4 + j high), so a block's 192 bytes leave in 16 stores of 8 and 16 of 4 bytes.
template <bool VEC>
__global__ void __launch_bounds__(kBlock) encode_kernel(const uint16_t* __restrict__ w, int64_t rows, int K, uint8_t* __restrict__ out,
                                                        unsigned long long* __restrict__ area) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const int H = x16::header_bytes(K), P = x16::patch_slots(K), B = x16::blocks(K);
  const uint16_t* src = w + row * K;
  uint8_t* rec = out + row * x16::row_bytes(K);
  uint32_t* slots = reinterpret_cast<uint32_t*>(rec);
  // header: empty slots, zero padding after the base bytes
  for (int i = lane; i < P; i += 32) slots[i] = x16::kNoPatch;
  for (int i = 4 * P + B + lane; i < H; i += 32) rec[i] = 0;
  __syncwarp();
  int placed = 0;  // patches so far (the same in every lane)
  for (int k_base = 0; k_base < K; k_base += 256 * kInFlight) {
    uint4 v[kInFlight];
#pragma unroll
    for (int i = 0; i < kInFlight; ++i) v[i] = load8<VEC>(src, k_base + 256 * i + 8 * lane, K);
    uint32_t base_byte = 0;  // lane l keeps the base of block l of this iteration's
#pragma unroll
    for (int i = 0; i < kInFlight; ++i) {
      const int k0 = k_base + 256 * i + 8 * lane;
      const uint32_t base = block_base(v[i]);
      const uint32_t mask = patch_mask(v[i], base, K - k0);
      const uint32_t b0 = __shfl_sync(0xffffffffu, base, 0), b1 = __shfl_sync(0xffffffffu, base, 16);
      if (lane == 2 * i) base_byte = b0 >> 7;
      if (lane == 2 * i + 1) base_byte = b1 >> 7;
      const uint32_t words[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      uint32_t sm[4], d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sm[j] = ((words[j] >> 8) & 0x00800080u) | (words[j] & 0x007f007fu);
        d[j] = (base * 0x10001u - (words[j] & kExpBits)) >> 7;  // per half: base - exponent, below 16 unless patched
      }
      if (__any_sync(0xffffffffu, mask)) {
        int before;
        const int n = place_patches(mask, lane, before);
        int at = placed + before;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (mask >> j & 1) {
            if (at < P) slots[at] = (static_cast<uint32_t>(k0 + j) << 8) | ((words[j >> 1] >> (16 * (j & 1) + 7)) & 0xffu);
            ++at;
            d[j >> 1] &= j & 1 ? 0x0000ffffu : 0xffff0000u;  // a patched value's code is 0
          }
        }
        placed += n;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (k0 + j >= K) d[j >> 1] &= j & 1 ? 0x0000ffffu : 0xffff0000u;  // so is one past the row's end
      if (k0 < 128 * B) {
        uint8_t* blk = rec + H + static_cast<int64_t>(k0 >> 7) * 192;
        *reinterpret_cast<uint2*>(blk + (k0 & 127)) = make_uint2(__byte_perm(sm[0], sm[1], 0x6420), __byte_perm(sm[2], sm[3], 0x6420));
        *reinterpret_cast<uint32_t*>(blk + 128 + ((k0 & 127) >> 1)) = __byte_perm(d[0] | (d[2] << 4), d[1] | (d[3] << 4), 0x6420);
      }
    }
    if (lane < 2 * kInFlight && k_base / 128 + lane < B) rec[4 * P + k_base / 128 + lane] = static_cast<uint8_t>(base_byte);
  }
  if (placed <= P) return;
  __syncwarp();
  for (int i = lane; i < P; i += 32) slots[i] = i == 0 ? 0x80000000u | static_cast<uint32_t>(placed) : x16::kNoPatch;
  if (lane == 0) atomicAdd(area, static_cast<unsigned long long>(record_bytes(placed)));
}

__device__ __forceinline__ bool overflowed(uint32_t slot0) { return slot0 != x16::kNoPatch && (slot0 & 0x80000000u); }

// One CTA, after encode_kernel: the places of the overflow records, in row order (an exclusive prefix sum over the counts
// that encode_kernel left), take the place of the counts in slot 0. room: the bytes there are for records; a row whose record would end
// past them is left without its patches.
__global__ void __launch_bounds__(1024) place_records_kernel(uint8_t* __restrict__ out, int64_t rows, int64_t rb, int64_t room) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  __shared__ int64_t warp_sum_of[32];
  const int t = threadIdx.x, lane = t & 31;
  const int64_t per = (rows + 1023) / 1024;
  const int64_t r0 = min(rows, t * per), r1 = min(rows, r0 + per);
  auto slot0 = [&](int64_t r) { return reinterpret_cast<uint32_t*>(out + r * rb); };
  int64_t sum = 0;
  for (int64_t r = r0; r < r1; ++r) {
    const uint32_t s = *slot0(r);
    if (overflowed(s)) sum += record_bytes(s & 0x7fffffffu);
  }
  int64_t upto = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t v = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += v;
  }
  if (lane == 31) warp_sum_of[t >> 5] = upto;
  __syncthreads();
  int64_t run = upto - sum;
  for (int i = 0; i < (t >> 5); ++i) run += warp_sum_of[i];
  for (int64_t r = r0; r < r1; ++r) {
    const uint32_t s = *slot0(r);
    if (!overflowed(s)) continue;
    const int64_t at = run;
    run += record_bytes(s & 0x7fffffffu);
    *slot0(r) = run <= room ? 0x80000000u | static_cast<uint32_t>((rows * rb + at - r * rb) / 8) : x16::kNoPatch;  // from the row's own start, in 8 bytes
  }
}

// After encode_kernel, where the overflow records do not fit: no row is left with a count where a reader expects a record's place.
__global__ void __launch_bounds__(kBlock) drop_counts_kernel(uint8_t* __restrict__ out, int64_t rows, int64_t rb) {
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (row >= rows) return;
  uint32_t* slot0 = reinterpret_cast<uint32_t*>(out + row * rb);
  if (overflowed(*slot0)) *slot0 = x16::kNoPatch;
}

// One warp per row that has an overflow record: reads the row again and writes the record.
template <bool VEC>
__global__ void __launch_bounds__(kBlock) overflow_kernel(const uint16_t* __restrict__ w, int64_t rows, int K, uint8_t* __restrict__ out) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  uint8_t* rec = out + row * x16::row_bytes(K);
  const uint32_t s0 = *reinterpret_cast<const uint32_t*>(rec);
  if (!overflowed(s0)) return;
  uint32_t* list = reinterpret_cast<uint32_t*>(rec + static_cast<int64_t>(s0 & 0x7fffffffu) * 8);
  const uint16_t* src = w + row * K;
  int placed = 0;
  for (int k_base = 0; k_base < K; k_base += 256) {
    const int k0 = k_base + 8 * lane;
    const uint4 v = load8<VEC>(src, k0, K);
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
    const uint32_t mask = patch_mask(v, block_base(v), K - k0);
    int before;
    const int n = place_patches(mask, lane, before);
    int at = placed + before;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (mask >> j & 1) list[1 + at++] = (static_cast<uint32_t>(k0 + j) << 8) | ((words[j >> 1] >> (16 * (j & 1) + 7)) & 0xffu);
    placed += n;
  }
  if (lane == 0) {
    list[0] = static_cast<uint32_t>(placed);
    list[placed + 1] = x16::kNoPatch;
    if (placed & 1) list[placed + 2] = 0;  // padding to whole 8 bytes
  }
}

// One warp per row: every value from its byte, code and base, then the row's patches over them. VEC: records on 8-byte
// boundaries, rows of whole 16-byte words; a lane takes eight values (8 bytes, one word of codes) and stores 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(kBlock) decode_kernel(const uint8_t* __restrict__ data, int64_t rows, int K,
                                                        uint16_t* __restrict__ w) {
  // no early trigger: what this kernel writes may be the weight of the next product, whose kernels read weights
  // before their own wait
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const int H = x16::header_bytes(K), P = x16::patch_slots(K);
  const uint8_t* rec = data + row * x16::row_bytes(K);
  uint16_t* dst = w + row * K;
  if constexpr (VEC) {
    for (int k_base = 0; k_base < K; k_base += 256 * kInFlight) {
      uint2 sm[kInFlight];
      uint32_t codes[kInFlight], base[kInFlight];
#pragma unroll
      for (int i = 0; i < kInFlight; ++i) {
        const int k0 = k_base + 256 * i + 8 * lane, b = k0 >> 7, off = k0 & 127;
        if (k0 >= K) continue;
        const uint8_t* blk = rec + H + static_cast<int64_t>(b) * 192;
        sm[i] = __ldg(reinterpret_cast<const uint2*>(blk + off));
        codes[i] = __ldg(reinterpret_cast<const uint32_t*>(blk + 128 + (off >> 1)));
        base[i] = __ldg(rec + 4 * P + b);
      }
#pragma unroll
      for (int i = 0; i < kInFlight; ++i) {
        const int k0 = k_base + 256 * i + 8 * lane;
        if (k0 >= K) continue;
        const uint32_t b2 = base[i] * 0x10001u | 0x01000100u;  // the guard bit keeps a half's borrow to itself
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t s = __byte_perm(j < 2 ? sm[i].x : sm[i].y, 0, j & 1 ? 0x4342 : 0x4140);
          const uint32_t c = (__byte_perm(codes[i], 0, j & 1 ? 0x4342 : 0x4140) >> (j < 2 ? 0 : 4)) & 0x000f000fu;
          o[j] = ((s & 0x00800080u) << 8) | (((b2 - c) & 0x00ff00ffu) << 7) | (s & 0x007f007fu);
        }
        *reinterpret_cast<uint4*>(dst + k0) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  } else {
    for (int k = lane; k < K; k += 32) {
      const int b = k >> 7, off = k & 127;
      const uint8_t* blk = rec + H + static_cast<int64_t>(b) * 192;
      const uint32_t sm = blk[off];
      const uint32_t cb = blk[128 + (off >> 3) * 4 + (off & 3)];
      const uint32_t e = (rec[4 * P + b] - ((off & 4) ? cb >> 4 : cb & 15u)) & 0xffu;
      dst[k] = static_cast<uint16_t>(((sm & 0x80u) << 8) | (e << 7) | (sm & 0x7fu));
    }
  }
  __syncwarp();
  const uint32_t* list = reinterpret_cast<const uint32_t*>(rec);
  int n = P;
  const uint32_t s0 = list[0];
  if (overflowed(s0)) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(rec + static_cast<int64_t>(s0 & 0x7fffffffu) * 8);
    n = static_cast<int>(r[0]);
    list = r + 1;
  }
  for (int i = lane; i < n; i += 32) {
    const uint32_t p = list[i];
    if (p == x16::kNoPatch) continue;
    const uint32_t k = p >> 8;
    if (k < static_cast<uint32_t>(K)) dst[k] = static_cast<uint16_t>((dst[k] & 0x807fu) | ((p & 0xffu) << 7));
  }
}

dim3 row_grid(int64_t rows) { return dim3(static_cast<unsigned>((rows + kWarpsPerBlock - 1) / kWarpsPerBlock)); }
bool whole_rows(const void* w, int K) { return K % 8 == 0 && aligned(w, 16); }

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" int64_t lx_bf16x_row_bytes(int K) { return K > 0 && K < (1 << 23) ? x16::row_bytes(K) : -1; }

extern "C" int64_t lx_bf16x_bytes(const void* w, int64_t rows, int K, void* stream) {
  if (rows <= 0 || K <= 0 || K >= (1 << 23) || !w) return -static_cast<int64_t>(kInvalid);
  ResultWord area(static_cast<cudaStream_t>(stream));
  int e = area.status;
  if (!e)
    e = launch_kernel(whole_rows(w, K) ? count_kernel<true> : count_kernel<false>, row_grid(rows), dim3(kBlock), 0, area.stream,
                      static_cast<const uint16_t*>(w), rows, K, area.dev);
  unsigned long long bytes = 0;
  if (!e) e = area.read(&bytes);
  if (e) return -static_cast<int64_t>(e);
  return rows * x16::row_bytes(K) + static_cast<int64_t>(bytes);
}

// The rows, and what the whole encoding takes (*total, as lx_bf16x_bytes answers): rows with more patches than slots are left with their counts.
static int encode_rows(const void* w, int64_t rows, int K, void* out, int64_t* total, cudaStream_t stream) {
  ResultWord area(stream);
  if (area.status) return area.status;
  if (int e = launch_kernel(whole_rows(w, K) ? encode_kernel<true> : encode_kernel<false>, row_grid(rows), dim3(kBlock), 0, area.stream,
                            static_cast<const uint16_t*>(w), rows, K, static_cast<uint8_t*>(out), area.dev))
    return e;
  unsigned long long bytes = 0;
  if (int e = area.read(&bytes)) return e;
  *total = rows * x16::row_bytes(K) + static_cast<int64_t>(bytes);
  return kOk;
}
// The overflow records of encoded rows, which take the place of their counts.
static int encode_records(const void* w, int64_t rows, int K, void* out, int64_t out_bytes, cudaStream_t stream) {
  const int64_t rb = x16::row_bytes(K);
  auto* dst = static_cast<uint8_t*>(out);
  if (int e = launch_kernel(place_records_kernel, dim3(1), dim3(1024), 0, stream, dst, rows, rb, out_bytes - rows * rb)) return e;
  return launch_kernel(whole_rows(w, K) ? overflow_kernel<true> : overflow_kernel<false>, row_grid(rows), dim3(kBlock), 0, stream, static_cast<const uint16_t*>(w), rows,
                       K, dst);
}

// A buffer too small for the overflow records is refused after the rows themselves (which fit) have been written: whether it is, only the
// encoder finds out, and counting first reads the matrix once more (25 us of 14336 x 4096). Such rows are left without their patches.
extern "C" int lx_bf16x_encode(const void* w, int64_t rows, int K, void* out, int64_t out_bytes, void* stream) {
  if (rows <= 0) return kOk;
  const int64_t rb = K > 0 && K < (1 << 23) ? x16::row_bytes(K) : 0;
  if (!rb || !w || !out || !aligned(out, 8) || out_bytes < rows * rb) return kInvalid;
  auto s = static_cast<cudaStream_t>(stream);
  int64_t total = 0;
  if (int e = encode_rows(w, rows, K, out, &total, s)) return e;
  if (total == rows * rb) return kOk;
  if (total <= out_bytes) return encode_records(w, rows, K, out, out_bytes, s);
  const int e = launch_kernel(drop_counts_kernel, dim3(static_cast<unsigned>((rows + kBlock - 1) / kBlock)), dim3(kBlock), 0, s, static_cast<uint8_t*>(out), rows, rb);
  return e ? e : kInvalid;
}

// Sizing and encoding in one call, the matrix read once: few matrices have overflow records at all, so a caller begins with a buffer of
// rows * lx_bf16x_row_bytes(K). One that turns out too small keeps the encoded rows, and lx_b200_bf16x_encode_rest takes them from there
// (copied, 3 bytes per value; encoded again, 3.5 and the host waits once more).
extern "C" int lx_b200_bf16x_encode_sized(const void* w, int64_t rows, int K, void* out, int64_t out_bytes, int64_t* bytes, void* stream) {
  const int64_t rb = K > 0 && K < (1 << 23) ? x16::row_bytes(K) : 0;
  if (rows <= 0 || !rb || !w || !out || !bytes || !aligned(out, 8) || out_bytes < rows * rb) return kInvalid;
  auto s = static_cast<cudaStream_t>(stream);
  if (int e = encode_rows(w, rows, K, out, bytes, s)) return e;
  if (*bytes == rows * rb) return kOk;
  return *bytes <= out_bytes ? encode_records(w, rows, K, out, out_bytes, s) : LX_B200_ERR_SCRATCH;
}
extern "C" int lx_b200_bf16x_encode_rest(const void* w, int64_t rows, int K, const void* encoded, void* out, int64_t out_bytes, void* stream) {
  const int64_t rb = K > 0 && K < (1 << 23) ? x16::row_bytes(K) : 0;
  if (rows <= 0 || !rb || !w || !encoded || !out || !aligned(out, 8) || out_bytes < rows * rb) return kInvalid;
  auto s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = out == encoded ? cudaSuccess : cudaMemcpyAsync(out, encoded, static_cast<size_t>(rows * rb), cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return static_cast<int>(e);
  }
  return encode_records(w, rows, K, out, out_bytes, s);
}

extern "C" int lx_bf16x_decode(const void* data, int64_t rows, int K, void* w, void* stream) {
  if (rows <= 0) return kOk;
  if (K <= 0 || K >= (1 << 23) || !data || !w) return kInvalid;
  // (rows of less than a block, eight values a lane, leave most lanes idle: 50000 x 64 12.9 us, one value a lane 10.8; 40000 x 128 10.6 and 11.2)
  return launch_kernel(whole_rows(w, K) && K >= 128 && aligned(data, 8) ? decode_kernel<true> : decode_kernel<false>, row_grid(rows), dim3(kBlock), 0,
                       static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(data), rows, K, static_cast<uint16_t*>(w));
}
