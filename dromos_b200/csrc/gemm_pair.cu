// lx_gemm_w with more activation rows than one pass of the decode product takes (prefill and large batches): BF16, INT8
// and FP8 weights on pairs of SMs (tcgen05 cta_group::2).
//
// The decode product (gemm_tc.cu) re-reads the weights for every 64 activation rows and multiplies tiles of 64 columns: past
// 64 rows it is bound by neither HBM nor the tensor pipe. Here a tile is 256 weight rows x up to 256 columns of
// activations, the two CTAs of a cluster hold 128 weight rows and half of the columns each, and one product of the pair
// reads both halves: per 32 bytes of K an SM fetches 8 KB for 128 cycles of its tensor pipe, where two lone CTAs of
// 128 x 256 would fetch 12 KB each (96 bytes per cycle and SM, more than L2 gives 148 SMs). No multicast loads.
//
//   * The math per format is the decode product's: the weights as stored, the activations as digit planes (BF16: the bf16
//     value; FP8: two e4m3 digits; INT8: three int8 digits) or one quantized plane, K in the same order and the same
//     32-byte products, so that a row's bits do not depend on whether it came alone or with 1000 others.
//   * Activations lie row-major by plane, [planes][rows][K], and come as 128-byte-swizzled tile copies like the weights.
//     bf16 activations of a BF16 product are read where the caller has them when their rows are 16-byte aligned;
//     everything else is prepared into the workspace by pair_prep_kernel.
//   * Roles per CTA: warps 0..7 epilogue (two per quarter of the accumulator's lanes, each half of the columns), warps 8 and 10
//     one producer thread each (weights, activations), warp 9 of the pair's first CTA one issuing thread. Ring of stages of 128 bytes of K; a stage's
//     bytes of both CTAs complete on the first CTA's barrier, tcgen05.commit frees it in both. Two accumulators of 256
//     columns, so that a tile's epilogue runs under the next tile's products.
//   * Tiles are dealt out in turn, the columns of a weight panel next to each other, so that its later readers find it in L2.
//
// Measured (replayed graphs; before: passes of 64 rows through gemm_tc.cu): 14336 x 4096, BF16, 512 rows 50.7 us = 1.19 PFLOP/s
// (was 230), FP8 under FP8 math, 1000 rows, 61.5 us = 1.9 PFLOP/s (was 280). With every pair busy for whole waves (18944
// weight rows, 1024 rows) BF16 runs at 1.42 PFLOP/s, 0.87 of the measured cuBLAS burst, and a wave more costs 26.5 us against
// 24.4 at that rate; what is left of a call is ~10 us of head and last epilogue, and the waves that 112 tiles of 74 pairs
// leave three quarters full. Without three in four of the products a wave takes 14 us, L2's 20 TB/s.
//
// Every wait is bounded; a role that gives up leaves its loop, the producer then waits (bounded) for the copies in flight,
// and both CTAs of a pair meet before either leaves.
#include "tc.cuh"

namespace b200 {
namespace {

constexpr int kPairTile = 256;      // weight rows per tile, 128 per CTA
constexpr int kPairCols = 256;      // the most accumulator columns per tile
constexpr int kPairStageK = 128;    // bytes of K per stage: one swizzled box
constexpr int kPairEpilogueWarps = 8, kPairThreads = (kPairEpilogueWarps + 3) * 32;
constexpr int kPairABytes = 128 * kPairStageK;

struct PairParams {
  const float* row_scale;   // f32 [N] (INT8 / FP8), null for BF16
  const float* inv_scales;  // per activation row, null when all are 1
  int N, M, n_stages;
  int half;                 // activation rows per CTA and tile, a multiple of 8
  int x_rows;               // rows from one plane to the next in the activation map
  float digit;
  int col_tiles, tiles;
  int b_bytes;              // planes * half * 128
  int S;                    // ring depth
  const void* bias;
  int bias_dtype;
  void* y;
  int y_dtype, ld_y;
  float alpha, beta;
  int* status;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A tile copy of this CTA that completes on the barrier at the same offset in the pair's first CTA.
__device__ __forceinline__ void pair_tile_g2s(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(bar & 0xfeffffffu)
      : "memory");
}
// One arrival on the barrier at this offset in the pair's first CTA.
__device__ __forceinline__ void pair_arrive_first(uint32_t bar) {
  asm volatile(
      "{ .reg .b32 a; mapa.shared::cluster.u32 a, %0, 0;\n"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a]; }" ::"r"(bar)
      : "memory");
}
// One arrival on the barrier at this offset in both CTAs when every product issued so far is done.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(static_cast<uint16_t>(3))
               : "memory");
}
template <int kAct>
__device__ __forceinline__ void pair_umma(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
#define B200_PAIR_UMMA(KIND)                                                                                                    \
  asm volatile(                                                                                                                 \
      "{ .reg .pred p; .reg .b64 da, db; setp.ne.u32 p, %5, 0; mov.b64 da, {%1, %3}; mov.b64 db, {%2, %3};\n"                   \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], da, db, %4, p; }" ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), \
      "r"(accumulate)                                                                                                           \
      : "memory")
  if constexpr (kAct == kActE4m3) B200_PAIR_UMMA("f8f6f4");
  else if constexpr (kAct == kActS8) B200_PAIR_UMMA("i8");
  else B200_PAIR_UMMA("f16");
#undef B200_PAIR_UMMA
}

// ---- activations, row-major by plane ------------------------------------------------------------------------------------
// Block (chunk, u): 128 threads, each 16 bytes of K of every plane of activation row u (as tc_prep_kernel, which writes
// core-matrix order); plane j of row u starts at out + (j * rows + u) * ld.
template <int ACT, bool XBF, int MODE>
__global__ void __launch_bounds__(128) pair_prep_kernel(const void* __restrict__ x, int ld_x, int rows, int K, int planes, int ld,
                                                        uint8_t* __restrict__ out, float* __restrict__ inv_scales) {
  constexpr int kElem = act_elem(ACT), V = 16 / kElem;
  constexpr bool QUANT = MODE == kPrepQuant, AS_BF16 = XBF || MODE == kPrepRound;
  pdl_trigger();
  pdl_wait();  // the kernel before this one may still be reading the workspace
  __shared__ float part[4];
  const int u = blockIdx.y, tid = threadIdx.x;
  const int k0 = (blockIdx.x * 128 + tid) * V;
  const bool in_range = k0 < K;
  const int64_t row = static_cast<int64_t>(u) * ld_x;
  const bool aligned16 = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ld_x % (XBF ? 8 : 4) == 0;
  float v[V];
  if (in_range) {
    load_values<XBF, V>(x, row, k0, K, aligned16, v);
    if constexpr (MODE == kPrepRound) {
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = bf16_bits_to_f32(f32_to_bf16_bits(v[i]));
    }
  }
  float sc = 1.0f, back = 1.0f;
  if constexpr (ACT != kActBf16) {
    float a = warp_max(row_max_share<XBF>(x, row, K, aligned16, tid, 128));
    if ((tid & 31) == 0) part[tid >> 5] = a;
    __syncthreads();
    a = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
    if constexpr (MODE == kPrepRound) a = bf16_bits_to_f32(f32_to_bf16_bits(a));
    if constexpr (QUANT) {
      quant_scales<ACT>(a, sc, back);
    } else {
      sc = scale_of<ACT>(a);
      back = 1.0f / sc;
    }
    if (blockIdx.x == 0 && tid == 0) inv_scales[u] = back;
  }
  if (!in_range) return;
  uint32_t w[3][4];
  if constexpr (QUANT) quantize_plane<ACT>(v, sc, w[0]);
  else make_planes<ACT, AS_BF16, V>(v, sc, w);
  for (int j = 0; j < planes; ++j)
    *reinterpret_cast<uint4*>(out + static_cast<int64_t>(j * rows + u) * ld + static_cast<int64_t>(k0) * kElem) = make_uint4(w[j][0], w[j][1], w[j][2], w[j][3]);
}

// ---- a tile's outputs ------------------------------------------------------------------------------------------------------
// The calling thread owns one weight row (accumulator lane) and `rows` activation rows from y on, P.ld_y apart; inv: lane l
// holds the inverse scales of rows l, 32 + l, ... Sixteen rows at a time, the addresses in one running pointer: with an
// index multiplied out per output the epilogue of a 128 x 256 tile took 10 us, longer than an FP8 tile's products.
// BETA: what y holds at up to sixteen of them. Those of the next sixteen are asked for before these are stored, the first before the
// wait for the accumulator: asked for in turn, each sixteen cost a round trip to memory. (Kernels of their own: the 32 registers that
// are in flight leave the next kernel in the stream no room beside this one's CTAs.)
template <typename Y>
__device__ __forceinline__ void pair_old(const PairParams& P, const Y* y, int rows, bool live, float (&old)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) old[j] = 0.0f;
  if (!live) return;
#pragma unroll
  for (int j = 0; j < 16; ++j, y += P.ld_y)
    if (j < rows) old[j] = sizeof(Y) == 4 ? static_cast<float>(*y) : bf16_bits_to_f32(static_cast<uint32_t>(*y));
}
template <int kAct, int PLANES, bool BETA, typename Y>
__device__ __forceinline__ void pair_store(const PairParams& P, Y* y, uint32_t d_addr, int rows, bool live, float rf, float bias,
                                           const float (&inv)[4], float (&next)[16]) {
  const int64_t ld = P.ld_y;
  auto value = [&](const uint32_t (&raw)[PLANES][16], int j, float scale) {
    float sum = 0.0f, digit = 1.0f;
#pragma unroll
    for (int p = 0; p < PLANES; ++p) {
      const float v = kAct == kActS8 ? static_cast<float>(static_cast<int>(raw[p][j])) : __uint_as_float(raw[p][j]);
      sum += v * digit;
      digit *= P.digit;
    }
    return P.alpha * (rf * (sum * scale) + bias);
  };
  auto put = [&](Y* at, float v, float old) {
    if constexpr (BETA) v = fmaf(P.beta, old, v);
    if constexpr (sizeof(Y) == 4) *at = v;
    else *at = static_cast<uint16_t>(f32_to_bf16_bits(v));
  };
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (16 * q >= rows) break;
    uint32_t raw[PLANES][16];
#pragma unroll
    for (int p = 0; p < PLANES; ++p) tmem_ld16(d_addr + p * P.half + 16 * q, raw[p]);
    const int left = rows - 16 * q;
    float old[16];
    if constexpr (BETA) {
#pragma unroll
      for (int j = 0; j < 16; ++j) old[j] = next[j];
      if (left > 16) pair_old(P, y + 16 * ld, left - 16, live, next);
    }
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float scale = PLANES == 1 && kAct == kActBf16 ? 1.0f : __shfl_sync(0xffffffffu, inv[q / 2], 16 * (q & 1) + j);
      const float v = value(raw, j, scale);
      if (live && j < left) put(y, v, BETA ? old[j] : 0.0f);
      y += ld;
    }
  }
}

// ---- the product ----------------------------------------------------------------------------------------------------------
template <int F, int PLANES, bool BETA>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    tc_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const PairParams P) {
  constexpr int kAct = TcFmt<F>::kAct;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int S = P.S, b_bytes = P.b_bytes, stage_bytes = kPairABytes + b_bytes;
  const uint32_t ring0 = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(S) * stage_bytes);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };          // (first CTA) both CTAs' copies of the stage landed
  auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };   // its products are done
  auto d_full = [&](int b) { return bar0 + 8u * (2 * S + b); };  // accumulator b is complete
  auto d_empty = [&](int b) { return bar0 + 8u * (2 * S + 2 + b); };  // (first CTA) read by the epilogue warps of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int n_stages = P.n_stages;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(d_full(b), 1);
      mbar_init(d_empty(b), 2 * kPairEpilogueWarps);
    }
    mbar_init_fence();
  }
  if (warp == kPairEpilogueWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  cluster_meet();  // the other CTA's barriers are initialised too
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kPairEpilogueWarps) {
    // ================================ producer of weights ================================
    // The two producers are warps of their own, with a stage's addresses in running registers: a stage is consumed in 512
    // cycles, and one thread that issued both operands and divided to find its tile took longer than that (73 us for
    // M = 512 on 14336 x 4096 BF16).
    pdl_trigger();
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
      Ring r;
      bool ok = true, wrapped = false;
      int issued = 0;
      for (int tile = pair; tile < P.tiles && ok; tile += pairs) {
        const int row = tile / P.col_tiles * kPairTile + static_cast<int>(rank) * 128;
        for (int s = 0; s < n_stages; ++s) {
          if (wrapped && !tc_wait(empty_bar(r.slot), r.lap ^ 1u, P.status)) {
            ok = false;
            break;
          }
          if (rank == 0) mbar_arrive_expect_tx(full_bar(r.slot), 2u * static_cast<uint32_t>(stage_bytes));
          pair_tile_g2s(ring0 + static_cast<uint32_t>(r.slot) * stage_bytes, &wmap, s * (kPairStageK / 4), row, full_bar(r.slot));  // static: no wait
          ++issued;
          r.advance(S);
          wrapped |= r.slot == 0;
        }
      }
      // given up: the copies in flight (which complete on the first CTA's barriers) land before either CTA leaves
      if (!ok && rank == 0)
        for (int i = max(0, issued - S); i < issued; ++i) tc_wait(full_bar(i % S), (i / S) & 1, P.status);
    }
    __syncwarp();
  } else if (warp == kPairEpilogueWarps + 2) {
    // ================================ producer of activations ================================
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
      pdl_wait();  // they come from the kernel before this one
      Ring r;
      bool ok = true, wrapped = false;
      for (int tile = pair; tile < P.tiles && ok; tile += pairs) {
        const int m0 = tile % P.col_tiles * 2 * P.half + static_cast<int>(rank) * P.half;
        for (int s = 0; s < n_stages; ++s) {
          if (wrapped && !tc_wait(empty_bar(r.slot), r.lap ^ 1u, P.status)) {
            ok = false;
            break;
          }
          uint32_t dst = ring0 + static_cast<uint32_t>(r.slot) * stage_bytes + kPairABytes;
          for (int j = 0, y = m0; j < PLANES; ++j, y += P.x_rows, dst += P.half * kPairStageK) pair_tile_g2s(dst, &xmap, s * (kPairStageK / 4), y, full_bar(r.slot));
          r.advance(S);
          wrapped |= r.slot == 0;
        }
      }
    }
    __syncwarp();
  } else if (warp == kPairEpilogueWarps + 1) {
    // ================================ issuer (the pair's first CTA) ================================
    if (lane == 0 && rank == 0) {
      const uint32_t cfmt = kAct == kActS8 ? 2u : 1u, abfmt = kAct == kActE4m3 ? 0u : 1u;
      const uint32_t idesc = (cfmt << 4) | (abfmt << 7) | (abfmt << 10) | (static_cast<uint32_t>(2 * PLANES * P.half / 8) << 17) |
                             (static_cast<uint32_t>(kPairTile / 16) << 24);
      const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 128-byte swizzle, groups of 8 rows 1024 bytes apart
      const uint32_t lo0 = ((ring0 & 0x3ffffu) >> 4) | (1u << 16);
      Ring r;
      bool ok = true;
      for (int tile = pair, t = 0; tile < P.tiles && ok; tile += pairs, ++t) {
        const int buf = t & 1;
        const uint32_t d_tmem = tmem_base + buf * kPairCols;
        if (t >= 2) {
          if (!tc_wait(d_empty(buf), ((t >> 1) - 1) & 1, P.status)) break;
          tc_fence_after();
        }
        for (int s = 0; s < n_stages; ++s) {
          if (!tc_wait(full_bar(r.slot), r.lap, P.status)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_lo = lo0 + ((static_cast<uint32_t>(r.slot) * stage_bytes) >> 4), b_lo = a_lo + (kPairABytes >> 4);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) pair_umma<kAct>(d_tmem, a_lo + ks * 2, b_lo + ks * 2, hi, idesc, (s | ks) ? 1u : 0u);
          pair_commit(empty_bar(r.slot));
          r.advance(S);
        }
        if (ok) pair_commit(d_full(buf));
      }
    }
    __syncwarp();
  } else {
    // ================================ epilogue ================================
    const int quarter = warp & 3, part = warp >> 2;  // this warp takes the half of the columns that CTA `part` brought
    const int row = quarter * 32 + lane;             // of this CTA's 128
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    pdl_wait();  // y and the activation scales come from earlier kernels
    for (int tile = pair, t = 0; tile < P.tiles; tile += pairs, ++t) {
      const int buf = t & 1;
      const int n = tile / P.col_tiles * kPairTile + static_cast<int>(rank) * 128 + row;
      const int m0 = tile % P.col_tiles * 2 * P.half + part * P.half;
      const int rows = min(P.half, P.M - m0);  // (none or fewer: the last tile of the columns is ragged)
      const bool live = n < P.N;
      float rf = 1.0f, bias = 0.0f;
      if (live) {
        if (P.row_scale) rf = P.row_scale[n];
        if (P.bias) bias = load_f32(P.bias, P.bias_dtype, n);
      }
      float inv[4] = {1.0f, 1.0f, 1.0f, 1.0f};  // lane l: rows l, 32 + l, 64 + l, 96 + l of this half
      if (P.inv_scales) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (32 * q + lane < rows) inv[q] = P.inv_scales[m0 + 32 * q + lane];
      }
      const uint32_t d_addr = lane_addr + buf * kPairCols + part * PLANES * P.half;
      const int64_t at = static_cast<int64_t>(m0) * P.ld_y + n;
      float next[16];
      if constexpr (BETA) {
        if (P.y_dtype == LX_BF16) pair_old(P, static_cast<const uint16_t*>(P.y) + at, rows, live, next);
        else pair_old(P, static_cast<const float*>(P.y) + at, rows, live, next);
      }
      if (!tc_wait(d_full(buf), (t >> 1) & 1, P.status)) break;
      tc_fence_after();
      if (P.y_dtype == LX_BF16) pair_store<kAct, PLANES, BETA, uint16_t>(P, static_cast<uint16_t*>(P.y) + at, d_addr, rows, live, rf, bias, inv, next);
      else pair_store<kAct, PLANES, BETA, float>(P, static_cast<float*>(P.y) + at, d_addr, rows, live, rf, bias, inv, next);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_arrive_first(d_empty(buf));
    }
  }
  __syncthreads();
  cluster_meet();  // nothing of this CTA is reached from the other one any more
  if (warp == kPairEpilogueWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColumns) : "memory");
}

// ---- host ------------------------------------------------------------------------------------------------------------------
// Activation rows per CTA and tile: the multiple of 8 or 16 with `planes` planes within 128 columns for which the busiest pair
// has the fewest columns of products. A product of fewer than ~160 columns is charged as that many: its operands come in
// no faster (8 KB per SM at 256 columns, 6 KB at 128).
int pair_half(int M, int N, int planes, int pairs) {
  const int step = planes == 2 ? 8 : 16;  // a product of a pair takes its columns in whole 32s
  const int most = 128 / planes / step * step;
  const int64_t row_tiles = (N + kPairTile - 1) / kPairTile;
  int best = most;
  int64_t best_cost = -1;
  for (int h = most; h >= step; h -= step) {
    const int64_t tiles = row_tiles * ((M + 2 * h - 1) / (2 * h));
    const int64_t cost = (tiles + pairs - 1) / pairs * std::max(160, 2 * h * planes);
    if (best_cost < 0 || cost < best_cost) best = h, best_cost = cost;
  }
  return best;
}

template <int F, int PLANES, bool BETA>
int launch_pair(const CUtensorMap& wmap, const CUtensorMap& xmap, const PairParams& P, int pairs, size_t smem, cudaStream_t stream) {
  if (int e = allow_big_smem<200 + F * 8 + PLANES * 2 + BETA>(tc_pair_kernel<F, PLANES, BETA>)) return e;
  return launch_kernel(tc_pair_kernel<F, PLANES, BETA>, dim3(2 * static_cast<unsigned>(std::min(P.tiles, pairs))), dim3(kPairThreads), smem, stream, wmap, xmap, P);
}
template <int F, int PLANES>
int launch_pair(const CUtensorMap& wmap, const CUtensorMap& xmap, const PairParams& P, int pairs, size_t smem, cudaStream_t stream) {
  return P.beta != 0.0f ? launch_pair<F, PLANES, true>(wmap, xmap, P, pairs, smem, stream) : launch_pair<F, PLANES, false>(wmap, xmap, P, pairs, smem, stream);
}

}  // namespace

// The most rows one call of the kernel takes (more come in passes of as many): bounds the workspace.
constexpr int kPairMaxRows = 2048;

int64_t pair_workspace_bytes(int M, int K) {
  const int64_t rows = std::min(M, kPairMaxRows);
  return rows * K * 3 + 15 + rows * 4 + 256;  // int8: three planes of a byte
}

// All of M, prepared activations and their scales in `workspace` (pair_workspace_bytes). kNotSupported: not a shape for this
// kernel, the caller's other product takes it.
int pair_product(const void* x, int x_dtype, int ld_x, const lx_weight& w, const void* bias, int bias_dtype, void* y, int y_dtype, int ld_y,
                 int M, int N, int K, float alpha, float beta, void* workspace, cudaStream_t stream, bool quantized) {
  if (w.type != LX_W_BF16 && w.type != LX_W_INT8 && w.type != LX_W_FP8) return kNotSupported;
  const bool x_bf16 = x_dtype == LX_BF16;
  const int act = act_of(w.type), elem = act_elem(act);
  const int planes = quantized ? 1 : act_planes(act, true);
  const int pairs = sm_count() / 2;
  if (!pairs) return kInvalid;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  alignas(64) CUtensorMap wmap, xmap;
  if (int e = make_tile_map(&wmap, w.data, static_cast<int64_t>(K) * elem, N, 128, 128, 4, true)) return e;
  for (int m0 = 0; m0 < M; m0 += kPairMaxRows) {
    const int rows = std::min(kPairMaxRows, M - m0);
    const uint8_t* xrow = static_cast<const uint8_t*>(x) + static_cast<int64_t>(m0) * ld_x * (x_bf16 ? 2 : 4);
    PairParams P{};
    P.N = N, P.M = rows;
    P.n_stages = (K * elem + kPairStageK - 1) / kPairStageK;
    P.x_rows = rows;
    P.digit = act == kActS8 ? 0.0078125f : act == kActE4m3 ? 0.0625f : 1.0f;
    P.half = pair_half(rows, N, planes, pairs);
    P.b_bytes = planes * P.half * kPairStageK;
    P.col_tiles = (rows + 2 * P.half - 1) / (2 * P.half);
    P.tiles = (N + kPairTile - 1) / kPairTile * P.col_tiles;
    P.bias = bias, P.bias_dtype = bias_dtype;
    P.y = static_cast<uint8_t*>(y) + static_cast<int64_t>(m0) * ld_y * (y_dtype == LX_BF16 ? 2 : 4);
    P.y_dtype = y_dtype, P.ld_y = ld_y;
    P.alpha = alpha, P.beta = beta;
    P.status = status_word();
    if (w.type != LX_W_BF16) P.row_scale = static_cast<const float*>(w.scale);
    const bool in_place = w.type == LX_W_BF16 && x_bf16 && aligned(xrow, 16) && ld_x % 8 == 0;
    if (in_place) {
      if (int e = make_tile_map(&xmap, xrow, 2ll * K, rows, 128, P.half, 4, true, 2ll * ld_x)) return e;
    } else {
      const int64_t ld = static_cast<int64_t>(K) * elem;
      float* inv = reinterpret_cast<float*>(ws + (planes * rows * ld + 15) / 16 * 16);
      if (act != kActBf16) P.inv_scales = inv;
      const int per_block = 128 * 16 / elem;
      const dim3 grid((K + per_block - 1) / per_block, rows);
      auto prep = [&](auto kernel) {
        return launch_kernel(kernel, grid, dim3(128), 0, stream, static_cast<const void*>(xrow), ld_x, rows, K, planes, static_cast<int>(ld), ws, inv);
      };
      int e;
      if (quantized) {
        if (act == kActS8) e = x_bf16 ? prep(pair_prep_kernel<kActS8, true, kPrepQuant>) : prep(pair_prep_kernel<kActS8, false, kPrepQuant>);
        else e = x_bf16 ? prep(pair_prep_kernel<kActE4m3, true, kPrepQuant>) : prep(pair_prep_kernel<kActE4m3, false, kPrepQuant>);
      } else if (act == kActBf16) {
        e = x_bf16 ? prep(pair_prep_kernel<kActBf16, true, kPrepExact>) : prep(pair_prep_kernel<kActBf16, false, kPrepRound>);
      } else if (act == kActE4m3) {
        e = x_bf16 ? prep(pair_prep_kernel<kActE4m3, true, kPrepExact>) : prep(pair_prep_kernel<kActE4m3, false, kPrepRound>);
      } else {
        e = x_bf16 ? prep(pair_prep_kernel<kActS8, true, kPrepExact>) : prep(pair_prep_kernel<kActS8, false, kPrepRound>);
      }
      if (e) return e;
      if (int e2 = make_tile_map(&xmap, ws, ld, static_cast<int64_t>(planes) * rows, 128, P.half, 4, true)) return e2;
    }
    const int stage = kPairABytes + P.b_bytes;
    P.S = std::min(8, (200 * 1024) / stage);
    const size_t smem = std::max<size_t>(static_cast<size_t>(P.S) * stage + 1024, 120 * 1024);  // one CTA per SM: it takes all of tensor memory
    int e;
    if (w.type == LX_W_BF16) e = launch_pair<LX_W_BF16, 1>(wmap, xmap, P, pairs, smem, stream);
    else if (w.type == LX_W_INT8) e = planes == 1 ? launch_pair<LX_W_INT8, 1>(wmap, xmap, P, pairs, smem, stream) : launch_pair<LX_W_INT8, 3>(wmap, xmap, P, pairs, smem, stream);
    else e = planes == 1 ? launch_pair<LX_W_FP8, 1>(wmap, xmap, P, pairs, smem, stream) : launch_pair<LX_W_FP8, 2>(wmap, xmap, P, pairs, smem, stream);
    if (e) return e;
  }
  return kOk;
}

}  // namespace b200
