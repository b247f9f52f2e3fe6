// Decode attention over a paged KV cache on tensor cores (flash-decoding with split keys).
//
// One CTA = (key split, KV head, request).  The `GROUP` query heads that share the KV head form the M dimension of
// mma.sync.m16n8k16 (rows ≥ GROUP are zero padding), so every K/V row fetched from HBM is used by all heads of the group
// and the score / PV products cost a handful of tensor-core instructions instead of per-key warp shuffles.
// K/V tiles of 64 keys are gathered from their cache pages with cp.async into XOR-swizzled shared memory, double
// buffered; each of the 4 warps owns 16 keys of a tile with its own running (max, sum, O) which are merged through
// shared memory at the end.  Split partials are combined by `paged_merge_kernel2`.
//
// More than 32 (request, KV head) segments in caches whose pages hold a multiple of 64 tokens (the engine's do) take the form by tiles at the
// end of this file instead: the same arithmetic, an even share of ALL the 64-key tiles of the batch per CTA, tiles by TMA.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdlib>

#include "launch.h"
#include "debug.cuh"
#include "mma_sync.cuh"
#include "pdl.cuh"
#include "ptx.cuh"
#include "rope.cuh"

namespace mb {
int make_tmap_bf16_2d(CUtensorMap* out, const void* base, long long rows, long long cols, long long ld, int box_rows, int box_cols);
}

namespace mbpd {

typedef __nv_bfloat16 bf16;
static constexpr float kLog2e = 1.4426950408889634f;
static constexpr int TK = 64;  // keys per tile

using namespace mb::ms;
template <int D>
__device__ __forceinline__ int toff(int row, int chunk) { return row * D + ((chunk ^ (row & 7)) << 3); }

template <int D>
__global__ void __launch_bounds__(128) paged_decode_mma_kernel(const bf16* q, const bf16* kc,
                                                               const bf16* vc, const int* block_table,
                                                               const int* seq_lens, float* part_o,
                                                               float* part_ml, int max_blocks, int block_size, int Hq,
                                                               int Hkv, int group, float scale, int num_splits, bf16* out,
                                                               int* counters) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  bf16* sQ = reinterpret_cast<bf16*>(smem_raw);   // 16 × D
  bf16* sK = sQ + 16 * D;                         // 2 × TK × D
  bf16* sV = sK + 2 * TK * D;                     // 2 × TK × D
  float* sM = reinterpret_cast<float*>(sV + 2 * TK * D);  // [4][8] max, [4][8] sum
  float* sL = sM + 32;
  float* sO = sL + 32;                            // [4][8][D]
  mb::pdl_trigger();
  mb::pdl_wait();
  const int req = blockIdx.z, hk = blockIdx.y, split = blockIdx.x;
  const int L = seq_lens[req];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kChunks = D / 8;
  const int per = ((L + num_splits - 1) / num_splits + TK - 1) / TK * TK;   // keys per split, whole tiles
  const int k_begin = split * per, k_end = min(L, k_begin + per);
  const int n_tiles = (k_end > k_begin) ? (k_end - k_begin + TK - 1) / TK : 0;
  const int* bt = block_table + static_cast<long long>(req) * max_blocks;

  // Q rows (heads of this group), zero padded to 16 rows
  for (int i = threadIdx.x; i < 16 * kChunks; i += 128) {
    const int r = i / kChunks, c = i % kChunks;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < group) v = *reinterpret_cast<const uint4*>(q + (static_cast<long long>(req) * Hq + hk * group + r) * D + c * 8);
    *reinterpret_cast<uint4*>(sQ + toff<D>(r, c)) = v;
  }
  auto load_tile = [&](int t, int st) {
    const int k0 = k_begin + t * TK;
    for (int i = threadIdx.x; i < TK * kChunks; i += 128) {
      const int r = i / kChunks, c = i % kChunks;
      const int key = k0 + r;
      bool ok = key < k_end;
      const int kk = ok ? key : k_begin;
      long long blk = bt[kk / block_size];
      if (!mb::dbg::in_bounds(mb::dbg::kKvBlocks, blk, 301)) { ok = false; blk = 0; }   // debug build: zero-filled instead of read
      const long long slot = blk * block_size + kk % block_size;
      const long long off = (slot * Hkv + hk) * D + c * 8;
      cp_async16(sK + st * TK * D + toff<D>(r, c), kc + off, ok);
      cp_async16(sV + st * TK * D + toff<D>(r, c), vc + off, ok);
    }
    cp_async_commit();
  };
  if (n_tiles > 0) load_tile(0, 0);
  __syncthreads();
  // Q fragments stay in registers
  uint32_t qa[D / 16][4];
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    const int row = lane & 15, chunk = ks * 2 + (lane >> 4);
    ldsm_x4(s_addr(sQ + toff<D>(row, chunk)), qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);
  }
  float o_acc[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;
  float m_i = -INFINITY, l_i = 0.f;   // row lane/4 (the rows lane/4 + 8 are padding)
  const float sl2 = scale * kLog2e;

  for (int t = 0; t < n_tiles; ++t) {
    const int st = t & 1;
    if (t + 1 < n_tiles) {
      load_tile(t + 1, st ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const bf16* tK = sK + st * TK * D;
    const bf16* tV = sV + st * TK * D;
    const int key0 = k_begin + t * TK + warp * 16;
    if (key0 < k_end) {
      float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t b[4];
        const int row = warp * 16 + (lane & 7) + ((lane >> 4) << 3);
        const int chunk = ks * 2 + ((lane >> 3) & 1);
        ldsm_x4(s_addr(tK + toff<D>(row, chunk)), b[0], b[1], b[2], b[3]);
        mma16816(s[0], qa[ks], b[0], b[1]);
        mma16816(s[1], qa[ks], b[2], b[3]);
      }
      float mx = m_i;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int key = key0 + nt * 8 + (lane & 3) * 2 + e;
          if (key >= k_end) s[nt][e] = -INFINITY;
          mx = fmaxf(mx, s[nt][e]);
        }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float msc = (mx == -INFINITY) ? 0.f : mx * sl2;
      const float alpha = (m_i == -INFINITY) ? 0.f : exp2f(m_i * sl2 - msc);
      m_i = mx;
      float rs = 0.f;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float p = exp2f(s[nt][e] * sl2 - msc);
          s[nt][e] = p;
          rs += p;
        }
      l_i = l_i * alpha + rs;
#pragma unroll
      for (int i = 0; i < D / 8; ++i) { o_acc[i][0] *= alpha; o_acc[i][1] *= alpha; }
      // P (rows 0..7 real, rows 8..15 zero) as the A operand for 16 keys
      const uint32_t pa[4] = {pack2(s[0][0], s[0][1]), 0u, pack2(s[1][0], s[1][1]), 0u};
#pragma unroll
      for (int nc = 0; nc < D / 16; ++nc) {
        uint32_t b[4];
        const int row = warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3);
        const int chunk = nc * 2 + (lane >> 4);
        ldsm_x4_t(s_addr(tV + toff<D>(row, chunk)), b[0], b[1], b[2], b[3]);
        mma16816(o_acc[2 * nc], pa, b[0], b[1]);
        mma16816(o_acc[2 * nc + 1], pa, b[2], b[3]);
      }
    }
    __syncthreads();
  }
  // merge the four warps (each holds rows 0..7 in lanes' c0/c1)
  l_i += __shfl_xor_sync(0xffffffffu, l_i, 1);
  l_i += __shfl_xor_sync(0xffffffffu, l_i, 2);
  const int r = lane >> 2;
  if ((lane & 3) == 0) { sM[warp * 8 + r] = m_i; sL[warp * 8 + r] = l_i; }
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    sO[(warp * 8 + r) * D + i * 8 + (lane & 3) * 2] = o_acc[i][0];
    sO[(warp * 8 + r) * D + i * 8 + (lane & 3) * 2 + 1] = o_acc[i][1];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < group * D; i += 128) {
    const int g = i / D, d = i % D;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) mm = fmaxf(mm, sM[w * 8 + g]);
    float ll = 0.f, oo = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float mw = sM[w * 8 + g];
      const float a = (mw == -INFINITY) ? 0.f : exp2f((mw - mm) * sl2);
      ll += sL[w * 8 + g] * a;
      oo += sO[(w * 8 + g) * D + d] * a;
    }
    const long long base = (static_cast<long long>(req) * Hq + hk * group + g) * num_splits + split;
    if (counters != nullptr && num_splits == 1) {          // a single split: normalise and write the result directly
      out[(static_cast<long long>(req) * Hq + hk * group + g) * D + d] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
      continue;
    }
    __stcg(&part_o[base * D + d], oo);
    if (d == 0) { __stcg(&part_ml[base * 2], (mm == -INFINITY) ? -INFINITY : mm * sl2); __stcg(&part_ml[base * 2 + 1], ll); }
  }
  if (counters == nullptr || num_splits == 1) return;      // merged by paged_merge_kernel2 / nothing to merge
  // the last split of this (request, kv head) to arrive merges all of them: no second kernel
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&counters[req * Hkv + hk], 1) == num_splits - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int i = threadIdx.x; i < group * D; i += 128) {
    const int g = i / D, d = i % D;
    const long long rh = static_cast<long long>(req) * Hq + hk * group + g;
    float mm = -INFINITY;
    for (int sp = 0; sp < num_splits; ++sp) mm = fmaxf(mm, __ldcg(&part_ml[(rh * num_splits + sp) * 2]));
    float ll = 0.f, oo = 0.f;
    for (int sp = 0; sp < num_splits; ++sp) {
      const float ms = __ldcg(&part_ml[(rh * num_splits + sp) * 2]);
      const float a = (ms == -INFINITY) ? 0.f : exp2f(ms - mm);
      ll += __ldcg(&part_ml[(rh * num_splits + sp) * 2 + 1]) * a;
      oo += __ldcg(&part_o[(rh * num_splits + sp) * D + d]) * a;
    }
    out[rh * D + d] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
  }
  if (threadIdx.x == 0) counters[req * Hkv + hk] = 0;
}

// partial maxima are stored pre-multiplied by scale·log2(e)
template <int D>
__global__ void paged_merge_kernel2(const float* part_o, const float* part_ml, bf16* out,
                                    int num_splits) {
  mb::pdl_trigger();
  mb::pdl_wait();
  const long long rh = blockIdx.x;
  const int d = threadIdx.x;
  float mm = -INFINITY;
  for (int s = 0; s < num_splits; ++s) mm = fmaxf(mm, part_ml[(rh * num_splits + s) * 2]);
  float ll = 0.f, oo = 0.f;
  for (int s = 0; s < num_splits; ++s) {
    const float ms = part_ml[(rh * num_splits + s) * 2];
    const float a = (ms == -INFINITY) ? 0.f : exp2f(ms - mm);
    ll += part_ml[(rh * num_splits + s) * 2 + 1] * a;
    oo += part_o[(rh * num_splits + s) * D + d] * a;
  }
  out[rh * D + d] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
}

template <int D>
static size_t smem_bytes() { return static_cast<size_t>(16 * D + 4 * TK * D) * 2 + 64 * sizeof(float) + 4 * 8 * D * sizeof(float); }

// ---- by tiles --------------------------------------------------------------------------------------------------------------------
//
// Work is counted in units of (request, KV head, 64-key tile), requests outermost; CTA c takes units [c·per, (c + 1)·per).  A CTA walks
// through segments (its tiles of one request and KV head): a whole one goes straight to the output, a part goes to one of the CTA's
// two slots of the partial buffers (0: the segment that holds its first unit, 1: a later one) and a second kernel adds up the
// slots of a segment in order.  Which CTAs share a segment follows from the units before each request and `per`, which the last CTA
// leaves in `plan`; lengths are read on the device, so that one captured launch serves any of them.  No pointer here is __restrict__: these
// kernels start before the ones in front of them have finished, and a load that the compiler takes for invariant may move up across the
// dependency wait (read that early, `plan` holds whatever the scratch memory held before).
//
// What bounds it: the cache's bytes.  An even split of every request into as many ranges (the form above) lets the longest
// request of a ragged batch set the time, and two tiles per CTA in flight behind CTA-wide barriers leave the memory idle between them.  Here a
// producer warp keeps three 32 KB tiles in flight per CTA, two CTAs per SM, and the warps that compute wait for data only.  Attention and merge,
// the form above → this one (32 query and 4 KV heads of 128): 61 requests of 290 to 4090 tokens 62.3 → 40.2 µs (bytes alone: 28.1), 19 of
// 300 to 2500 with 8 KV heads 35.2 → 19.7 (12.8), 64 × 4096 102.7 → 88.8 (83.2).  With little to read per CTA the chain length → unit →
// page → tile shows: 8 × 700 10.1 → 12.5.  `paged_attention` has the rule and both sides of it.
static constexpr int kTileStages = 3, kTileThreads = 160;      // four warps that compute, one that loads

template <int D>
struct TileSmem {
  static constexpr int kTile = TK * D * 2;                      // K or V of 64 keys: D / 64 atoms of 64 rows × 128 B
  static constexpr int o = kTileStages * 2 * kTile;             // [4][8][D] floats
  static constexpr int ml = o + 4 * 8 * D * 4;                  // [4][8] maxima, [4][8] sums
  static constexpr int bars = ml + 2 * 32 * 4;
  static constexpr int total = bars + 64;
};

// tiles of the request; its units are this times the number of KV heads
__device__ __forceinline__ int tiles_of(const int* seq_lens, int req) { return (max(seq_lens[req], 0) + TK - 1) / TK; }

template <int D>
__global__ void __launch_bounds__(kTileThreads, 2)
paged_decode_tiles_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const bf16* q,
                          const int* block_table, const int* seq_lens, bf16* out,
                          float* part_o, float* part_ml, int* plan, int batch, int max_blocks,
                          int block_size, int cache_rows, int Hq, int Hkv, float scale, int* error_flag) {
  using S = TileSmem<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (mb::smem_u32(smem) & 1023u) {   // swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicExch(error_flag, 61);
    return;
  }
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::bars);
  uint64_t* empty = full + kTileStages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kTileStages; ++i) { mb::mbar_init(&full[i], 1); mb::mbar_init(&empty[i], 4); }
    mb::mbar_fence_init();
    mb::tma_prefetch_desc(&tm_k);
    mb::tma_prefetch_desc(&tm_v);
  }
  __syncthreads();
  mb::pdl_trigger();
  mb::pdl_wait();
  const int group = Hq / Hkv;
  const int mine = lane < batch ? tiles_of(seq_lens, lane) * Hkv : 0;       // units of requests 0..31: most batches need no second look
  auto units_of = [&](int r0) { return r0 == 0 ? mine : (r0 + lane < batch ? tiles_of(seq_lens, r0 + lane) * Hkv : 0); };
  auto sum_to = [&](int n) {                                                // inclusive sum over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, n, o);
      if (lane >= o) n += v;
    }
    return n;
  };
  int units = mine;
  for (int r0 = 32; r0 < batch; r0 += 32) units += units_of(r0);
  units = __reduce_add_sync(0xffffffffu, units);
  const int per = (units + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int begin = static_cast<int>(blockIdx.x) * per, end = min(units, begin + per);
  if (blockIdx.x == gridDim.x - 1 && warp == 0) {                           // the last CTA has the fewest units, often none
    int before = 0;
    for (int r0 = 0; r0 < batch; r0 += 32) {
      const int n = units_of(r0), sum = sum_to(n);
      if (r0 + lane < batch) plan[r0 + lane] = before + sum - n;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) { plan[batch] = before; plan[batch + 1] = per; }
  }
  if (begin >= end) return;
  // where the first unit is
  int req = 0, at = begin;
  for (int r0 = 0, before = 0;; r0 += 32) {
    const int n = units_of(r0), sum = sum_to(n);
    const uint32_t beyond = __ballot_sync(0xffffffffu, before + sum > begin);
    if (beyond) {
      const int l = __ffs(beyond) - 1;
      req = r0 + l;
      at = begin - before - __shfl_sync(0xffffffffu, sum - n, l);
      break;
    }
    before += __shfl_sync(0xffffffffu, sum, 31);
  }
  int tiles = tiles_of(seq_lens, req);
  int hk = at / tiles, tile = at % tiles;
  int stage = 0;
  uint32_t phase = 0;
  bool ok = true;

  for (int u = begin; u < end;) {                           // after a failed wait a warp goes on without tiles: it still meets the barriers below
    const int n = min(tiles - tile, end - u);               // this segment's tiles
    if (warp == 4) {
      // ------------------------------ TMA producer ------------------------------
      const int* bt = block_table + static_cast<long long>(req) * max_blocks;
      for (int i0 = 0; i0 < n && ok; i0 += 32) {
        int row = 0;                                        // lane i: first cache row of tile i0 + i
        if (i0 + lane < n) {
          const int key = (tile + i0 + lane) * TK;
          const long long blk = bt[key / block_size];
          row = mb::dbg::in_bounds(mb::dbg::kKvBlocks, blk, 301) ? static_cast<int>(blk) * block_size + key % block_size : cache_rows;   // past the end: zeros
        }
        for (int i = 0; i < min(32, n - i0) && ok; ++i) {
          const int r = __shfl_sync(0xffffffffu, row, i);
          ok = __all_sync(0xffffffffu, mb::mbar_wait(&empty[stage], phase ^ 1));
          if (ok && lane == 0) {
            mb::mbar_expect_tx(&full[stage], 2 * S::kTile);
            uint8_t* dst = smem + stage * 2 * S::kTile;
#pragma unroll
            for (int a = 0; a < D / 64; ++a) {
              mb::tma_load_2d(dst + a * (TK * 128), &tm_k, &full[stage], hk * D + a * 64, r);
              mb::tma_load_2d(dst + S::kTile + a * (TK * 128), &tm_v, &full[stage], hk * D + a * 64, r);
            }
          }
          if (++stage == kTileStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok && lane == 0) atomicExch(error_flag, 62);
    } else {
      // ------------------------------ scores, softmax, values: 16 keys of each tile per warp ------------------------------
      const int L = seq_lens[req];
      uint32_t qa[D / 16][2];                               // A operand: rows 0..7 are the group's heads, 8..15 zero
      {
        const int g = lane >> 2;
        const bf16* qr = q + (static_cast<long long>(req) * Hq + hk * group + g) * D + (lane & 3) * 2;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          qa[ks][0] = g < group ? *reinterpret_cast<const uint32_t*>(qr + ks * 16) : 0u;
          qa[ks][1] = g < group ? *reinterpret_cast<const uint32_t*>(qr + ks * 16 + 8) : 0u;
        }
      }
      float o_acc[D / 8][4];
#pragma unroll
      for (int i = 0; i < D / 8; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;
      float m_i = -INFINITY, l_i = 0.f;                     // row lane / 4
      const float sl2 = scale * kLog2e;
      for (int i = 0; i < n && ok; ++i) {
        ok = __all_sync(0xffffffffu, mb::mbar_wait(&full[stage], phase));
        if (!ok) break;
        uint8_t* sK = smem + stage * 2 * S::kTile;
        uint8_t* sV = sK + S::kTile;
        const int key0 = (tile + i) * TK + warp * 16;
        auto unit16 = [](uint8_t* base, int row, int chunk) {   // 16-byte unit `chunk` of a row, atoms of 64 columns, 128-byte swizzle
          return base + (chunk >> 3) * (TK * 128) + row * 128 + (((chunk & 7) ^ (row & 7)) << 4);
        };
        if (key0 < L) {
          if (key0 + 16 > L) {                              // rows behind the sequence: weight 0, but whatever the page holds may be no number
            for (int v = lane; v < 16 * (D / 8); v += 32) {
              const int row = v / (D / 8);
              if (key0 + row >= L) *reinterpret_cast<uint4*>(unit16(sV, warp * 16 + row, v % (D / 8))) = make_uint4(0, 0, 0, 0);
            }
            mb::fence_proxy_async();                        // … before the next tile is copied over it
            __syncwarp();
          }
          float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t b[4];
            ldsm_x4(s_addr(unit16(sK, warp * 16 + (lane & 7) + ((lane >> 4) << 3), ks * 2 + ((lane >> 3) & 1))), b[0], b[1], b[2], b[3]);
            const uint32_t a[4] = {qa[ks][0], 0u, qa[ks][1], 0u};
            mma16816(s[0], a, b[0], b[1]);
            mma16816(s[1], a, b[2], b[3]);
          }
          float mx = m_i;
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              if (key0 + nt * 8 + (lane & 3) * 2 + e >= L) s[nt][e] = -INFINITY;
              mx = fmaxf(mx, s[nt][e]);
            }
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          const float msc = (mx == -INFINITY) ? 0.f : mx * sl2;
          const float alpha = (m_i == -INFINITY) ? 0.f : exp2f(m_i * sl2 - msc);
          m_i = mx;
          float rs = 0.f;
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              s[nt][e] = exp2f(s[nt][e] * sl2 - msc);
              rs += s[nt][e];
            }
          l_i = l_i * alpha + rs;
#pragma unroll
          for (int c = 0; c < D / 8; ++c) { o_acc[c][0] *= alpha; o_acc[c][1] *= alpha; }
          const uint32_t pa[4] = {pack2(s[0][0], s[0][1]), 0u, pack2(s[1][0], s[1][1]), 0u};
#pragma unroll
          for (int nc = 0; nc < D / 16; ++nc) {
            uint32_t b[4];
            ldsm_x4_t(s_addr(unit16(sV, warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), nc * 2 + (lane >> 4))), b[0], b[1], b[2], b[3]);
            mma16816(o_acc[2 * nc], pa, b[0], b[1]);
            mma16816(o_acc[2 * nc + 1], pa, b[2], b[3]);
          }
        }
        __syncwarp();
        if (lane == 0) mb::mbar_arrive(&empty[stage]);
        if (++stage == kTileStages) { stage = 0; phase ^= 1; }
      }
      // merge the four warps
      if (!ok && lane == 0) atomicExch(error_flag, 63);
      float* sO = reinterpret_cast<float*>(smem + S::o);
      float* sM = reinterpret_cast<float*>(smem + S::ml);
      float* sL = sM + 32;
      l_i += __shfl_xor_sync(0xffffffffu, l_i, 1);
      l_i += __shfl_xor_sync(0xffffffffu, l_i, 2);
      const int r = lane >> 2;
      if ((lane & 3) == 0) { sM[warp * 8 + r] = m_i; sL[warp * 8 + r] = l_i; }
#pragma unroll
      for (int c = 0; c < D / 8; ++c)
        *reinterpret_cast<float2*>(&sO[(warp * 8 + r) * D + c * 8 + (lane & 3) * 2]) = make_float2(o_acc[c][0], o_acc[c][1]);
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const bool whole = tile == 0 && n == tiles;
      const long long slot = 2 * static_cast<long long>(blockIdx.x) + (u == begin ? 0 : 1);
      for (int v = threadIdx.x; v < group * (D / 4); v += 128) {
        const int g = v / (D / 4), d = v % (D / 4) * 4;
        float mm = -INFINITY, ll = 0.f;
        float4 oo = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 4; ++w) mm = fmaxf(mm, sM[w * 8 + g]);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const float mw = sM[w * 8 + g];
          const float a = (mw == -INFINITY) ? 0.f : exp2f((mw - mm) * sl2);
          const float4 x = *reinterpret_cast<const float4*>(&sO[(w * 8 + g) * D + d]);
          ll += sL[w * 8 + g] * a;
          oo.x += x.x * a; oo.y += x.y * a; oo.z += x.z * a; oo.w += x.w * a;
        }
        if (whole) {
          const float inv = ll > 0.f ? 1.f / ll : 0.f;
          *reinterpret_cast<uint2*>(out + (static_cast<long long>(req) * Hq + hk * group + g) * D + d) =
              make_uint2(pack2(oo.x * inv, oo.y * inv), pack2(oo.z * inv, oo.w * inv));
        } else {
          __stcg(reinterpret_cast<float4*>(part_o + (slot * group + g) * D + d), oo);
          if (d == 0) __stcg(reinterpret_cast<float2*>(part_ml + (slot * group + g) * 2), make_float2((mm == -INFINITY) ? -INFINITY : mm * sl2, ll));
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");      // sO is free again
    }
    u += n;
    tile += n;
    if (tile == tiles && u < end) {
      tile = 0;
      if (++hk == Hkv) {
        hk = 0;
        do { tiles = tiles_of(seq_lens, ++req); } while (tiles == 0);       // u < end: some request behind has units
      }
    }
  }
}

// grid (Hq, batch), 128 threads: the slots of one head's segment.  A segment that one CTA did alone is already in place; a request
// without keys gets zeros.
template <int D>
__global__ void __launch_bounds__(128) paged_merge_tiles_kernel(const float* part_o, const float* part_ml,
                                                               const int* plan, bf16* out, int batch, int Hq, int Hkv) {
  __shared__ float4 s_o[4][D / 4];
  __shared__ float s_l[4];
  mb::pdl_trigger();
  mb::pdl_wait();
  const int h = blockIdx.x, req = blockIdx.y, group = Hq / Hkv, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = __ldcg(plan + batch + 1), u_req = __ldcg(plan + req), tiles = (__ldcg(plan + req + 1) - u_req) / Hkv;
  bf16* o = out + (static_cast<long long>(req) * Hq + h) * D;
  if (tiles == 0) {
    if (threadIdx.x < D / 4) *reinterpret_cast<uint2*>(o + threadIdx.x * 4) = make_uint2(0u, 0u);
    return;
  }
  const int u0 = u_req + h / group * tiles, c0 = u0 / per, c1 = (u0 + tiles - 1) / per;
  if (c0 == c1) return;
  const int first = u0 == c0 * per ? 0 : 1;                 // the first CTA's slot; the others start with this segment
  auto at = [&](int c) { return (2ll * c + (c == c0 ? first : 0)) * group + h % group; };
  float mm = -INFINITY;
  for (int c = c0 + lane; c <= c1; c += 32) mm = fmaxf(mm, __ldcg(part_ml + at(c) * 2));
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, i));
  float ll = 0.f;
  float4 oo = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int c = c0 + warp; c <= c1; c += 4) {
    const float2 ml = __ldcg(reinterpret_cast<const float2*>(part_ml + at(c) * 2));
    const float a = (ml.x == -INFINITY) ? 0.f : exp2f(ml.x - mm);
    ll += ml.y * a;
    if (lane < D / 4) {
      const float4 x = __ldcg(reinterpret_cast<const float4*>(part_o + at(c) * D) + lane);
      oo.x += x.x * a; oo.y += x.y * a; oo.z += x.z * a; oo.w += x.w * a;
    }
  }
  if (lane < D / 4) s_o[warp][lane] = oo;
  if (lane == 0) s_l[warp] = ll;
  __syncthreads();
  if (threadIdx.x < D / 4) {
    const float4 a = s_o[0][lane], b = s_o[1][lane], c = s_o[2][lane], d = s_o[3][lane];
    const float l = (s_l[0] + s_l[1]) + (s_l[2] + s_l[3]), inv = l > 0.f ? 1.f / l : 0.f;
    *reinterpret_cast<uint2*>(o + lane * 4) = make_uint2(pack2((a.x + b.x + c.x + d.x) * inv, (a.y + b.y + c.y + d.y) * inv),
                                                         pack2((a.z + b.z + c.z + d.z) * inv, (a.w + b.w + c.w + d.w) * inv));
  }
}

// The same with a warp per head, eight heads per CTA, for batches whose segments have few parts each (`launch_tiles`).  What bounds it is the
// chain plan → parts → sum: the parts' maxima and the first four parts are requested together, and nothing waits for another warp.
template <int D>
__global__ void __launch_bounds__(256) paged_merge_heads_kernel(const float* part_o, const float* part_ml, const int* plan, bf16* out, int batch, int Hq,
                                                               int Hkv) {
  constexpr int VPL = D / 32;                               // output columns per lane
  struct alignas(4 * VPL) Piece { float v[VPL]; };
  mb::pdl_trigger();
  mb::pdl_wait();
  const int row = static_cast<int>(blockIdx.x) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= batch * Hq) return;
  const int req = row / Hq, h = row % Hq, group = Hq / Hkv;
  const int per = __ldcg(plan + batch + 1), u_req = __ldcg(plan + req), tiles = (__ldcg(plan + req + 1) - u_req) / Hkv;
  bf16* o = out + static_cast<long long>(row) * D + lane * VPL;
  auto store = [&](const float (&x)[VPL], float f) {
#pragma unroll
    for (int i = 0; i < VPL; i += 2) *reinterpret_cast<uint32_t*>(o + i) = pack2(x[i] * f, x[i + 1] * f);
  };
  float oo[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) oo[i] = 0.f;
  if (tiles == 0) {
    store(oo, 0.f);
    return;
  }
  const int u0 = u_req + h / group * tiles, c0 = u0 / per, c1 = (u0 + tiles - 1) / per;
  if (c0 == c1) return;
  const int first = u0 == c0 * per ? 0 : 1;
  auto at = [&](int c) { return (2ll * c + (c == c0 ? first : 0)) * group + h % group; };
  auto part = [&](int c) {
    Piece x;
    const float* p = part_o + at(c) * D + lane * VPL;
    if (VPL == 4) {
      const float4 y = __ldcg(reinterpret_cast<const float4*>(p));
      x.v[0] = y.x; x.v[1] = y.y; x.v[VPL - 2] = y.z; x.v[VPL - 1] = y.w;
    } else {
      const float2 y = __ldcg(reinterpret_cast<const float2*>(p));
      x.v[0] = y.x; x.v[1] = y.y;
    }
    return x;
  };
  float mm = -INFINITY, ll = 0.f;
  for (int b = c0; b <= c1; b += 32) {                      // 32 parts at a time: lane i holds the maximum and the sum of part b + i
    const int n = min(32, c1 - b + 1);
    float2 ml = make_float2(-INFINITY, 0.f);
    if (lane < n) ml = __ldcg(reinterpret_cast<const float2*>(part_ml + at(b + lane) * 2));
    Piece x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < n) x[i] = part(b + i);
    float m = fmaxf(mm, ml.x);
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, i));
    const float a = ml.x == -INFINITY ? 0.f : exp2f(ml.x - m), old = mm == -INFINITY ? 0.f : exp2f(mm - m);
    float l = ml.y * a;
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) l += __shfl_xor_sync(0xffffffffu, l, i);
    ll = ll * old + l;
    mm = m;
#pragma unroll
    for (int k = 0; k < VPL; ++k) oo[k] *= old;
    for (int i0 = 0; i0 < n; i0 += 4) {
      if (i0 > 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i0 + i < n) x[i] = part(b + i0 + i);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float w = __shfl_sync(0xffffffffu, a, (i0 + i) & 31);
        if (i0 + i < n) {
#pragma unroll
          for (int k = 0; k < VPL; ++k) oo[k] += x[i].v[k] * w;
        }
      }
    }
  }
  store(oo, ll > 0.f ? 1.f / ll : 0.f);
}

template <int D>
static int launch_tiles(const bf16* q, const void* kc, const void* vc, const int* block_table, const int* seq_lens, bf16* out, float* part_o,
                        float* part_ml, int* plan, int batch, int max_blocks, int block_size, int cache_rows, int Hq, int Hkv, float scale,
                        int ctas, int* error_flag, cudaStream_t s) {
  CUtensorMap tk, tv;
  int rc = mb::make_tmap_bf16_2d(&tk, kc, cache_rows, static_cast<long long>(Hkv) * D, static_cast<long long>(Hkv) * D, TK, 64);
  if (rc) return 1000 + rc;
  rc = mb::make_tmap_bf16_2d(&tv, vc, cache_rows, static_cast<long long>(Hkv) * D, static_cast<long long>(Hkv) * D, TK, 64);
  if (rc) return 2000 + rc;
  static const cudaError_t configured =
      cudaFuncSetAttribute(paged_decode_tiles_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, TileSmem<D>::total);
  if (configured != cudaSuccess) return static_cast<int>(configured);
  cudaError_t e = mb::launch_pdl(paged_decode_tiles_kernel<D>, dim3(ctas), dim3(kTileThreads), TileSmem<D>::total, s, tk, tv, q, block_table,
                                 seq_lens, out, part_o, part_ml, plan, batch, max_blocks, block_size, cache_rows, Hq, Hkv, scale, error_flag);
  if (e != cudaSuccess) return static_cast<int>(e);
  // a segment is shared by ctas / (batch · Hkv) CTAs on average: up to 4 a warp adds them up (61 requests, 4 KV heads: 43.3 → 40.2 µs with the
  // attention), beyond that four warps do (7 requests, 11 on average: 12.7 µs, 14.7 with one warp)
  if (ctas <= 4 * batch * Hkv)
    e = mb::launch_pdl(paged_merge_heads_kernel<D>, dim3((batch * Hq + 7) / 8), dim3(256), 0, s, static_cast<const float*>(part_o),
                       static_cast<const float*>(part_ml), static_cast<const int*>(plan), out, batch, Hq, Hkv);
  else
    e = mb::launch_pdl(paged_merge_tiles_kernel<D>, dim3(Hq, batch), dim3(128), 0, s, static_cast<const float*>(part_o), static_cast<const float*>(part_ml),
                       static_cast<const int*>(plan), out, batch, Hq, Hkv);
  return static_cast<int>(e);
}

}  // namespace mbpd

#include "decode_attend.cuh"

using namespace mbpd;

MB_DEFINE_BOUNDS_API(mb_paged_bounds)

// part_o: [B·Hq·splits·D] floats, part_ml: [B·Hq·splits·2] floats.  Hq/Hkv ≤ 8.
extern "C" int mb_paged_decode(const void* q, const void* kc, const void* vc, const int* block_table, const int* seq_lens, void* out,
                               float* part_o, float* part_ml, int batch, int max_blocks, int block_size, int Hq, int Hkv, int D,
                               float scale, int num_splits, cudaStream_t s) {
  if (batch == 0) return 0;
  const int group = Hq / Hkv;
  if (group > 8 || group * Hkv != Hq) return -2;
  dim3 grid(num_splits, Hkv, batch);
  // Optional in-kernel merge (MILES_DECODE_FUSED_MERGE=1): the last split of a (request, kv head) to arrive merges them,
  // which saves the merge launch but leaves the whole GQA group to one CTA; measured slower than the separate merge
  // kernel at the batch sizes of the rollout (21 µs against 11 + 4 µs at batch 8), so it is off by default.
  // Arrival counters: one per (request, kv head), zero between calls; allocated on first use outside stream capture.
  static const bool fused_merge = [] { const char* e = getenv("MILES_DECODE_FUSED_MERGE"); return e != nullptr && e[0] == '1'; }();
  static int* counter_buf[64] = {};
  static int counter_cap[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int* counters = nullptr;
  if (fused_merge && dev < 64) {
    if (counter_cap[dev] < batch * Hkv) {
      cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
      cudaStreamIsCapturing(s, &st);
      if (st == cudaStreamCaptureStatusNone) {
        const int cap = batch * Hkv > 16384 ? batch * Hkv : 16384;
        int* fresh = nullptr;
        if (cudaMalloc(&fresh, cap * sizeof(int)) == cudaSuccess && cudaMemset(fresh, 0, cap * sizeof(int)) == cudaSuccess) {
          counter_buf[dev] = fresh;      // an older, smaller buffer may still be referenced by captured graphs: it is kept
          counter_cap[dev] = cap;
        }
      }
    }
    if (counter_cap[dev] >= batch * Hkv) counters = counter_buf[dev];
  }
  bf16* O = reinterpret_cast<bf16*>(out);
  auto Q = reinterpret_cast<const bf16*>(q);
  auto KC = reinterpret_cast<const bf16*>(kc);
  auto VC = reinterpret_cast<const bf16*>(vc);
  if (D == 128) {
    static bool once = false;
    if (!once) {
      cudaError_t e = cudaFuncSetAttribute(paged_decode_mma_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(smem_bytes<128>()));
      if (e != cudaSuccess) return static_cast<int>(e);
      once = true;
    }
    cudaError_t e = mb::launch_pdl(paged_decode_mma_kernel<128>, grid, dim3(128), smem_bytes<128>(), s, Q, KC, VC, block_table, seq_lens, part_o,
                               part_ml, max_blocks, block_size, Hq, Hkv, group, scale, num_splits, O, counters);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (counters == nullptr) e = mb::launch_pdl(paged_merge_kernel2<128>, dim3(batch * Hq), dim3(128), 0, s, static_cast<const float*>(part_o),
                   static_cast<const float*>(part_ml), reinterpret_cast<bf16*>(out), num_splits);
    if (e != cudaSuccess) return static_cast<int>(e);
  } else if (D == 64) {
    static bool once = false;
    if (!once) {
      cudaError_t e = cudaFuncSetAttribute(paged_decode_mma_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(smem_bytes<64>()));
      if (e != cudaSuccess) return static_cast<int>(e);
      once = true;
    }
    cudaError_t e = mb::launch_pdl(paged_decode_mma_kernel<64>, grid, dim3(128), smem_bytes<64>(), s, Q, KC, VC, block_table, seq_lens, part_o,
                               part_ml, max_blocks, block_size, Hq, Hkv, group, scale, num_splits, O, counters);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (counters == nullptr) e = mb::launch_pdl(paged_merge_kernel2<64>, dim3(batch * Hq), dim3(64), 0, s, static_cast<const float*>(part_o),
                   static_cast<const float*>(part_ml), reinterpret_cast<bf16*>(out), num_splits);
    if (e != cudaSuccess) return static_cast<int>(e);
  } else {
    return -1;
  }
  return static_cast<int>(cudaGetLastError());
}

// The form by tiles: block_size a multiple of 64.  cache_rows: pages × block_size.  `ctas` CTAs share the work; part_o: 2 · ctas · Hq/Hkv · D
// floats, part_ml: 2 · ctas · Hq/Hkv · 2 floats, plan: batch + 2 ints (all scratch, written before they are read).
extern "C" int mb_paged_decode_tiles(const void* q, const void* kc, const void* vc, const int* block_table, const int* seq_lens, void* out,
                                     float* part_o, float* part_ml, int* plan, int batch, int max_blocks, int block_size, int cache_rows, int Hq,
                                     int Hkv, int D, float scale, int ctas, int* error_flag, cudaStream_t s) {
  if (batch == 0) return 0;
  const int group = Hq / Hkv;
  if (group > 8 || group * Hkv != Hq || block_size % TK != 0 || batch > 65535) return -2;
  auto Q = reinterpret_cast<const bf16*>(q);
  bf16* O = reinterpret_cast<bf16*>(out);
  if (D == 128)
    return launch_tiles<128>(Q, kc, vc, block_table, seq_lens, O, part_o, part_ml, plan, batch, max_blocks, block_size, cache_rows, Hq, Hkv, scale, ctas,
                             error_flag, s);
  if (D == 64)
    return launch_tiles<64>(Q, kc, vc, block_table, seq_lens, O, part_o, part_ml, plan, batch, max_blocks, block_size, cache_rows, Hq, Hkv, scale, ctas,
                            error_flag, s);
  return -1;
}

// See decode_attend.cuh.  q, k, v: the step's projections [batch, heads, 128] bf16, `*_stride` elements between tokens; qw, kw: norm weights or null; slots[b]: where the
// new key and value go (< 0: nowhere); pages of a multiple of 16 tokens; cache_rows: pages × block_size.  split: CTAs per (request, KV head), 1 to 16.
extern "C" int mb_decode_attend(const void* q, const void* k, const void* v, long long q_stride, long long k_stride, long long v_stride, const void* qw,
                                const void* kw, const int* positions, float theta, float eps, void* kc, void* vc, const long long* slots, const int* block_table,
                                const int* seq_lens, void* out, int batch, int max_blocks, int block_size, int cache_rows, int Hq, int Hkv, int D, float scale,
                                int split, int* error_flag, cudaStream_t s) {
  if (batch == 0) return 0;
  if (D != 128 || Hq % Hkv || Hq / Hkv > 8 || block_size % kDaKeys || split < 1 || split > kDaMaxSplit || batch > 65535) return -2;
  CUtensorMap tk, tv;
  int rc = mb::make_tmap_bf16_2d(&tk, kc, cache_rows, static_cast<long long>(Hkv) * D, static_cast<long long>(Hkv) * D, kDaKeys, 64);
  if (rc) return 1000 + rc;
  rc = mb::make_tmap_bf16_2d(&tv, vc, cache_rows, static_cast<long long>(Hkv) * D, static_cast<long long>(Hkv) * D, kDaKeys, 64);
  if (rc) return 2000 + rc;
  static const cudaError_t configured = [] {
    cudaError_t e = cudaFuncSetAttribute(decode_attend_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, DaSmem<128>::total);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(decode_attend_kernel<128>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }();
  if (configured != cudaSuccess) return static_cast<int>(configured);
  auto b = [](const void* x) { return reinterpret_cast<const bf16*>(x); };
  const DecodeAttend p{b(q), b(k), b(v), q_stride, k_stride, v_stride, b(qw), b(kw), positions, block_table, seq_lens, slots, reinterpret_cast<bf16*>(kc),
                       reinterpret_cast<bf16*>(vc), reinterpret_cast<bf16*>(out), max_blocks, block_size, cache_rows, Hq, Hkv, split, log2f(theta), eps, scale, error_flag};
  return static_cast<int>(mb::launch_pdl_cluster(decode_attend_kernel<128>, dim3(split, Hkv, batch), dim3(kDaWarps * 32), split, DaSmem<128>::total, s, tk, tv, p));
}
