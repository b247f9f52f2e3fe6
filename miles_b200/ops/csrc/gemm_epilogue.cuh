// Accumulator → global memory, shared by the bf16 GEMM kernels.
#pragma once
#include "ptx.cuh"

namespace mb {

// Where a warp's 32 rows go and what is done to them on the way.
struct TileOut {
  uint8_t* c_tile;                 // first of the warp's 32 rows, column 0
  long long ldc;                   // elements
  int rows_left;                   // valid rows from the first one (may be ≤ 0 or > 32)
  int N;
  int out_fp32, accumulate;
  const __nv_bfloat16* bias;       // or null
};

// The accumulator arrives one row per thread, but whole 128-byte lines are what the memory system wants.  Each warp turns 128 bytes of
// output per row at a time (64 bf16 or 32 fp32 columns) through its 4 KB staging tile (16-byte units, XOR-swizzled against bank
// conflicts): written row-per-lane, read back with 8 lanes covering one row, so every store instruction writes four full lines.
// Needs 16-byte aligned rows and N a multiple of 16 bytes.  `t_row`: the warp's lane quadrant at the accumulator's first column;
// columns col0 .. col0 + BN − 1; `empty`: nothing was accumulated, zeros are written.
template <int BN>
__device__ __forceinline__ void store_tile_staged(const TileOut& t, uint32_t t_row, uint8_t* stage, int col0, bool empty) {
  const int lane = static_cast<int>(lane_id());
  const int esz = t.out_fp32 ? 4 : 2;
  const int cols_per_round = 128 / esz;
#pragma unroll 1
  for (int c2 = 0; c2 < BN / cols_per_round; ++c2) {
    const int colr = col0 + c2 * cols_per_round;
    if (colr >= t.N) break;                                  // uniform over the warp
    if (t.out_fp32) {
      uint32_t r[32];
      tmem_ld_32x32(t_row + c2 * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float4 o;
        o.x = empty ? 0.f : __uint_as_float(r[4 * i]);
        o.y = empty ? 0.f : __uint_as_float(r[4 * i + 1]);
        o.z = empty ? 0.f : __uint_as_float(r[4 * i + 2]);
        o.w = empty ? 0.f : __uint_as_float(r[4 * i + 3]);
        *reinterpret_cast<float4*>(stage + lane * 128 + ((i ^ (lane & 7)) << 4)) = o;
      }
    } else {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c2 * 64 + half * 32, r);
        tmem_ld_wait();
        if (empty) {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (t.bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int col = colr + half * 32 + i;
            if (col < t.N) r[i] = __float_as_uint(__uint_as_float(r[i]) + __bfloat162float(t.bias[col]));
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1]));
          o.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
          o.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
          o.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
          *reinterpret_cast<uint4*>(stage + lane * 128 + (((half * 4 + i) ^ (lane & 7)) << 4)) = o;
        }
      }
    }
    __syncwarp();
    const int unit = lane & 7;
    const int col = colr + unit * (16 / esz);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int rr = k * 4 + (lane >> 3);
      if (rr < t.rows_left && col < t.N) {
        uint8_t* dst = t.c_tile + (static_cast<long long>(rr) * t.ldc + col) * esz;
        if (t.out_fp32) {
          float4 o = *reinterpret_cast<const float4*>(stage + rr * 128 + ((unit ^ (rr & 7)) << 4));
          if (t.bias != nullptr) {
            o.x += __bfloat162float(t.bias[col]); o.y += __bfloat162float(t.bias[col + 1]);
            o.z += __bfloat162float(t.bias[col + 2]); o.w += __bfloat162float(t.bias[col + 3]);
          }
          if (t.accumulate) {
            const float4 old = *reinterpret_cast<const float4*>(dst);
            o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
          }
          *reinterpret_cast<float4*>(dst) = o;
        } else {
          *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(stage + rr * 128 + ((unit ^ (rr & 7)) << 4));
        }
      }
    }
    __syncwarp();
  }
}

}  // namespace mb
