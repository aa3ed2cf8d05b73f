// Pieces the tcgen05 backward kernels share: packing to 16 bits, the work order of their 1-D grids and
// the store of an accumulator row.
#pragma once

#include "pjx_common.cuh"
#include "sm100_ptx.cuh"

namespace pjx {
namespace sm100 {

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  } else {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  }
}

// Work order of a 1-D grid over (tile, pair) with `n_tiles` tiles per pair and `n_pairs` pairs
// (a pair is a (batch, head)): pairs are taken in blocks of `order_w`; inside a block the tile
// index is the slow axis, so that under a causal band the long CTAs of a block start first
// (callers number the tiles heaviest-first) while the CTAs in flight share few K/V heads.
__device__ __forceinline__ void work_item(int id, int n_tiles, int n_pairs, int order_w, int& tile, int& pair) {
  const int blk = id / (order_w * n_tiles);
  const int rem = id - blk * (order_w * n_tiles);
  const int wc = min(order_w, n_pairs - blk * order_w);
  tile = rem / wc;
  pair = blk * order_w + rem % wc;
}

// Rows of `Dh` 16-bit elements leave tensor memory (32 columns at a time), are scaled and
// written to a [.., rows, heads, Dh] tensor; `dst` points at this thread's row.
template <int Dh, bool BF16>
__device__ __forceinline__ void store_row(uint32_t taddr, unsigned char* dst, float scale, bool have_acc, bool row_ok) {
#pragma unroll
  for (int c = 0; c < Dh / 32; ++c) {
    float o[32];
    if (have_acc) {
      tmem_ld32f(taddr + c * 32, o);
      tmem_wait_ld();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) o[i] = 0.f;
    }
    if (row_ok) {
      uint4* d4 = reinterpret_cast<uint4*>(dst + c * 64);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 w;
        w.x = pack16<BF16>(o[8 * i + 0] * scale, o[8 * i + 1] * scale);
        w.y = pack16<BF16>(o[8 * i + 2] * scale, o[8 * i + 3] * scale);
        w.z = pack16<BF16>(o[8 * i + 4] * scale, o[8 * i + 5] * scale);
        w.w = pack16<BF16>(o[8 * i + 6] * scale, o[8 * i + 7] * scale);
        d4[i] = w;
      }
    }
  }
}

}  // namespace sm100
}  // namespace pjx
