// Flash-attention backward for sm_100a with P and dS carried at 32-bit grade: score modifiers
// (segments, ALiBi, relative tables, soft cap, dropout, ...), a dense fp32 bias and its gradient, and the
// latent head shape (192, 128).  Same two-kernel split, warp roles and half-step issue order as
// attn_bwd_sm100.cu (dQ owns query tiles, dK/dV owns key tiles, no atomics); what differs:
//
// * P and dS enter the accumulating products as a sum of two 16-bit numbers, x = hi + lo with hi = round16(x)
//   and lo = round16(x - hi): two MMAs against the same B descriptor
//   instead of one.  The calls that arrive here ran on CUDA cores with P and dS in fp32 before, and 16 + 16 bits
//   keep what that gave (2^-18 relative in bf16 against the 2^-9 of the stored gradients).  Per 128 x 128 tile that is 10
//   products of 128 x 128 x D for both kernels instead of 7.  A 16-column chunk of scores (16 columns of
//   tensor memory) is overwritten by its own 8 columns of hi and 8 of lo pairs, so the split costs no
//   tensor memory.
// * fp16 has no exponent range to spare for lo (its lowest step is 2^-24): what a thread packs belongs to one row of
//   the accumulator it feeds, so every row has a power of two of its own, undone when the accumulators leave tensor
//   memory.  dQ: from the row's |dO|, its delta and the longest V row of the key tiles it walks (`v_norm_kernel`).  dK
//   and dV: from the largest P and the largest term of dS of the key over all rows and heads that see it, which the dQ
//   kernel collects on its way (`add_col_max`).  One power of two for the whole call, from the largest |dO| and |V|,
//   took the bits of every row far below the largest: beside a row of dO 1e6 times larger the others' dQ was off by 40
//   to 120 times its rounding.
// * head shape (192, 128): dV and dK take 320 columns of tensor memory, so the dK/dV kernel walks query
//   tiles of 96 rows (two halves of 48: 2 x 96 + 320 = 512 columns) instead of 128.
// * a segment mask cuts the tile loops to the ranges that can match (one range per 128 rows, both ways).
// * a dense bias is read with keys on the lanes (coalesced) in the dK/dV and dbias kernels; the dQ kernel,
//   whose threads own query rows, transposes it through its ring in shared memory.
// * the gradient of the bias is a kernel of its own: one CTA per 128 x 128 tile of the bias, walking the
//   (batch, head) pairs that share it and summing dS in registers in a fixed order (no atomics).
//
// FEAT: bit 0 = structured masks and terms added to the scores (ALiBi, relative table), bit 1 = dense bias, bit 2 =
// head scale, soft cap and dropout (a hash and a tanhf per score: inlined for a whole tile they make the loop
// miss the instruction cache, 45% of the time of the packed ALiBi step); band and key-length masks always.
// The row vector `lse2` is base 2 unless a relative table or a dense bias is added to the scores: then it is
// the natural log-sum-exp, subtracted before the change of base, so that an entry of the type's lowest value
// cannot overflow to inf - inf.
//
// Bound by the element work of the compute warps at D = 64 and with modifiers (20 to 30 issue slots per score), by the
// chain of MMAs, element work and barrier round trips at D = 128 and 192 without.
// Spills (bytes stored / loaded, -Xptxas -v; a thread has 168 registers): dK/dV with modifiers 24 to 68 / 32 to 112, with a
// dense bias beside them 168 to 200 / 180 to 236; the bias gradient 4 to 24 / 4 to 44, with modifiers 304 to 340 / 304 to 360;
// the other kernels 28 / 60 at most.
// Measured (forward + backward, against the CUDA-core kernels these calls ran on before; B200):
//   packed documents + ALiBi, B1 S4096 Hq32 Hkv8 D128 bf16     41.9 ms -> 0.48 ms
//   dense bias with gradient, B8 S1024 H16 D64 bf16            6.26 ms -> 0.49 ms
//   latent training step, B2 S2048 H16 (192,128) bf16          16.6 ms -> 0.42 ms
#include <atomic>

#include "attn_bwd_sm100.cuh"

namespace pjx {

int make_tmap_blhd(CUtensorMap* m, const void* base, int dtype, int B, int L, int H, int Dim, int rows);

namespace {

using namespace sm100;

constexpr int BM = 128;        // query rows per tile of the dQ and dbias kernels
constexpr int BN = 128;        // keys per tile
constexpr int NTHREADS = 320;  // 10 warps: TMA producer, MMA issuer, two compute groups of four
constexpr int CH = 16;         // score columns a thread works on at a time

// What the kernels need beside BwdParams.
struct ExactArgs {
  int order_w;
  const int32_t* q_range;  // [nb, ceil(Lq/128), 2]: keys a query tile can see (segments), or null
  const int32_t* k_range;  // [nb, ceil(Lkv/128), 2]: query rows a key tile is seen by, or null
  int64_t q_range_bs, k_range_bs;  // batch strides in tiles (0 = shared)
  const float* v_norm;     // fp16: longest finite V row of each key tile, [B, Hkv, ceil(Lkv/128)]
  uint32_t* col_max;       // fp16: per key the largest term of dS and the largest P, bit patterns, [B, Hkv, 2, Lkv]
  bool bias_vec;           // rows of the dense bias are whole aligned 16-byte units
};

// fp16: the power of two that takes `bound` into [2^top, 2^(top+1)); 1 where there is no positive finite bound.
__device__ __forceinline__ float pack_scale(float bound, int top) {
  const int e = (int)(__float_as_uint(bound) >> 23);  // (never negative: 255 is inf or NaN)
  if (!(bound > 0.f) || e == 255) return 1.f;
  return __uint_as_float((uint32_t)(127 + max(-126, min(126, top + 127 - e))) << 23);
}

// fp16: largest magnitudes of a chunk's CH keys over the warp's 32 query rows, added to those of the keys: of dS (together
// with P dP, the term its difference is formed from: where the two cancel the result is rounding noise of that
// size, another one in the dK/dV kernel) and of P.  The upper halves of the fp32 words order like the values; both are
// reduced at once, each step leaving a lane half of the columns.  `out` points at the chunk's first key.
__device__ __forceinline__ void add_col_max(const float2 (&pr)[CH / 2], const float2 (&ds)[CH / 2], const float (&dp)[CH],
                                            uint32_t* out, int n_cols, int Lkv, int lane) {
  uint32_t v[CH];
#pragma unroll
  for (int i = 0; i < CH / 2; ++i) {
    // (fmaxf drops a NaN: of a masked entry, 0 times a dP that may be anything)
    const float x = fmaxf(fabsf(ds[i].x), fabsf(pr[i].x * dp[2 * i])), y = fmaxf(fabsf(ds[i].y), fabsf(pr[i].y * dp[2 * i + 1]));
    v[2 * i] = __byte_perm(__float_as_uint(pr[i].x), __float_as_uint(x), 0x7632) & 0x7fff7fffu;
    v[2 * i + 1] = __byte_perm(__float_as_uint(pr[i].y), __float_as_uint(y), 0x7632) & 0x7fff7fffu;
  }
#pragma unroll
  for (int w = CH / 2; w >= 1; w /= 2) {
    const bool upper = lane & w;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + w], w);
      v[i] = __vmaxu2(upper ? v[i + w] : v[i], other);
    }
  }
  const uint32_t m = __vmaxu2(v[0], __shfl_xor_sync(0xffffffffu, v[0], CH));  // of key lane % CH
  const uint32_t mine = lane < CH ? m & 0xffff0000u : m << 16;                // dS in the lower lanes, P in the upper
  const int col = lane % CH;
  if (mine && col < n_cols) atomicMax(out + (lane < CH ? 0 : Lkv) + col, mine);
}

// A chunk of CH fp32 values as hi pairs (8 registers) and lo pairs (8 registers), both rounded: 2^-18 of x at most in
// bf16.  (hi cut off instead, one byte permute per pair, left 2^-16.)
template <bool BF16>
__device__ __forceinline__ void split_pack(const float2 (&x)[CH / 2], float scale, uint32_t (&r)[CH]) {
#pragma unroll
  for (int i = 0; i < CH / 2; ++i) {
    if constexpr (BF16) {
      const uint32_t hi = pack16<true>(x[i].x, x[i].y);
      const float2 lo = __fadd2_rn(x[i], make_float2(-__uint_as_float(hi << 16), -__uint_as_float(hi & 0xffff0000u)));
      r[i] = hi;
      r[CH / 2 + i] = pack16<true>(lo.x, lo.y);
    } else {
      const float2 y = __fmul2_rn(x[i], make_float2(scale, scale));
      const uint32_t hi = pack16<false>(y.x, y.y);
      const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
      r[i] = hi;
      r[CH / 2 + i] = pack16<false>(y.x - h.x, y.y - h.y);
    }
  }
}

// Dense bias: a ring of CH-column chunks per compute warp (2 KB each: 32 lanes x 16 values), filled by asynchronous copies
// a half step (D = 64) or two chunks (D = 128, where the tiles leave no more room) ahead of their use.  Loads into
// registers one chunk ahead did not cover the L2 latency: 600 to 1900 cycles per chunk against 350 without a bias.  Rows
// of whole aligned 16-byte units are copied in such units, four copies per lane and chunk; others (an odd number of keys)
// 4 bytes at a time, sixteen.
template <int D>
constexpr int BIAS_RING = D > 64 ? 2 : 4;
constexpr int BIAS_SLOT = 32 * CH * 4;

__device__ __forceinline__ void copy4_async(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ float lds(uint32_t addr) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr) : "memory");
  return x;
}

// Thread-block clusters: shared memory of CTA `rank`, and a barrier of all threads.
__device__ __forceinline__ int cluster_size() {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return (int)n;
}
__device__ __forceinline__ int cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ float lds_cluster(uint32_t addr, int rank) {
  float x;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
               : "=f"(x)
               : "r"(addr), "r"(rank)
               : "memory");
  return x;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void copy16_async(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

// Keys on the lanes: keys key0 .. key0 + 31, rows i0 .. i0 + CH - 1 of a plane, rows and keys past the tensor clamped (their
// values are masked).  Slot layout [CH rows][32 keys].  Callers leave out chunks wholly past the tensor: clamped, they read
// the last row or key only, and with short sequences that share a plane every SM hit those few lines of the L2 (backward at
// B64 L64 H16 D64: 482 us with one plane, 107 with a plane per head; now 98 with either).
__device__ __forceinline__ void fetch_bias_column(uint32_t slot, const float* plane, int key0, int i0, int Lq, int Lkv, bool vec, int lane) {
  if (vec) {
    const float* src = plane + min(key0 + 4 * (lane & 7), Lkv - 4);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = 4 * e + (lane >> 3);
      copy16_async(slot + row * 128 + (lane & 7) * 16, src + (int64_t)min(i0 + row, Lq - 1) * Lkv);
    }
  } else {
    const float* ptr = plane + min(key0 + lane, Lkv - 1) + (int64_t)min(i0, Lq - 1) * Lkv;
#pragma unroll
    for (int e = 0; e < CH; ++e) {
      copy4_async(slot + (e * 32 + lane) * 4, ptr);
      ptr += i0 + e + 1 < Lq ? Lkv : 0;
    }
  }
}
__device__ __forceinline__ void read_bias_column(uint32_t slot, int lane, float (&out)[CH]) {
#pragma unroll
  for (int e = 0; e < CH; ++e) out[e] = lds(slot + (e * 32 + lane) * 4);
}
// Rows on the lanes: rows r0 .. r0 + 31 of keys j0 .. j0 + CH - 1, read a row per lane.  Slot layout [32 rows][4 units of 16
// bytes], unit c of row r at c ^ (r / 2 % 4): free of bank conflicts both ways.
__device__ __forceinline__ void fetch_bias_rows(uint32_t slot, const float* plane, int r0, int j0, int Lq, int Lkv, bool vec, int lane) {
  if (vec) {
    const int c = lane & 3;
    const float* src = plane + min(j0 + 4 * c, Lkv - 4);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = 8 * e + (lane >> 2);
      copy16_async(slot + r * 64 + (c ^ ((r >> 1) & 3)) * 16, src + (int64_t)min(r0 + r, Lq - 1) * Lkv);
    }
  } else {
    const int k = lane & 15;
    const float* src = plane + min(j0 + k, Lkv - 1);
#pragma unroll
    for (int e = 0; e < CH; ++e) {
      const int r = 2 * e + (lane >> 4);
      copy4_async(slot + r * 64 + ((k >> 2) ^ ((r >> 1) & 3)) * 16 + (k & 3) * 4, src + (int64_t)min(r0 + r, Lq - 1) * Lkv);
    }
  }
}
__device__ __forceinline__ void read_bias_row(uint32_t slot, int lane, float (&out)[CH]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(out[4 * c]), "=f"(out[4 * c + 1]), "=f"(out[4 * c + 2]), "=f"(out[4 * c + 3])
                 : "r"(slot + lane * 64 + (c ^ ((lane >> 1) & 3)) * 16)
                 : "memory");
}

// Chunks of a half step in straight line; with modifiers as a loop, whose code stays in the instruction cache.
template <int FEAT>
constexpr int UNROLL = (FEAT & 1) ? 2 : 4;

// The element (i, j) a column e of a chunk stands for.  ROWS: the thread owns query row i0 and the columns are
// keys j0 + e; otherwise it owns key j0 and the columns are query rows i0 + e.
struct Place {
  int kv_len, Lq, Lkv, band_lo, band_hi;
};

// Bit e of the result: column e is visible.
template <int FEAT, bool ROWS>
__device__ __forceinline__ uint32_t keep_bits(const Place& pl, const ScoreModView& mv, bool seg_mixed, int own_seg, int i0, int j0) {
  constexpr uint32_t ALL = (1u << CH) - 1;
  const int i_last = ROWS ? i0 : i0 + CH - 1, j_last = ROWS ? j0 + CH - 1 : j0;
  bool inside = j_last < pl.kv_len && i_last < pl.Lq && j_last <= i0 + pl.band_hi && j0 >= i_last + pl.band_lo;
  if constexpr ((FEAT & 1) != 0) {
    if (mv.row_limit) inside = inside && ROWS && j_last < mv.row_limit[min(i0, pl.Lq - 1)];
    inside = inside && !seg_mixed;
  }
  if (inside) return ALL;
  // the columns' ids and limits first, all loads in flight together (one at a time they cost a latency per column)
  [[maybe_unused]] int col_seg[CH], col_limit[CH];
  if constexpr ((FEAT & 1) != 0) {
    if (seg_mixed) {
      const int32_t* src = ROWS ? mv.seg_k : mv.seg_q;
      const int first = ROWS ? j0 : i0, last = (ROWS ? pl.Lkv : pl.Lq) - 1;
#pragma unroll
      for (int e = 0; e < CH; ++e) col_seg[e] = __ldg(src + min(first + e, last));
    }
    if (mv.row_limit) {
#pragma unroll
      for (int e = 0; e < CH; ++e) col_limit[e] = __ldg(mv.row_limit + min(ROWS ? i0 : i0 + e, pl.Lq - 1));
    }
  }
  // band, lengths and prefix are ranges of columns
  auto below = [](int e) { return (1u << max(0, min(CH, e))) - 1u; };  // bits of the columns before e
  uint32_t bits = ROWS ? below(i0 + pl.band_hi - j0 + 1) & ~below(i0 + pl.band_lo - j0)
                       : below(j0 - pl.band_lo - i0 + 1) & ~below(j0 - pl.band_hi - i0);
  if constexpr ((FEAT & 1) != 0) bits |= ROWS ? below(mv.prefix - j0) : (j0 < mv.prefix ? ALL : 0u);
  bits &= ROWS ? below(pl.kv_len - j0) : below(pl.Lq - i0);
  if (ROWS ? i0 >= pl.Lq : j0 >= pl.kv_len) bits = 0;
  if constexpr ((FEAT & 1) != 0) {
    if (seg_mixed) {
#pragma unroll
      for (int e = 0; e < CH; ++e) bits &= col_seg[e] == own_seg ? ALL : ALL ^ (1u << e);
    }
    if (mv.row_limit) {
#pragma unroll
      for (int e = 0; e < CH; ++e) bits &= (ROWS ? j0 + e : j0) < col_limit[e] ? ALL : ALL ^ (1u << e);
    }
  }
  return bits;
}

// P (dropped and rescaled under dropout) and dS of one chunk.  `lse` and `delta` hold one value (ROWS) or one per column.
// NL = false: no head_scale / softcap (refused together with a bias gradient).  Packed arithmetic (two columns per
// instruction) throughout: the issue slots of the compute warps are what bounds the modifier variants.
template <int FEAT, bool ROWS, bool NL = true>
__device__ __forceinline__ void chunk_p_ds(const float (&s)[CH], const float (&dp)[CH], float c, const Place& pl,
                                           const ScoreModView& mv, uint32_t keep, int i0, int j0, const float* lse,
                                           const float* delta, const float* bias, float2 (&pr)[CH / 2], float2 (&ds)[CH / 2]) {
  auto two = [](float x) { return make_float2(x, x); };
  auto at = [](const float* v, int e) { return ROWS ? make_float2(v[0], v[0]) : make_float2(v[e], v[e + 1]); };
  auto neg = [](float2 v) { return make_float2(-v.x, -v.y); };
  float2 y[CH / 2];  // exponents, base 2
  float2 g[CH / 2];  // d(modified score) / d(scaled score)
  const bool nonlinear = NL && (FEAT & 4) && (mv.hscale_m1 != 0.f || mv.softcap > 0.f);
  if (!(FEAT & 2) && !((FEAT & 1) && mv.rel) && !nonlinear) {
    // `lse` in base 2 here and below unless a table or a dense bias is added
    const float2 c2 = two(c * kLog2e);
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) y[i] = __ffma2_rn(make_float2(s[2 * i], s[2 * i + 1]), c2, neg(at(lse, 2 * i)));
    if ((FEAT & 1) && mv.alibi_mode) {
      const float base = (float)(i0 - j0);
      const float2 slope = two(-mv.slope * kLog2e);
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) {
        const float e = 2.f * i;
        float2 d = __fadd2_rn(two(base), ROWS ? make_float2(-e, -e - 1.f) : make_float2(e, e + 1.f));  // i - j, exact
        d = mv.alibi_mode == 1 ? make_float2(fmaxf(d.x, 0.f), fmaxf(d.y, 0.f)) : make_float2(fabsf(d.x), fabsf(d.y));
        y[i] = __ffma2_rn(d, slope, y[i]);
      }
    }
  } else {
    float2 x[CH / 2];
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) x[i] = __fmul2_rn(make_float2(s[2 * i], s[2 * i + 1]), two(c));
    if (nonlinear) {
      const float inv_cap = mv.softcap > 0.f ? 1.f / mv.softcap : 0.f;
      auto modify = [&](float sx, float& out, float& d) {
        out = fmaf(sx, mv.hscale_m1, sx);
        d = 1.f + mv.hscale_m1;
        if (mv.softcap > 0.f) {
          const float t = tanhf(sx * inv_cap);
          out += mv.softcap * t - sx;
          d -= t * t;
        }
      };
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) {
        float2 o;
        modify(x[i].x, o.x, g[i].x);
        modify(x[i].y, o.y, g[i].y);
        x[i] = o;
      }
    }
    if ((FEAT & 1) && mv.alibi_mode) {
      const float base = (float)(i0 - j0);
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) {
        const float e = 2.f * i;
        float2 d = __fadd2_rn(two(base), ROWS ? make_float2(-e, -e - 1.f) : make_float2(e, e + 1.f));
        d = mv.alibi_mode == 1 ? make_float2(fmaxf(d.x, 0.f), fmaxf(d.y, 0.f)) : make_float2(fabsf(d.x), fabsf(d.y));
        x[i] = __ffma2_rn(d, two(-mv.slope), x[i]);
      }
    }
    if ((FEAT & 1) && mv.rel) {
      auto entry = [&](int e) {  // clamped: rows and keys past the tensors
        return __ldg(mv.rel + max(1 - pl.Lq, min(pl.Lkv - 1, ROWS ? j0 + e - i0 : j0 - i0 - e)));
      };
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) x[i] = __fadd2_rn(x[i], make_float2(entry(2 * i), entry(2 * i + 1)));
    }
    if constexpr ((FEAT & 2) != 0) {
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) x[i] = __fadd2_rn(x[i], make_float2(bias[2 * i], bias[2 * i + 1]));
    }
    if ((FEAT & 2) || ((FEAT & 1) && mv.rel)) {
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) y[i] = __fmul2_rn(__fadd2_rn(x[i], neg(at(lse, 2 * i))), two(kLog2e));
    } else {
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) y[i] = __ffma2_rn(x[i], two(kLog2e), neg(at(lse, 2 * i)));
    }
  }
#pragma unroll
  for (int i = 0; i < CH / 2; ++i) pr[i] = make_float2(ex2_approx(y[i].x), ex2_approx(y[i].y));
  if ((FEAT & 4) && mv.drop_rate > 0.f) {
    // dV sees the dropped, rescaled probabilities and dP is dropped the same way; delta includes it already
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) {
      const int e = 2 * i;
      const float2 dm = make_float2(mod_dropout(mv, ROWS ? i0 : i0 + e, ROWS ? j0 + e : j0),
                                    mod_dropout(mv, ROWS ? i0 : i0 + e + 1, ROWS ? j0 + e + 1 : j0));
      ds[i] = __fmul2_rn(pr[i], __ffma2_rn(make_float2(dp[e], dp[e + 1]), dm, neg(at(delta, e))));
      pr[i] = __fmul2_rn(pr[i], dm);
    }
  } else {
#pragma unroll
    for (int i = 0; i < CH / 2; ++i)
      ds[i] = __fmul2_rn(pr[i], __fadd2_rn(make_float2(dp[2 * i], dp[2 * i + 1]), neg(at(delta, 2 * i))));
  }
  if (nonlinear) {
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) ds[i] = __fmul2_rn(ds[i], g[i]);
  }
  if (keep != (1u << CH) - 1) {  // selects, not products: masked scores may be anything
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) {
      const bool k0 = (keep >> (2 * i)) & 1u, k1 = (keep >> (2 * i + 1)) & 1u;
      pr[i] = make_float2(k0 ? pr[i].x : 0.f, k1 ? pr[i].y : 0.f);
      ds[i] = make_float2(k0 ? ds[i].x : 0.f, k1 ? ds[i].y : 0.f);
    }
  }
}

// Whether the ids of a warp's 32 own rows (or keys) and of `n` columns from c0 on are not all the same.
__device__ __forceinline__ bool segments_mixed(const int32_t* col_seg, int c0, int n, int limit, int own, int lane) {
  const int ref = __shfl_sync(0xffffffffu, own, 0);
  const int a = col_seg[min(c0 + lane, limit - 1)];
  const int b = col_seg[min(c0 + min(32 + lane, n - 1), limit - 1)];
  return !__all_sync(0xffffffffu, own == ref && a == ref && b == ref);
}

// Rows [kv_len, tile end) of a K or V tile hold anything (a cache tail that was never written) and 0 x NaN inside
// an accumulating product is not 0: one warp zeroes them in shared memory.
template <int SUB>
__device__ __forceinline__ void clear_rows(uint32_t tile, int first, int lane) {
  for (int r = first + lane; r < BN; r += 32) {
    const uint32_t row = tile + r * 128;
#pragma unroll
    for (int sub = 0; sub < SUB; ++sub)
#pragma unroll
      for (int u = 0; u < 8; ++u)
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(row + sub * BN * 128 + u * 16), "r"(0) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// dQ kernel
// ---------------------------------------------------------------------------------------------
template <int D, int DV, int FEAT>
struct DqCfg {
  static constexpr int SUBQ = D / 64, SUBV = DV / 64;  // 64-element (128-byte) column blocks of a row
  static constexpr int TQ = SUBQ * 128 * 128, TV = SUBV * 128 * 128;  // bytes of a 128-row tile
  // A K tile is held from its score products to its accumulation one step later and the next one is wanted half a step
  // after that: three stages.  dO, the other operand that stays for the whole loop, sits in tensor memory (DV / 2
  // columns, written once by the compute warps), which makes the room.
  static constexpr int KST = 3, VST = D > 128 ? 1 : 2;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = TQ;
  static constexpr int OFF_V = OFF_K + KST * TQ;
  static constexpr int OFF_BIAS = OFF_V + VST * TV;                    // dense bias: a ring per compute warp
  static constexpr int OFF_BAR = OFF_BIAS + ((FEAT & 2) ? 8 * BIAS_RING<D> * BIAS_SLOT : 0);
  // barriers: Q_FULL, K_FULL[3], K_EMPTY[3], V_FULL[2], V_EMPTY[2], SP_FULL[2], DS_FULL[2], DQ_FULL, K_CLEAN, DO_READY
  static constexpr int N_BAR = 18;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BAR * 8 + 16 + 1024;
  static constexpr int TMEM_COLS = 512;  // S 128 | dP 128 | dQ D | dO DV / 2
  static_assert(2 * BN + D + DV / 2 <= 512, "tensor memory has 512 columns");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

template <int D, int DV, bool BF16, int FEAT>
__global__ void __launch_bounds__(NTHREADS, 1)
bwd_dq_exact_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                          const __grid_constant__ CUtensorMap tm_v,
                          const __grid_constant__ BwdParams p, const __grid_constant__ ExactArgs a) {
  using C = DqCfg<D, DV, FEAT>;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = uniform(smem_u32(smem));
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR = [&](int i) { return bar0 + 8u * i; };
  const int Q_FULL = 0, K_FULL = 1, K_EMPTY = 4, V_FULL = 7, V_EMPTY = 9, SP_FULL = 11, DS_FULL = 13, DQ_FULL = 15, K_CLEAN = 16,
            DO_READY = 17;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + C::N_BAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int n_qt = (p.Lq + BM - 1) / BM;
  int tile, pair;
  work_item(blockIdx.x, n_qt, p.Hq * p.B, a.order_w, tile, pair);
  const int qt = n_qt - 1 - tile;  // the last query tiles see the most keys under a causal band
  const int h = pair % p.Hq, b = pair / p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const int q0 = qt * BM;

  int kv_len = p.Lkv;
  if (p.kv_lengths) kv_len = max(0, min(kv_len, p.kv_lengths[b]));
  // KV tiles any row of this query tile can see
  int kv_end = max(0, min(kv_len, min(q0 + BM, p.Lq) + p.band_hi));
  int kv_begin = max(0, q0 + p.band_lo);
  if constexpr ((FEAT & 1) != 0) {
    if (a.q_range) {
      const int32_t* r = a.q_range + ((int64_t)b * a.q_range_bs + qt) * 2;
      kv_begin = max(kv_begin, r[0]);
      kv_end = min(kv_end, r[1]);
    }
    if (p.mod.prefix_len) {  // prefix keys are visible to every row
      const int pre = min(kv_len, p.mod.prefix_len[b]);
      if (pre > 0) {
        kv_end = max(kv_end, pre);
        kv_begin = 0;
      }
    }
  }
  const int j_lo = kv_begin / BN;
  const int n = uniform(kv_begin < kv_end ? (kv_end + BN - 1) / BN - j_lo : 0);
  const int clean_j = uniform((n > 0 && (j_lo + n) * BN > kv_len) ? n - 1 : -1);  // a last tile with rows past the valid length

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::N_BAR; ++i)
      mbar_init(BAR(i), i == K_CLEAN ? 32u : ((i == DS_FULL || i == DS_FULL + 1) ? 128u : i == DO_READY ? 256u : 1u));
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);
  const uint32_t T_S = tmem, T_DP = tmem + BN, T_DQ = tmem + 2 * BN, T_DO = T_DQ + D;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && n > 0) {
      prefetch_tmap(&tm_q);
      prefetch_tmap(&tm_k);
      prefetch_tmap(&tm_v);
      mbar_arrive_expect_tx(BAR(Q_FULL), C::TQ);
#pragma unroll
      for (int s = 0; s < C::SUBQ; ++s) tma_load_4d(sbase + C::OFF_Q + s * BM * 128, &tm_q, BAR(Q_FULL), s * 64, h, q0, b);
      for (int j = 0; j < n; ++j) {
        const int ks = j % C::KST, vs = j % C::VST;
        if (!mbar_wait(BAR(K_EMPTY + ks), ((j / C::KST) & 1) ^ 1, abort_flag)) break;
        mbar_arrive_expect_tx(BAR(K_FULL + ks), C::TQ);
#pragma unroll
        for (int s = 0; s < C::SUBQ; ++s)
          tma_load_4d(sbase + C::OFF_K + ks * C::TQ + s * BN * 128, &tm_k, BAR(K_FULL + ks), s * 64, hk, (j_lo + j) * BN, b);
        if (!mbar_wait(BAR(V_EMPTY + vs), ((j / C::VST) & 1) ^ 1, abort_flag)) break;
        mbar_arrive_expect_tx(BAR(V_FULL + vs), C::TV);
#pragma unroll
        for (int s = 0; s < C::SUBV; ++s)
          tma_load_4d(sbase + C::OFF_V + vs * C::TV + s * BN * 128, &tm_v, BAR(V_FULL + vs), s * 64, hk, (j_lo + j) * BN, b);
      }
    }
    __syncwarp();
    if (clean_j >= 0) {
      const int ks = clean_j % C::KST;
      if (mbar_wait(BAR(K_FULL + ks), (clean_j / C::KST) & 1, abort_flag)) {
        clear_rows<C::SUBQ>(sbase + C::OFF_K + ks * C::TQ, kv_len - (j_lo + clean_j) * BN, lane);
        fence_proxy_async();
      }
      mbar_arrive(BAR(K_CLEAN));
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (n > 0) {
      const uint32_t leader = elect_leader();
      constexpr uint32_t idesc_s = make_idesc(BM, BN / 2, BF16, false, false);
      constexpr uint32_t idesc_q = make_idesc(BM, D, BF16, false, true);
      const uint32_t qa = sbase + C::OFF_Q;
      // S and dP of one half (64 keys) of KV tile j
      auto issue_sdp = [&](int half, int j) {
        const uint32_t ka = sbase + C::OFF_K + (j % C::KST) * C::TQ + half * 64 * 128;
        const uint32_t va = sbase + C::OFF_V + (j % C::VST) * C::TV + half * 64 * 128;
#pragma unroll
        for (int s = 0; s < C::SUBQ; ++s)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ss(T_S + half * 64, make_smem_desc(qa + s * BM * 128 + kk * 32, 16, 1024),
                   make_smem_desc(ka + s * BN * 128 + kk * 32, 16, 1024), idesc_s, (s | kk) != 0, leader);
#pragma unroll
        for (int s = 0; s < C::SUBV; ++s)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ts(T_DP + half * 64, T_DO + (s * 4 + kk) * 8, make_smem_desc(va + s * BN * 128 + kk * 32, 16, 1024), idesc_s,
                   (s | kk) != 0, leader);
        mma_commit(BAR(SP_FULL + half), leader);
      };
      // dQ += (hi + lo of dS).K over one half, the K tile read MN-major
      auto issue_acc = [&](int half, int j) {
        const uint32_t ka = sbase + C::OFF_K + (j % C::KST) * C::TQ;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const uint64_t kd = make_smem_desc(ka + (half * 4 + kk) * 2048, BN * 128, 1024);
          mma_ts(T_DQ, T_S + half * 64 + kk * CH, kd, idesc_q, (j | half | kk) != 0, leader);
          mma_ts(T_DQ, T_S + half * 64 + kk * CH + CH / 2, kd, idesc_q, true, leader);
        }
      };
      bool ok = mbar_wait_all(BAR(Q_FULL), 0, abort_flag);
      if (ok) ok = mbar_wait_all(BAR(DO_READY), 0, abort_flag);
      if (ok) ok = mbar_wait_all(BAR(K_FULL), 0, abort_flag);
      if (ok && clean_j == 0) ok = mbar_wait_all(BAR(K_CLEAN), 0, abort_flag);
      if (ok) ok = mbar_wait_all(BAR(V_FULL), 0, abort_flag);
      if (ok) {
        tc_fence_after();
        issue_sdp(0, 0);
        issue_sdp(1, 0);
        mma_commit(BAR(V_EMPTY), leader);
      }
      for (int j = 0; ok && j < n; ++j) {
        const bool next = j + 1 < n;
        ok = mbar_wait_all(BAR(DS_FULL + 0), j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_acc(0, j);
        if (next) {
          ok = mbar_wait_all(BAR(K_FULL + (j + 1) % C::KST), ((j + 1) / C::KST) & 1, abort_flag);
          if (ok && j + 1 == clean_j) ok = mbar_wait_all(BAR(K_CLEAN), 0, abort_flag);
          if (ok) ok = mbar_wait_all(BAR(V_FULL + (j + 1) % C::VST), ((j + 1) / C::VST) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          issue_sdp(0, j + 1);  // over dS of half 0, which the MMAs just issued consume first
        }
        ok = mbar_wait_all(BAR(DS_FULL + 1), j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_acc(1, j);
        mma_commit(BAR(K_EMPTY + j % C::KST), leader);
        if (next) {
          issue_sdp(1, j + 1);
          mma_commit(BAR(V_EMPTY + (j + 1) % C::VST), leader);
        }
      }
      if (ok) mma_commit(BAR(DQ_FULL), leader);
    }
  } else {
    // --------------------------------------------------------------- compute warps
    const int grp = (warp - 2) >> 2;  // which half of the score columns
    const int quarter = warp & 3;
    const int r_in = quarter * 32 + lane;
    const int row = q0 + r_in;
    const bool row_ok = row < p.Lq;
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    [[maybe_unused]] float do_sq[2] = {0.f, 0.f};  // fp16: sum of squares of this group's half of the row's dO, of the other's
    if (n > 0) {  // this group's half of the row's dO into tensor memory: the A operand of dP
      const uint4* src = reinterpret_cast<const uint4*>(static_cast<const unsigned char*>(p.d_o) +
                                                        (((int64_t)b * p.Lq + min(row, p.Lq - 1)) * p.Hq + h) * DV * 2);
#pragma unroll
      for (int side = 0; side < (BF16 ? 1 : 2); ++side) {
#pragma unroll
        for (int u = 0; u < DV / 64; ++u) {  // 16 columns (32 elements) at a time
          uint32_t r[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 w = row_ok ? __ldg(src + (side ? 1 - grp : grp) * (DV / 16) + u * 4 + i) : make_uint4(0u, 0u, 0u, 0u);
            r[4 * i] = w.x;
            r[4 * i + 1] = w.y;
            r[4 * i + 2] = w.z;
            r[4 * i + 3] = w.w;
          }
          if (side == 0) tmem_st16(T_DO + lane_sel + grp * (DV / 4) + u * 16, r);
          if constexpr (!BF16) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r[i]));
              do_sq[side] = fmaf(f.x, f.x, fmaf(f.y, f.y, do_sq[side]));
            }
          }
        }
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(BAR(DO_READY));
    }
    const float c = p.sm_scale;
    // padded per-row vectors: +inf / 0 for rows past Lq and +inf for rows without keys, so P = 0 there
    const int64_t at = ((int64_t)b * p.Hq + h) * p.Lq_pad + row;
    const float lse = p.lse2[at], delta = p.delta[at];
    // fp16: |dS| <= P (keep |dO||v_j| + |delta|) |ds'/ds|, packed below 2^15; the two groups, which share the row of the
    // accumulator, arrive at the same value (the sum of the halves does not depend on their order)
    float pack = 1.f;
    [[maybe_unused]] uint32_t* col_max = nullptr;
    if constexpr (!BF16) {
      col_max = a.col_max + ((int64_t)b * p.Hkv + hk) * 2 * p.Lkv;
      const float* norms = a.v_norm + ((int64_t)b * p.Hkv + hk) * ((p.Lkv + BN - 1) / BN) + j_lo;
      float v_max = 0.f;
      for (int t = lane; t < n; t += 32) v_max = fmaxf(v_max, __ldg(norms + t));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v_max = fmaxf(v_max, __shfl_xor_sync(0xffffffffu, v_max, o));
      float bound = sqrtf(do_sq[0] + do_sq[1]) * v_max;
      if constexpr ((FEAT & 4) != 0) {
        if (p.mod.dropout_rate > 0.f) bound /= 1.f - p.mod.dropout_rate;
      }
      bound += fabsf(delta);
      if constexpr ((FEAT & 4) != 0) {  // ds'/ds is head_scale, or under a cap between head_scale - 1 and head_scale
        if (p.mod.head_scale) bound *= 1.f + fabsf(p.mod.head_scale[h]);
      }
      pack = pack_scale(bound, 14);
    }
    const uint32_t s_addr = T_S + lane_sel + grp * 64, dp_addr = T_DP + lane_sel + grp * 64;
    const Place pl = {kv_len, p.Lq, p.Lkv, p.band_lo, p.band_hi};
    ScoreModView mv = {};
    int own_seg = 0;
    if constexpr ((FEAT & 1) != 0) {
      mv = view_of(p.mod, b, h, p.Lq);
      if (mv.seg_q) own_seg = mv.seg_q[min(row, p.Lq - 1)];
    }
    constexpr int NB = BIAS_RING<D>;
    [[maybe_unused]] const uint32_t ring = sbase + C::OFF_BIAS + (warp - 2) * NB * BIAS_SLOT;
    [[maybe_unused]] const float* bsrc = (FEAT & 2) ? p.bias + (int64_t)b * p.bias_bs + (int64_t)h * p.bias_hs : nullptr;
    // chunk t of this warp: CH keys, four chunks per tile; the chunks before t_end have a row and a key within the tensor
    const int keys = p.Lkv - j_lo * BN - grp * 64;
    [[maybe_unused]] const int t_end =
        q0 + quarter * 32 < p.Lq && keys > 0 ? min(4 * n, keys / BN * 4 + min(4, (keys % BN + CH - 1) / CH)) : 0;
    auto fetch_bias = [&](int t) {
      if (t < t_end)
        fetch_bias_rows(ring + (t % NB) * BIAS_SLOT, bsrc, q0 + quarter * 32, (j_lo + t / 4) * BN + grp * 64 + (t % 4) * CH, p.Lq,
                        p.Lkv, a.bias_vec, lane);
      copy_commit();
    };
    if constexpr ((FEAT & 2) != 0) {
      for (int t = 0; t < NB; ++t) fetch_bias(t);
    }
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int k0 = (j_lo + j) * BN + grp * 64;  // first key of this group's columns
      bool mixed = false;
      if constexpr ((FEAT & 1) != 0) {
        if (mv.seg_q) mixed = segments_mixed(mv.seg_k, k0, 64, p.Lkv, own_seg, lane);
      }
      ok = mbar_wait(BAR(SP_FULL + grp), j & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      float s_next[CH], dp_next[CH];
      tmem_ld16f(s_addr, s_next);
      tmem_ld16f(dp_addr, dp_next);
#pragma unroll(UNROLL<FEAT>)
      for (int cc = 0; cc < 64 / CH; ++cc) {
        tmem_wait_ld();
        float s[CH], dp[CH];
#pragma unroll
        for (int e = 0; e < CH; ++e) {
          s[e] = s_next[e];
          dp[e] = dp_next[e];
        }
        if (cc + 1 < 64 / CH) {
          tmem_ld16f(s_addr + (cc + 1) * CH, s_next);
          tmem_ld16f(dp_addr + (cc + 1) * CH, dp_next);
        }
        float bias[CH];
        float2 pr[CH / 2], ds[CH / 2];
        if constexpr ((FEAT & 2) != 0) {
          copy_wait<NB - 1>();
          __syncwarp();
          read_bias_row(ring + (cc % NB) * BIAS_SLOT, lane, bias);
          __syncwarp();  // the slot has been read by all lanes
          fetch_bias(4 * j + cc + NB);
        }
        const int j0 = k0 + cc * CH;
        const uint32_t keep = keep_bits<FEAT, true>(pl, mv, mixed, own_seg, row, j0);
        chunk_p_ds<FEAT, true>(s, dp, c, pl, mv, keep, row, j0, &lse, &delta, bias, pr, ds);
        if constexpr (!BF16) add_col_max(pr, ds, dp, col_max + j0, p.Lkv - j0, p.Lkv, lane);
        uint32_t pk[CH];
        split_pack<BF16>(ds, pack, pk);
        tmem_st16(s_addr + cc * CH, pk);  // over the chunk's own scores, which were read already
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(BAR(DS_FULL + grp));
    }
    if constexpr ((FEAT & 2) != 0) copy_wait<0>();  // none in flight at the exit, should a wait have expired
    if (ok && q0 < p.Lq) {
      if (n > 0) {
        ok = mbar_wait(BAR(DQ_FULL), 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok) {
        tc_fence_after();
        // each group stores one half of the row's D columns
        unsigned char* dst = static_cast<unsigned char*>(p.dq) + ((((int64_t)b * p.Lq + row) * p.Hq + h) * D) * 2;
        store_row<D / 2, BF16>(T_DQ + lane_sel + grp * (D / 2), dst + grp * D, p.sm_scale / pack, n > 0, row_ok);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, C::TMEM_COLS);
    if (lane == 0 && *abort_flag && p.status) atomicExch(p.status, (int)PJX_ERR_DEVICE_TIMEOUT);
  }
}

// ---------------------------------------------------------------------------------------------
// dK/dV kernel
// ---------------------------------------------------------------------------------------------
template <int D, int DV, int FEAT>
struct DkvCfg {
  static constexpr int SUBQ = D / 64, SUBV = DV / 64;
  static constexpr int QT = D > 128 ? 96 : 128;      // query rows per step: S^T | dP^T | dV | dK fill tensor memory
  static constexpr int HALF = QT / 2;
  static constexpr int TK = SUBQ * BN * 128, TV = SUBV * BN * 128;
  // Q and dO travel as half tiles (a slot: HALF rows of Q | of dO), the unit the issuer works in; a slot is free as soon
  // as its half has been accumulated.
  static constexpr int HQ = SUBQ * HALF * 128, HDO = SUBV * HALF * 128, SLOT = HQ + HDO;
  static constexpr int NS = D > 128 || (D > 64 && (FEAT & 2)) ? 4 : D > 64 ? 5 : 6;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = TK;
  static constexpr int OFF_Q = OFF_V + TV;
  static constexpr int OFF_ROW = OFF_Q + NS * SLOT;  // NS x { float lse[HALF]; float delta[HALF]; }
  static constexpr int OFF_BIAS = OFF_ROW + NS * 2 * HALF * 4;
  static constexpr int OFF_BAR = OFF_BIAS + ((FEAT & 2) ? 8 * BIAS_RING<D> * BIAS_SLOT : 0);
  // barriers: KV_FULL, QDO_FULL[NS], QDO_EMPTY[NS], SP_FULL[2], PDS_FULL[2], ACC_FULL
  static constexpr int N_BAR = 2 * NS + 6;
  // alignment slack: the dynamic shared memory of a kernel without static one starts at a multiple of 1024; the kernel
  // reports an error instead of running should it ever not
  static constexpr int SLACK = 256;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BAR * 8 + 16 + SLACK;
  static constexpr int TMEM_COLS = 512;              // S^T QT | dP^T QT | dV DV | dK D
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static_assert(2 * QT + DV + D <= 512, "tensor memory has 512 columns");
  static_assert(HALF % CH == 0 && (HALF * 128) % 1024 == 0, "halves are whole chunks and whole swizzle groups");
};

template <int D, int DV, bool BF16, int FEAT>
__global__ void __launch_bounds__(NTHREADS, 1)
bwd_dkdv_exact_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                            const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                            const __grid_constant__ BwdParams p, const __grid_constant__ ExactArgs a) {
  using C = DkvCfg<D, DV, FEAT>;
  constexpr int QT = C::QT, HALF = C::HALF, NCH = HALF / CH;
  extern __shared__ __align__(1024) unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = uniform(smem_u32(smem));
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR = [&](int i) { return bar0 + 8u * i; };
  constexpr int NS = C::NS;
  const int KV_FULL = 0, QDO_FULL = 1, QDO_EMPTY = QDO_FULL + NS, SP_FULL = QDO_EMPTY + NS, PDS_FULL = SP_FULL + 2,
            ACC_FULL = PDS_FULL + 2;
  if (smem - smem_unaligned > C::SLACK) {
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, (int)PJX_ERR_CUDA);
    return;
  }
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + C::N_BAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* row_s = reinterpret_cast<float*>(smem + C::OFF_ROW);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  int kt, pair;  // the first key tiles are seen by the most queries under a causal band
  work_item(blockIdx.x, (p.Lkv + BN - 1) / BN, p.Hkv * p.B, a.order_w, kt, pair);
  const int hk = pair % p.Hkv, b = pair / p.Hkv;
  const int G = p.Hq / p.Hkv;
  const int k0 = kt * BN;

  int kv_len = p.Lkv;
  if (p.kv_lengths) kv_len = max(0, min(kv_len, p.kv_lengths[b]));
  // query rows that see a key of this tile: [first key - band_hi, last valid key - band_lo]
  int q_begin = max(0, k0 - p.band_hi);
  int q_end = min(p.Lq, min(k0 + BN, kv_len) - p.band_lo);
  if constexpr ((FEAT & 1) != 0) {
    if (a.k_range) {
      const int32_t* r = a.k_range + ((int64_t)b * a.k_range_bs + kt) * 2;
      q_begin = max(q_begin, r[0]);
      q_end = min(q_end, r[1]);
    }
    if (p.mod.prefix_len && k0 < p.mod.prefix_len[b]) {  // a prefix key is seen by every row
      q_begin = 0;
      q_end = p.Lq;
    }
  }
  const int t_lo = q_begin / QT;
  const int n_t = (k0 < kv_len && q_begin < q_end) ? (q_end + QT - 1) / QT - t_lo : 0;
  const int n = uniform(n_t * G);  // steps: query heads of the group outer, query tiles inner

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::N_BAR; ++i)
      mbar_init(BAR(i), (i == PDS_FULL || i == PDS_FULL + 1) ? 128u : 1u);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);
  const uint32_t T_S = tmem, T_DP = tmem + QT, T_DV = tmem + 2 * QT, T_DK = tmem + 2 * QT + DV;

  if (warp == 0) {
    // ------------------------------------------------------------------- TMA producer
    if (lane == 0 && n > 0) {
      prefetch_tmap(&tm_q);
      prefetch_tmap(&tm_do);
      prefetch_tmap(&tm_k);
      prefetch_tmap(&tm_v);
      mbar_arrive_expect_tx(BAR(KV_FULL), C::TK + C::TV);
#pragma unroll
      for (int s = 0; s < C::SUBQ; ++s) tma_load_4d(sbase + C::OFF_K + s * BN * 128, &tm_k, BAR(KV_FULL), s * 64, hk, k0, b);
#pragma unroll
      for (int s = 0; s < C::SUBV; ++s) tma_load_4d(sbase + C::OFF_V + s * BN * 128, &tm_v, BAR(KV_FULL), s * 64, hk, k0, b);
      for (int hh = 0; hh < 2 * n; ++hh) {  // half tiles: step hh / 2, rows HALF (hh & 1) ..
        const int st = hh % NS, it = hh >> 1;
        const int h = hk * G + it / n_t;
        const int q0 = (t_lo + it % n_t) * QT + (hh & 1) * HALF;
        const uint32_t slot = sbase + C::OFF_Q + st * C::SLOT, rows_at = sbase + C::OFF_ROW + st * 2 * HALF * 4;
        // the rows' log-sum-exp and delta out of the padded workspace arrays (a 96-row tile may reach past their padding,
        // or lie past it with its second half: a multiple of 4 floats either way)
        const int rows = QT == 128 ? HALF : max(0, min(HALF, p.Lq_pad - q0));
        if (!mbar_wait(BAR(QDO_EMPTY + st), ((hh / NS) & 1) ^ 1, abort_flag)) break;
        mbar_arrive_expect_tx(BAR(QDO_FULL + st), C::SLOT + 2 * rows * 4);
#pragma unroll
        for (int s = 0; s < C::SUBQ; ++s) tma_load_4d(slot + s * HALF * 128, &tm_q, BAR(QDO_FULL + st), s * 64, h, q0, b);
#pragma unroll
        for (int s = 0; s < C::SUBV; ++s) tma_load_4d(slot + C::HQ + s * HALF * 128, &tm_do, BAR(QDO_FULL + st), s * 64, h, q0, b);
        if (rows > 0) {
          const int64_t at = ((int64_t)b * p.Hq + h) * p.Lq_pad + q0;
          bulk_load(rows_at, p.lse2 + at, rows * 4, BAR(QDO_FULL + st));
          bulk_load(rows_at + HALF * 4, p.delta + at, rows * 4, BAR(QDO_FULL + st));
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (n > 0) {
      const uint32_t leader = elect_leader();
      constexpr uint32_t idesc_s = make_idesc(BN, HALF, BF16, false, false);
      constexpr uint32_t idesc_v = make_idesc(BN, DV, BF16, false, true);
      constexpr uint32_t idesc_k = make_idesc(BN, D, BF16, false, true);
      const uint32_t ka = sbase + C::OFF_K, va = sbase + C::OFF_V;
      // S^T and dP^T of one half of step `it`: keys on the lanes, query rows on the columns
      auto issue_sdp = [&](int half, int it) {
        const uint32_t qa = sbase + C::OFF_Q + (2 * it + half) % NS * C::SLOT, doa = qa + C::HQ;
#pragma unroll
        for (int s = 0; s < C::SUBQ; ++s)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ss(T_S + half * HALF, make_smem_desc(ka + s * BN * 128 + kk * 32, 16, 1024),
                   make_smem_desc(qa + s * HALF * 128 + kk * 32, 16, 1024), idesc_s, (s | kk) != 0, leader);
#pragma unroll
        for (int s = 0; s < C::SUBV; ++s)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ss(T_DP + half * HALF, make_smem_desc(va + s * BN * 128 + kk * 32, 16, 1024),
                   make_smem_desc(doa + s * HALF * 128 + kk * 32, 16, 1024), idesc_s, (s | kk) != 0, leader);
        mma_commit(BAR(SP_FULL + half), leader);
      };
      // dV += (hi + lo of P^T).dO and dK += (hi + lo of dS^T).Q over one half, dO / Q tiles read MN-major
      auto issue_acc = [&](int half, int it) {
        const uint32_t qa = sbase + C::OFF_Q + (2 * it + half) % NS * C::SLOT, doa = qa + C::HQ;
#pragma unroll
        for (int kk = 0; kk < NCH; ++kk) {
          const uint64_t dd = make_smem_desc(doa + kk * 2048, HALF * 128, 1024);
          mma_ts(T_DV, T_S + half * HALF + kk * CH, dd, idesc_v, (it | half | kk) != 0, leader);
          mma_ts(T_DV, T_S + half * HALF + kk * CH + CH / 2, dd, idesc_v, true, leader);
        }
#pragma unroll
        for (int kk = 0; kk < NCH; ++kk) {
          const uint64_t qd = make_smem_desc(qa + kk * 2048, HALF * 128, 1024);
          mma_ts(T_DK, T_DP + half * HALF + kk * CH, qd, idesc_k, (it | half | kk) != 0, leader);
          mma_ts(T_DK, T_DP + half * HALF + kk * CH + CH / 2, qd, idesc_k, true, leader);
        }
        mma_commit(BAR(QDO_EMPTY + (2 * it + half) % NS), leader);
      };
      auto half_landed = [&](int hh) { return mbar_wait_all(BAR(QDO_FULL + hh % NS), (hh / NS) & 1, abort_flag); };
      bool ok = mbar_wait_all(BAR(KV_FULL), 0, abort_flag);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (ok) ok = half_landed(half);
        if (ok) {
          tc_fence_after();
          issue_sdp(half, 0);
        }
      }
      for (int it = 0; ok && it < n; ++it) {
        const bool next = it + 1 < n;
        ok = mbar_wait_all(BAR(PDS_FULL + 0), it & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_acc(0, it);
        if (next) {
          ok = half_landed(2 * it + 2);
          if (!ok) break;
          tc_fence_after();
          issue_sdp(0, it + 1);  // over P^T / dS^T of half 0, which the MMAs just issued consume first
        }
        ok = mbar_wait_all(BAR(PDS_FULL + 1), it & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_acc(1, it);
        if (next) {
          ok = half_landed(2 * it + 3);
          if (!ok) break;
          tc_fence_after();
          issue_sdp(1, it + 1);
        }
      }
      if (ok) mma_commit(BAR(ACC_FULL), leader);
    }
  } else {
    // --------------------------------------------------------------- compute warps
    const int grp = (warp - 2) >> 2;  // which half of the query columns
    const int quarter = warp & 3;
    const int r_in = quarter * 32 + lane;
    const int key = k0 + r_in;
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    const float c = p.sm_scale;
    // fp16: the key's own scales; two bits more room than the dQ kernel's maxima, whose products summed in another order
    float pack = 1.f, pack_p = 1.f;
    if constexpr (!BF16) {
      const uint32_t* col_max = a.col_max + ((int64_t)b * p.Hkv + hk) * 2 * p.Lkv + min(key, p.Lkv - 1);
      pack = pack_scale(__uint_as_float(col_max[0]), 12);
      pack_p = pack_scale(__uint_as_float(col_max[p.Lkv]), 12);
    }
    const uint32_t s_addr = T_S + lane_sel + grp * HALF, dp_addr = T_DP + lane_sel + grp * HALF;
    const Place pl = {kv_len, p.Lq, p.Lkv, p.band_lo, p.band_hi};
    ScoreModView mv = {};
    int own_seg = 0;
    constexpr int NB = BIAS_RING<D>;
    [[maybe_unused]] const uint32_t ring = sbase + C::OFF_BIAS + (warp - 2) * NB * BIAS_SLOT;
    // dense bias: position of the next chunk to fetch (chunk of the half, query tile, head of the group)
    [[maybe_unused]] int f_cc = 0, f_t = 0, f_g = n > 0 && k0 + quarter * 32 < p.Lkv ? 0 : G;
    [[maybe_unused]] const float* bsrc =
        (FEAT & 2) ? p.bias + (int64_t)b * p.bias_bs + (int64_t)hk * G * p.bias_hs : nullptr;
    auto fetch_bias = [&](int slot) {
      const int i0 = (t_lo + f_t) * QT + grp * HALF + f_cc * CH;
      if (f_g < G && i0 < p.Lq)
        fetch_bias_column(ring + slot * BIAS_SLOT, bsrc + (int64_t)f_g * p.bias_hs, k0 + quarter * 32, i0, p.Lq, p.Lkv, a.bias_vec, lane);
      copy_commit();
      if (++f_cc == NCH) {
        f_cc = 0;
        if (++f_t == n_t) {
          f_t = 0;
          ++f_g;
        }
      }
    };
    if constexpr ((FEAT & 2) != 0) {
      static_assert(!(FEAT & 2) || NCH % NB == 0, "slots follow the chunk index");
      for (int t = 0; t < NB; ++t) fetch_bias(t);
    }
    bool ok = true;
    for (int it = 0; it < n; ++it) {
      const int st = (2 * it + grp) % NS;
      const int q0 = (t_lo + it % n_t) * QT + grp * HALF;  // first query row of this group's columns
      bool mixed = false;
      if (it % n_t == 0) {  // the next query head of the group
        const int h = hk * G + it / n_t;
        if constexpr ((FEAT & 1) != 0) {
          mv = view_of(p.mod, b, h, p.Lq);
          if (mv.seg_q) own_seg = mv.seg_k[min(key, p.Lkv - 1)];
        }
      }
      if constexpr ((FEAT & 1) != 0) {
        if (mv.seg_q) mixed = segments_mixed(mv.seg_q, q0, HALF, p.Lq, own_seg, lane);
      }
      ok = mbar_wait(BAR(SP_FULL + grp), it & 1, abort_flag);
      if (ok) ok = mbar_wait(BAR(QDO_FULL + st), ((2 * it + grp) / NS) & 1, abort_flag);  // the row vectors landed with Q and dO
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float* lse_s = row_s + st * 2 * HALF;
      const float* delta_s = lse_s + HALF;
      float s_next[CH], dp_next[CH];
      tmem_ld16f(s_addr, s_next);
      tmem_ld16f(dp_addr, dp_next);
#pragma unroll(UNROLL<FEAT>)
      for (int cc = 0; cc < NCH; ++cc) {
        float lse[CH], delta[CH], bias[CH];
        float2 pr[CH / 2], ds[CH / 2];
#pragma unroll
        for (int e = 0; e < CH; e += 4) {
          *reinterpret_cast<float4*>(lse + e) = *reinterpret_cast<const float4*>(lse_s + cc * CH + e);
          *reinterpret_cast<float4*>(delta + e) = *reinterpret_cast<const float4*>(delta_s + cc * CH + e);
        }
        if constexpr ((FEAT & 2) != 0) {
          copy_wait<NB - 1>();
          __syncwarp();
          read_bias_column(ring + (cc % NB) * BIAS_SLOT, lane, bias);
          __syncwarp();  // the slot has been read by all lanes
          fetch_bias(cc % NB);
        }
        tmem_wait_ld();
        float s[CH], dp[CH];
#pragma unroll
        for (int e = 0; e < CH; ++e) {
          s[e] = s_next[e];
          dp[e] = dp_next[e];
        }
        if (cc + 1 < NCH) {
          tmem_ld16f(s_addr + (cc + 1) * CH, s_next);
          tmem_ld16f(dp_addr + (cc + 1) * CH, dp_next);
        }
        const int i0 = q0 + cc * CH;
        const uint32_t keep = keep_bits<FEAT, false>(pl, mv, mixed, own_seg, i0, key);
        chunk_p_ds<FEAT, false>(s, dp, c, pl, mv, keep, i0, key, lse, delta, bias, pr, ds);
        uint32_t pk[CH];
        split_pack<BF16>(pr, pack_p, pk);
        tmem_st16(s_addr + cc * CH, pk);  // over the chunk's own scores, which were read already
        split_pack<BF16>(ds, pack, pk);
        tmem_st16(dp_addr + cc * CH, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(BAR(PDS_FULL + grp));
    }
    if constexpr ((FEAT & 2) != 0) copy_wait<0>();
    if (ok && k0 < p.Lkv) {
      if (n > 0) {
        ok = mbar_wait(BAR(ACC_FULL), 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok) {
        tc_fence_after();
        const bool row_ok = key < p.Lkv;
        const int64_t at = ((int64_t)b * p.Lkv + key) * p.Hkv + hk;
        // group 0 stores the dV row, group 1 the dK row
        if (grp == 0) store_row<DV, BF16>(T_DV + lane_sel, static_cast<unsigned char*>(p.dv) + at * DV * 2, 1.f / pack_p, n > 0, row_ok);
        else store_row<D, BF16>(T_DK + lane_sel, static_cast<unsigned char*>(p.dk) + at * D * 2, p.sm_scale / pack, n > 0, row_ok);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, C::TMEM_COLS);
    if (lane == 0 && *abort_flag && p.status) atomicExch(p.status, (int)PJX_ERR_DEVICE_TIMEOUT);
  }
}

// ---------------------------------------------------------------------------------------------
// Gradient of the dense bias: dbias = sum of dS over the (batch, head) pairs that share an entry
// ---------------------------------------------------------------------------------------------
// One CTA per 128 x 128 tile of the bias.  S^T and dP^T of successive pairs alternate between the two halves of
// tensor memory, so that the products of the next pair run while the threads (one key, 64 query rows each) add dS
// of this one to their 64 registers; the tile is written once, coalesced over the keys.  Summing in registers
// costs two products per pair and no memory traffic; adding dS into memory from the dQ kernel instead would move
// 4 bytes per score through the L2's atomic units (537 MB at B8 S1024 H16) in an order that changes per run.
// Where the tiles leave SMs idle and many pairs share them (short sequences, a bias shared by the heads) a cluster of up to
// sixteen CTAs shares a tile: each walks a slice of the pairs and keeps its sum in shared memory, then each adds up a slice of
// the rows over the cluster in rank order.  One CTA per tile took 1.4 us per pair: B64 L64 H16 D64 with one plane (1024
// pairs, one tile) 1474 us for the whole backward, against 344 on the CUDA cores; with up
// to eight 236, with up to sixteen 172.
template <int D, int DV>
struct DbCfg {
  static constexpr int SUBQ = D / 64, SUBV = DV / 64;
  static constexpr int TQ = SUBQ * 128 * 128, TV = SUBV * 128 * 128;
  static constexpr int STAGE = 2 * TQ + 2 * TV;                  // Q | K | dO | V
  static constexpr int NST = STAGE <= 72 * 1024 ? 2 : 1;
  static constexpr int OFF_BIAS = NST * STAGE;                   // the tile of the bias, 128 x 128 fp32
  static constexpr int OFF_ROW = OFF_BIAS + BM * BN * 4;         // 2 x { float lse[128]; float delta[128]; }
  static constexpr int OFF_BAR = OFF_ROW + 2 * 2 * BM * 4;
  // barriers: FULL[NST], EMPTY[NST], ROW_FULL[2], SP_FULL[2], T_FREE[2]
  static constexpr int N_BAR = 2 * NST + 6;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BAR * 8 + 16 + 1024;
  static constexpr int TMEM_COLS = 512;                          // 2 x { S^T 128 | dP^T 128 }
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

template <int D, int DV, bool BF16, int FEAT, bool CLUSTER>
__global__ void __launch_bounds__(NTHREADS, 1)
bwd_dbias_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                       const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const __grid_constant__ BwdParams p) {
  using C = DbCfg<D, DV>;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = uniform(smem_u32(smem));
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR = [&](int i) { return bar0 + 8u * i; };
  const int FULL = 0, EMPTY = C::NST, ROW_FULL = 2 * C::NST, SP_FULL = ROW_FULL + 2, T_FREE = SP_FULL + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + C::N_BAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* row_s = reinterpret_cast<float*>(smem + C::OFF_ROW);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int n_kt = (p.Lkv + BN - 1) / BN, n_qt = (p.Lq + BM - 1) / BM;
  auto n_ranks = [] { return CLUSTER ? cluster_size() : 1; };  // (read where they are needed: nothing held over the loop)
  auto rank = [] { return CLUSTER ? cluster_rank() : 0; };
  const int item = blockIdx.x / n_ranks();
  const int k0 = item % n_kt * BN, q0 = item / n_kt % n_qt * BM;
  const int plane = item / (n_kt * n_qt);  // (batch, head) plane of the bias
  const int nhb = p.bias_hs ? p.Hq : 1;
  // the pairs of this plane: b0 .. b0 + nb - 1 times h0 .. h0 + nh - 1
  const int h0 = p.bias_hs ? plane % nhb : 0, nh = p.bias_hs ? 1 : p.Hq;
  const int b0 = p.bias_bs ? plane / nhb : 0, nb = p.bias_bs ? 1 : p.B;
  const bool in_band = p.mod.prefix_len || (k0 <= min(q0 + BM, p.Lq) - 1 + p.band_hi && min(k0 + BN, p.Lkv) - 1 >= q0 + p.band_lo);
  // this CTA's slice of them
  const int64_t n_all = in_band ? (int64_t)nb * nh : 0;
  const int pi_begin = (int)(n_all * rank() / n_ranks()), pi_end = (int)(n_all * (rank() + 1) / n_ranks());
  const int G = p.Hq / p.Hkv;
  auto len_of = [&](int b) { return p.kv_lengths ? max(0, min(p.Lkv, p.kv_lengths[b])) : p.Lkv; };

  if (threadIdx.x == 0) {
    // compute warps with rows and keys within the tensor; the others keep out of the loop
    const int active = min(4, (p.Lkv - k0 + 31) / 32) * (q0 + 64 < p.Lq ? 2 : 1);
    for (int i = 0; i < C::N_BAR; ++i) mbar_init(BAR(i), i >= T_FREE ? 32u * active : 1u);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);

  // every role walks the pairs the same way; `it` counts those with a valid key in the tile
  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int pi = pi_begin; pi < pi_end; ++pi) {
        const int b = b0 + pi / nh, h = h0 + pi % nh, hk = h / G;
        if (k0 >= len_of(b)) continue;
        const int st = it % C::NST, buf = it & 1;
        const uint32_t sa = sbase + st * C::STAGE;
        if (!mbar_wait(BAR(EMPTY + st), ((it / C::NST) & 1) ^ 1, abort_flag)) break;
        mbar_arrive_expect_tx(BAR(FULL + st), C::STAGE);
#pragma unroll
        for (int s = 0; s < C::SUBQ; ++s) {
          tma_load_4d(sa + s * BM * 128, &tm_q, BAR(FULL + st), s * 64, h, q0, b);
          tma_load_4d(sa + C::TQ + s * BN * 128, &tm_k, BAR(FULL + st), s * 64, hk, k0, b);
        }
#pragma unroll
        for (int s = 0; s < C::SUBV; ++s) {
          tma_load_4d(sa + 2 * C::TQ + s * BM * 128, &tm_do, BAR(FULL + st), s * 64, h, q0, b);
          tma_load_4d(sa + 2 * C::TQ + C::TV + s * BN * 128, &tm_v, BAR(FULL + st), s * 64, hk, k0, b);
        }
        if (!mbar_wait(BAR(T_FREE + buf), ((it >> 1) & 1) ^ 1, abort_flag)) break;  // row vectors of pair it - 2 were read
        mbar_arrive_expect_tx(BAR(ROW_FULL + buf), 2 * BM * 4);
        const int64_t at = ((int64_t)b * p.Hq + h) * p.Lq_pad + q0;
        bulk_load(sbase + C::OFF_ROW + buf * 2 * BM * 4, p.lse2 + at, BM * 4, BAR(ROW_FULL + buf));
        bulk_load(sbase + C::OFF_ROW + buf * 2 * BM * 4 + BM * 4, p.delta + at, BM * 4, BAR(ROW_FULL + buf));
        ++it;
      }
    }
  } else if (warp == 1) {
    {
      const uint32_t leader = elect_leader();
      constexpr uint32_t idesc = make_idesc(BN, BM, BF16, false, false);
      int it = 0;
      for (int pi = pi_begin; pi < pi_end; ++pi) {
        if (uniform(static_cast<int>(k0 >= len_of(b0 + pi / nh)))) continue;
        const int st = it % C::NST, buf = it & 1;
        const uint32_t sa = sbase + st * C::STAGE;
        if (!mbar_wait_all(BAR(FULL + st), (it / C::NST) & 1, abort_flag)) break;
        if (!mbar_wait_all(BAR(T_FREE + buf), ((it >> 1) & 1) ^ 1, abort_flag)) break;
        tc_fence_after();
#pragma unroll
        for (int s = 0; s < C::SUBQ; ++s)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ss(tmem + buf * 256, make_smem_desc(sa + C::TQ + s * BN * 128 + kk * 32, 16, 1024),
                   make_smem_desc(sa + s * BM * 128 + kk * 32, 16, 1024), idesc, (s | kk) != 0, leader);
#pragma unroll
        for (int s = 0; s < C::SUBV; ++s)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ss(tmem + buf * 256 + 128, make_smem_desc(sa + 2 * C::TQ + C::TV + s * BN * 128 + kk * 32, 16, 1024),
                   make_smem_desc(sa + 2 * C::TQ + s * BM * 128 + kk * 32, 16, 1024), idesc, (s | kk) != 0, leader);
        mma_commit(BAR(EMPTY + st), leader);
        mma_commit(BAR(SP_FULL + buf), leader);
        ++it;
      }
    }
  } else {
    const int grp = (warp - 2) >> 2, quarter = warp & 3;
    const int key = k0 + quarter * 32 + lane;
    const int i_first = q0 + grp * 64;
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    const float* bsrc = p.bias + (int64_t)b0 * p.bias_bs + (int64_t)h0 * p.bias_hs + min(key, p.Lkv - 1);
    // every pair adds the same tile of the bias: read from memory once, each thread keeps its values in shared memory
    const uint32_t btile = sbase + C::OFF_BIAS + grp * 64 * BN * 4 + (quarter * 32 + lane) * 4;
    if (pi_begin < pi_end) {
      for (int e = 0; e < 64; e += 8) {
        float t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) t[u] = __ldg(bsrc + (int64_t)min(i_first + e + u, p.Lq - 1) * p.Lkv);
#pragma unroll
        for (int u = 0; u < 8; ++u) asm volatile("st.shared.f32 [%0], %1;" ::"r"(btile + (e + u) * BN * 4), "f"(t[u]) : "memory");
      }
    }
    float2 acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = make_float2(0.f, 0.f);
    int it = 0;
    bool ok = true;
    const int pi_stop = i_first < p.Lq && k0 + quarter * 32 < p.Lkv ? pi_end : pi_begin;
    for (int pi = pi_begin; pi < pi_stop; ++pi) {
      const int b = b0 + pi / nh, h = h0 + pi % nh;
      const int kv_len = len_of(b);
      if (k0 >= kv_len) continue;
      const int buf = it & 1;
      const Place pl = {kv_len, p.Lq, p.Lkv, p.band_lo, p.band_hi};
      ScoreModView mv = {};
      int own_seg = 0;
      bool mixed = false;
      if constexpr ((FEAT & 1) != 0) {
        mv = view_of(p.mod, b, h, p.Lq);
        if (mv.seg_q) {
          own_seg = mv.seg_k[min(key, p.Lkv - 1)];
          mixed = segments_mixed(mv.seg_q, i_first, 64, p.Lq, own_seg, lane);
        }
      }
      // with modifiers the mask of all chunks ahead of the wait and out of the straight line below, whose code and registers
      // it fills otherwise
      [[maybe_unused]] uint64_t visible = 0;
      if constexpr ((FEAT & 1) != 0) {
#pragma unroll 1
        for (int cc = 0; cc < 64 / CH; ++cc)
          visible |= (uint64_t)keep_bits<FEAT, false>(pl, mv, mixed, own_seg, i_first + cc * CH, key) << (CH * cc);
      }
      const uint32_t s_addr = tmem + buf * 256 + lane_sel + grp * 64, dp_addr = s_addr + 128;
      ok = mbar_wait(BAR(SP_FULL + buf), (it >> 1) & 1, abort_flag);
      if (ok) ok = mbar_wait(BAR(ROW_FULL + buf), (it >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float* lse_s = row_s + buf * 2 * BM + grp * 64;
      const float* delta_s = lse_s + BM;
#pragma unroll
      for (int cc = 0; cc < 64 / CH; ++cc) {
        float s[CH], dp[CH], lse[CH], delta[CH], bias[CH];
        float2 pr[CH / 2], ds[CH / 2];
        tmem_ld16f(s_addr + cc * CH, s);
        tmem_ld16f(dp_addr + cc * CH, dp);
#pragma unroll
        for (int e = 0; e < CH; e += 4) {
          *reinterpret_cast<float4*>(lse + e) = *reinterpret_cast<const float4*>(lse_s + cc * CH + e);
          *reinterpret_cast<float4*>(delta + e) = *reinterpret_cast<const float4*>(delta_s + cc * CH + e);
        }
#pragma unroll
        for (int e = 0; e < CH; ++e) bias[e] = lds(btile + (cc * CH + e) * BN * 4);
        tmem_wait_ld();
        int i0 = i_first + cc * CH;
        asm volatile("" : "+r"(i0));  // the tests below do not change over the pairs: not all of them ahead of the loop
        const uint32_t keep = (FEAT & 1) ? (uint32_t)(visible >> (CH * cc)) & ((1u << CH) - 1)
                                         : keep_bits<FEAT, false>(pl, mv, mixed, own_seg, i0, key);
        chunk_p_ds<FEAT, false, false>(s, dp, p.sm_scale, pl, mv, keep, i0, key, lse, delta, bias, pr, ds);
#pragma unroll
        for (int i = 0; i < CH / 2; ++i) acc[cc * CH / 2 + i] = __fadd2_rn(acc[cc * CH / 2 + i], ds[i]);
      }
      tc_fence_before();
      mbar_arrive(BAR(T_FREE + buf));
      ++it;
    }
    if constexpr (CLUSTER) {
#pragma unroll
      for (int e = 0; e < 64; ++e)
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(btile + e * BN * 4), "f"(e % 2 ? acc[e / 2].y : acc[e / 2].x) : "memory");
    } else if (ok && key < p.Lkv) {
      float* dst = p.dbias + (int64_t)b0 * p.bias_bs + (int64_t)h0 * p.bias_hs + key;
#pragma unroll
      for (int e = 0; e < 64; ++e)
        if (i_first + e < p.Lq) dst[(int64_t)(i_first + e) * p.Lkv] = e % 2 ? acc[e / 2].y : acc[e / 2].x;
    }
  }

  if constexpr (CLUSTER) {
    // (after a wait that expired in one of the CTAs the sum means nothing: the status word says so)
    cluster_sync();
    const int rows = BM / n_ranks(), row0 = rank() * rows, n = n_ranks();
    const int64_t plane_at = (int64_t)b0 * p.bias_bs + (int64_t)h0 * p.bias_hs;
    for (int u = threadIdx.x; u < rows * BN; u += NTHREADS) {
      const int i = q0 + row0 + u / BN, j = k0 + u % BN;
      const uint32_t mine = sbase + C::OFF_BIAS + (row0 * BN + u) * 4;
      float sum = 0.f;
      for (int r = 0; r < n; ++r) sum += lds_cluster(mine, r);
      if (i < p.Lq && j < p.Lkv) p.dbias[plane_at + (int64_t)i * p.Lkv + j] = sum;
    }
    cluster_sync();  // a CTA's shared memory outlives the reads of the others
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, C::TMEM_COLS);
    if (lane == 0 && *abort_flag && p.status) atomicExch(p.status, (int)PJX_ERR_DEVICE_TIMEOUT);
  }
}

// ---------------------------------------------------------------------------------------------
// fp16: the longest V row (2-norm) of each key tile, rows past the valid length and rows that are not finite left out
// ---------------------------------------------------------------------------------------------
template <int DV>
__global__ void __launch_bounds__(256) v_norm_kernel(const BwdParams p, float* out) {
  constexpr int LPR = DV / 8, ROWS = 256 / LPR;  // lanes per row (16 bytes each), rows at a time
  __shared__ float warp_max[8];
  const int n_kt = (p.Lkv + BN - 1) / BN;
  const int k0 = (int)(blockIdx.x % n_kt) * BN, pair = blockIdx.x / n_kt;
  const int hk = pair % p.Hkv, b = pair / p.Hkv;
  const int u = threadIdx.x % LPR;
  const int k_end = min(min(k0 + BN, p.Lkv), p.kv_lengths ? p.kv_lengths[b] : p.Lkv);
  float m = 0.f;
#pragma unroll
  for (int r = 0; r < BN / ROWS; ++r) {
    const int j = k0 + r * ROWS + (int)threadIdx.x / LPR;
    float sq = 0.f;
    if (j < k_end) {
      const uint4 w = __ldg(static_cast<const uint4*>(p.v) + (((int64_t)b * p.Lkv + j) * p.Hkv + hk) * LPR + u);
      const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&x[i]));
        sq = fmaf(f.x, f.x, fmaf(f.y, f.y, sq));
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (sq < INFINITY) m = fmaxf(m, sq);  // not for inf, nor for NaN
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x % 32 == 0) warp_max[threadIdx.x / 32] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) m = fmaxf(m, warp_max[i]);
    out[blockIdx.x] = sqrtf(m);
  }
}

template <typename... Params, typename... Args>
int launch_kernel(void (*kern)(Params...), int64_t grid, int smem, int cluster, cudaStream_t stream, const char* what,
                  const Args&... args) {
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), what);
  if (!rc && cluster > 8) rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), what);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  rc = check_cuda(cudaLaunchKernelEx(&cfg, kern, args...), what);
  count_launch();
  return rc;
}

// CTAs that share a tile of the bias gradient: as many as the SMs take, each with four pairs or more (below that the exchange
// costs what the shorter walk saves).  Sixteen, for a tile or a few that thousands of pairs share, is past the portable size:
// only as many such clusters as the device says find their SMs at a time (seven on this part; with eight planes of B1024 L64 H8
// a second wave of one cluster took as long as clusters of eight).
template <typename K>
int dbias_cluster(K kern, int smem, int64_t tiles, int64_t pairs) {
  static std::atomic<int> sixteen[64];  // clusters of sixteen at a time on each device: 0 not asked yet, -1 none
  int dev = 0, sms = 148, n = 1;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  while (n < 16 && 2 * n * tiles <= sms && pairs >= 8 * n) n *= 2;
  if (n < 16) return n;
  if (dev < 0 || dev >= 64) return 8;
  if (sixteen[dev] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 16;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int fit = 0;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) == cudaSuccess && fit > 0;
    if (!ok) (void)cudaGetLastError();
    sixteen[dev] = ok ? fit : -1;
  }
  return tiles <= sixteen[dev] ? 16 : 8;
}

template <int D, int DV, bool BF16, int FEAT>
int launch_dbias(const BwdParams& p, const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tk, const CUtensorMap& tv,
                 cudaStream_t stream) {
  constexpr int SMEM = DbCfg<D, DV>::SMEM_BYTES;
  const char* what = "sm100 dbias launch";
  const int64_t planes = (int64_t)(p.bias_bs ? p.B : 1) * (p.bias_hs ? p.Hq : 1);
  const int64_t tiles = planes * ((p.Lq + BM - 1) / BM) * ((p.Lkv + BN - 1) / BN);
  auto shared = bwd_dbias_sm100_kernel<D, DV, BF16, FEAT, true>;
  const int cluster = dbias_cluster(shared, SMEM, tiles, (int64_t)p.B * p.Hq / planes);
  if (cluster > 1) return launch_kernel(shared, tiles * cluster, SMEM, cluster, stream, what, tq, tdo, tk, tv, p);
  return launch_kernel(bwd_dbias_sm100_kernel<D, DV, BF16, FEAT, false>, tiles, SMEM, 1, stream, what, tq, tdo, tk, tv, p);
}

template <int D, int DV, bool BF16, int FEAT>
int launch_feat(const BwdParams& p, const ExactArgs& a, cudaStream_t stream) {
  using Q = DqCfg<D, DV, FEAT>;
  using KV = DkvCfg<D, DV, FEAT>;
  CUtensorMap tq, tdo, tk, tv, tq2, tdo2;
  int rc;
  if ((rc = make_tmap_blhd(&tq, p.q, p.dtype, p.B, p.Lq, p.Hq, D, BM))) return rc;
  if ((rc = make_tmap_blhd(&tdo, p.d_o, p.dtype, p.B, p.Lq, p.Hq, DV, BM))) return rc;
  if ((rc = make_tmap_blhd(&tk, p.k, p.dtype, p.B, p.Lkv, p.Hkv, D, BN))) return rc;
  if ((rc = make_tmap_blhd(&tv, p.v, p.dtype, p.B, p.Lkv, p.Hkv, DV, BN))) return rc;
  if ((rc = make_tmap_blhd(&tq2, p.q, p.dtype, p.B, p.Lq, p.Hq, D, KV::HALF))) return rc;
  if ((rc = make_tmap_blhd(&tdo2, p.d_o, p.dtype, p.B, p.Lq, p.Hq, DV, KV::HALF))) return rc;
  const int64_t n_q = (p.Lq + BM - 1) / BM, n_k = (p.Lkv + BN - 1) / BN;
  if ((rc = launch_kernel(bwd_dq_exact_sm100_kernel<D, DV, BF16, FEAT>, n_q * p.Hq * p.B, Q::SMEM_BYTES, 1, stream,
                          "sm100 exact dq launch", tq, tk, tv, p, a)))
    return rc;
  if ((rc = launch_kernel(bwd_dkdv_exact_sm100_kernel<D, DV, BF16, FEAT>, n_k * p.Hkv * p.B, KV::SMEM_BYTES, 1, stream,
                          "sm100 exact dk/dv launch", tq2, tdo2, tk, tv, p, a)))
    return rc;
  if constexpr ((FEAT & 2) != 0) {
    if (p.dbias) {
      // of head scale, soft cap and dropout only dropout comes with the gradient of a bias
      return p.mod.dropout_rate > 0.f ? launch_dbias<D, DV, BF16, FEAT>(p, tq, tdo, tk, tv, stream)
                                      : launch_dbias<D, DV, BF16, FEAT & 3>(p, tq, tdo, tk, tv, stream);
    }
  }
  return PJX_OK;
}

template <int D, bool BF16>
int launch_square(const BwdParams& p, const ExactArgs& a, cudaStream_t stream) {
  const bool heavy = p.mod.head_scale || p.mod.softcap > 0.f || p.mod.dropout_rate > 0.f;
  if (!p.bias) return heavy ? launch_feat<D, D, BF16, 5>(p, a, stream) : launch_feat<D, D, BF16, 1>(p, a, stream);
  return p.mod.on ? launch_feat<D, D, BF16, 7>(p, a, stream) : launch_feat<D, D, BF16, 2>(p, a, stream);
}

template <bool BF16>
int launch_shape(const BwdParams& p, const ExactArgs& a, cudaStream_t stream) {
  if (p.D == 192) return p.mod.on ? launch_feat<192, 128, BF16, 5>(p, a, stream) : launch_feat<192, 128, BF16, 0>(p, a, stream);
  return p.D == 128 ? launch_square<128, BF16>(p, a, stream) : launch_square<64, BF16>(p, a, stream);
}

}  // namespace

// 16-bit calls of the tensor-core head shapes that the two kernels of attn_bwd_sm100.cu do not take.  The dense bias
// at (192, 128) stays on the CUDA cores: its staging window does not fit beside the tiles.
bool bwd_exact_sm100_supported(const BwdParams& p) {
  if (p.dtype != PJX_BF16 && p.dtype != PJX_F16) return false;
  const bool square = p.D == p.Dv && (p.D == 64 || p.D == 128);
  if (!square && !(p.D == 192 && p.Dv == 128 && !p.bias)) return false;
  if (p.B < 1 || p.Lq < 1 || p.Lkv < 1) return false;
  const int64_t n_q = (p.Lq + BM - 1) / BM, n_k = (p.Lkv + BN - 1) / BN, planes = (int64_t)p.Hq * p.B;
  if (n_q * planes > 0x7fffffffLL || n_k * planes > 0x7fffffffLL || (p.dbias && n_q * n_k > 0x7fffffffLL / planes)) return false;
  if ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) |
       reinterpret_cast<uintptr_t>(p.d_o) | reinterpret_cast<uintptr_t>(p.dq) | reinterpret_cast<uintptr_t>(p.dk) |
       reinterpret_cast<uintptr_t>(p.dv) | reinterpret_cast<uintptr_t>(p.delta)) & 15)
    return false;
  return true;
}

// Scratch: [fp16: longest V rows | maxima of the keys] [segment ranges both ways], 4-byte words.  fp16 needs its part; the
// ranges only spare work and are left out where there is no room for them.
static size_t fp16_words(const BwdParams& p) {
  return p.dtype == PJX_F16 ? (size_t)p.B * p.Hkv * ((p.Lkv + BN - 1) / BN + 2 * (size_t)p.Lkv) : 0;
}

int launch_bwd_exact_sm100(const BwdParams& p, void* scratch, size_t scratch_bytes, cudaStream_t stream) {
  ExactArgs a = {};
  a.order_w = (p.band_hi < PJX_BAND_NO_UPPER && p.band_lo == PJX_BAND_NO_LOWER) ? 16 : 1;
  a.bias_vec = p.bias && p.Lkv % 4 == 0 && p.bias_bs % 4 == 0 && p.bias_hs % 4 == 0 && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
  int rc;
  if (p.dtype == PJX_F16) {
    const size_t tiles = (size_t)p.B * p.Hkv * ((p.Lkv + BN - 1) / BN);
    float* norms = static_cast<float*>(scratch);
    a.v_norm = norms;
    a.col_max = static_cast<uint32_t*>(scratch) + tiles;
    if ((rc = check_cuda(cudaMemsetAsync(a.col_max, 0, (fp16_words(p) - tiles) * 4, stream), "clear maxima"))) return rc;
    if (p.Dv == 64) v_norm_kernel<64><<<(unsigned)tiles, 256, 0, stream>>>(p, norms);
    else v_norm_kernel<128><<<(unsigned)tiles, 256, 0, stream>>>(p, norms);
    count_launch();
    if ((rc = check_cuda(cudaGetLastError(), "backward V norm launch"))) return rc;
  }
  if (bwd_exact_uses_ranges(p) && scratch_bytes >= bwd_exact_scratch_bytes(p)) {
    const int n_q = (p.Lq + BM - 1) / BM, n_k = (p.Lkv + BN - 1) / BN;
    const int nb = (p.mod.seg_q_bs == 0 && p.mod.seg_k_bs == 0) ? 1 : p.B;
    int32_t* qr = static_cast<int32_t*>(scratch) + fp16_words(p);
    int32_t* kr = qr + (int64_t)nb * n_q * 2;
    launch_seg_tile_range(p.mod.seg_q, p.mod.seg_k, p.mod.seg_q_bs, p.mod.seg_k_bs, p.Lq, p.Lkv, n_q, nb, qr, stream);
    launch_seg_tile_range(p.mod.seg_k, p.mod.seg_q, p.mod.seg_k_bs, p.mod.seg_q_bs, p.Lkv, p.Lq, n_k, nb, kr, stream);
    if ((rc = check_cuda(cudaGetLastError(), "segment ranges launch"))) return rc;
    a.q_range = qr;
    a.k_range = kr;
    a.q_range_bs = nb == 1 ? 0 : n_q;
    a.k_range_bs = nb == 1 ? 0 : n_k;
  }
  return p.dtype == PJX_BF16 ? launch_shape<true>(p, a, stream) : launch_shape<false>(p, a, stream);
}

// Segment masks cut the tile loops (prefix keys are visible to every row: no ranges then).
bool bwd_exact_uses_ranges(const BwdParams& p) {
  return p.mod.seg_q && p.mod.seg_k && !p.mod.prefix_len && p.B <= 65535;
}

size_t bwd_exact_scratch_bytes(const BwdParams& p) {
  size_t n = fp16_words(p) * 4;
  if (bwd_exact_uses_ranges(p)) n += (size_t)p.B * ((p.Lq + BM - 1) / BM + (p.Lkv + BN - 1) / BN) * 2 * sizeof(int32_t);
  return n;
}

size_t bwd_exact_scratch_bytes_needed(const BwdParams& p) { return fp16_words(p) * 4; }

}  // namespace pjx
