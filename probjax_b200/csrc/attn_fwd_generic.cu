// Generic flash-attention forward: exact fp32 FMA arithmetic on CUDA cores.
//
// Computes any call the C ABI accepts (fp32 / bf16 / fp16, any head width up to
// 256, ragged lengths, causal + key-length masks, dense bias).  It is the kernel
// for fp32 inputs -- tensor cores would round them to TF32, which misses the
// 1e-4 parity bound -- and for shapes the tcgen05 kernel does not take.
//
// Math follows the reference's forward kernel
// (probjax/nn/pallas_kernels/kernels/attention.py:456-529): scores in fp32,
// times sm_scale, plus bias, masked, exp2-domain online softmax, P rounded to the
// input dtype before P.V, final division by the row sum.
//
// One CTA owns a tile of 64 or 32 queries (RT = 4 or 2 rows per thread) of one (batch, query head) and walks the KV
// sequence in 64-key tiles staged in shared memory as fp32.  Threads form a 16 x 16 grid; thread (ty, tx) owns score
// rows RT*ty .. RT*ty+RT-1 and columns tx + 16*c, and the same rows of the output with columns 4*tx .. 4*tx+3 + 64*c.
// Bound by shared-memory loads: every inner loop reads 16 bytes per load (B2 L250 H4 D64 fp32: 84 -> 32 us
// together with the smaller tile, which doubles the CTAs of grids that leave SMs idle).
#include "pjx_common.cuh"

namespace pjx {
namespace {

constexpr int BN = 64;
constexpr int PP = BN + 4;  // pitch of the P tile
constexpr int NT = 256;

__host__ __device__ inline int pitch4(int d) { return (d + 3) / 4 * 4 + 4; }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}
__device__ __forceinline__ void axpy4(float4& s, float a, float4 x) {
  s.x = fmaf(a, x.x, s.x);
  s.y = fmaf(a, x.y, s.y);
  s.z = fmaf(a, x.z, s.z);
  s.w = fmaf(a, x.w, s.w);
}

// ROWS rows of `width` elements into a tile of pitch4(width), rows at or past `limit` and the padding up to the next
// multiple of 4 as zeros; 8 threads per row.  fp32 rows of whole aligned 16-byte units are copied as such.
template <typename T, int ROWS>
__device__ __forceinline__ void load_tile(float* dst, int pitch, const T* src, int64_t row_stride, int first, int limit, int width) {
  const bool vec = sizeof(T) == 4 && width % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  const int u = threadIdx.x & 7;
#pragma unroll
  for (int r = threadIdx.x >> 3; r < ROWS; r += NT / 8) {
    const int g = first + r;
    const T* row = src + (int64_t)g * row_stride;
    if (vec) {
      for (int d = u * 4; d < width; d += 32)
        *reinterpret_cast<float4*>(dst + r * pitch + d) =
            g < limit ? __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(row) + d)) : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      for (int d = u; d < (width + 3) / 4 * 4; d += 8) dst[r * pitch + d] = g < limit && d < width ? Elem<T>::to_f(row[d]) : 0.f;
    }
  }
}

template <typename T, int NCOL, int RT>  // NCOL: groups of four output columns per thread
__global__ void __launch_bounds__(NT) attn_fwd_generic_kernel(const FwdParams p) {
  extern __shared__ float smem[];
  constexpr int BM = 16 * RT;
  const int D = p.D, Dv = p.Dv;
  const int Dp = pitch4(D), Dvp = pitch4(Dv);
  float* Qs = smem;                 // [BM][Dp]
  float* Ks = Qs + BM * Dp;         // [BN][Dp]
  float* Vs = Ks + BN * Dp;         // [BN][Dvp]
  float* Ps = Vs + BN * Dvp;        // [BM][PP]

  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int q0 = blockIdx.x * BM, h = blockIdx.y, b = blockIdx.z;
  const int hk = h / (p.Hq / p.Hkv);
  const T* q = static_cast<const T*>(p.q);
  const T* k = static_cast<const T*>(p.k);
  const T* v = static_cast<const T*>(p.v);

  int kv_len = p.Lkv;
  if (p.kv_lengths) kv_len = max(0, min(kv_len, p.kv_lengths[b]));
  // keys outside [first query + band_lo, last query + band_hi] of the tile are masked for all its rows
  int kv_end = max(0, min(kv_len, min(q0 + BM, p.Lq) + p.band_hi));
  const int kv_begin = (max(0, q0 + p.band_lo) / BN) * BN;
  const bool has_mod = p.mod.on != 0;
  ScoreModView mv = {};
  if (has_mod) {
    mv = view_of(p.mod, b, h, p.Lq);
    kv_end = max(kv_end, min(kv_len, mv.prefix));  // prefix keys are visible to every row
  }

  load_tile<T, BM>(Qs, Dp, q + ((int64_t)b * p.Lq * p.Hq + h) * D, (int64_t)p.Hq * D, q0, p.Lq, D);

  float m[RT], l[RT];
  float4 acc[RT][NCOL];
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < NCOL; ++c) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float c1 = p.sm_scale * kLog2e;
  const float* bias = nullptr;
  if (p.bias) bias = p.bias + (int64_t)b * p.bias_bs + (int64_t)h * p.bias_hs;

  for (int k0 = kv_begin; k0 < kv_end; k0 += BN) {
    __syncthreads();  // previous tile fully consumed (also orders the Q staging)
    load_tile<T, BN>(Ks, Dp, k + ((int64_t)b * p.Lkv * p.Hkv + hk) * D, (int64_t)p.Hkv * D, k0, kv_len, D);
    load_tile<T, BN>(Vs, Dvp, v + ((int64_t)b * p.Lkv * p.Hkv + hk) * Dv, (int64_t)p.Hkv * Dv, k0, kv_len, Dv);
    __syncthreads();

    float s[RT][4];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[i][c] = 0.f;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 qv[RT], kv[4];
#pragma unroll
      for (int i = 0; i < RT; ++i) qv[i] = ld4(Qs + (ty * RT + i) * Dp + d);
#pragma unroll
      for (int c = 0; c < 4; ++c) kv[c] = ld4(Ks + (tx + 16 * c) * Dp + d);
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[i][c] = dot4(qv[i], kv[c], s[i][c]);
    }

    // scale -> bias -> mask, in the exp2 domain
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int qi = q0 + ty * RT + i;
      float tmax = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int kj = k0 + tx + 16 * c;
        float x = s[i][c] * c1;
        bool keep = kj <= qi + p.band_hi && kj >= qi + p.band_lo;
        if (has_mod && qi < p.Lq && kj < kv_len) {
          x = mod_score<true>(mv, s[i][c] * p.sm_scale, qi, kj, nullptr) * kLog2e;
          keep = mod_keep(mv, keep, qi, kj);
        }
        if (bias && qi < p.Lq && kj < p.Lkv) x = fmaf(bias[(int64_t)qi * p.Lkv + kj], kLog2e, x);
        keep = keep && (kj < kv_len);
        x = keep ? x : -INFINITY;
        s[i][c] = x;
        tmax = fmaxf(tmax, x);
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, off));
      const float m_new = fmaxf(m[i], tmax);
      const float m_safe = (m_new == -INFINITY) ? 0.f : m_new;
      const float corr = exp2f(m[i] - m_safe);
      float rsum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float pv = exp2f(s[i][c] - m_safe);
        rsum += pv;  // the row sum is taken before dropout (kernels/attention.py:497-505)
        const float dm = has_mod ? mod_dropout(mv, qi, k0 + tx + 16 * c) : 1.f;
        Ps[(ty * RT + i) * PP + tx + 16 * c] = Elem<T>::round(pv * dm);
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) rsum += __shfl_xor_sync(0xffffffffu, rsum, off);
      l[i] = l[i] * corr + rsum;
      m[i] = m_new;
#pragma unroll
      for (int c = 0; c < NCOL; ++c) {
        acc[i][c].x *= corr;
        acc[i][c].y *= corr;
        acc[i][c].z *= corr;
        acc[i][c].w *= corr;
      }
    }
    __syncthreads();

#pragma unroll 2
    for (int kk = 0; kk < BN; kk += 4) {
      float4 pv[RT];
#pragma unroll
      for (int i = 0; i < RT; ++i) pv[i] = ld4(Ps + (ty * RT + i) * PP + kk);
#pragma unroll
      for (int c = 0; c < NCOL; ++c) {
        const int d = tx * 4 + 64 * c;
        if (d >= Dv) break;
        const float* vr = Vs + kk * Dvp + d;
        const float4 v0 = ld4(vr), v1 = ld4(vr + Dvp), v2 = ld4(vr + 2 * Dvp), v3 = ld4(vr + 3 * Dvp);
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          axpy4(acc[i][c], pv[i].x, v0);
          axpy4(acc[i][c], pv[i].y, v1);
          axpy4(acc[i][c], pv[i].z, v2);
          axpy4(acc[i][c], pv[i].w, v3);
        }
      }
    }
  }

  T* o = static_cast<T*>(p.o);
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const int qi = q0 + ty * RT + i;
    if (qi >= p.Lq) continue;
    const bool nonempty = l[i] > 0.f;
    const float inv = nonempty ? 1.f / l[i] : 0.f;
#pragma unroll
    for (int c = 0; c < NCOL; ++c) {
      const float x[4] = {acc[i][c].x, acc[i][c].y, acc[i][c].z, acc[i][c].w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int d = tx * 4 + 64 * c + u;
        if (d < Dv) o[(((int64_t)b * p.Lq + qi) * p.Hq + h) * Dv + d] = Elem<T>::from_f(x[u] * inv);
      }
    }
    if (p.lse && tx == 0)
      p.lse[((int64_t)b * p.Hq + h) * p.Lq + qi] = nonempty ? (m[i] + log2f(l[i])) * kLn2 : INFINITY;
  }
}

template <typename T, int NCOL, int RT>
int launch_t(const FwdParams& p, cudaStream_t stream) {
  constexpr int BM = 16 * RT;
  const size_t smem = sizeof(float) * ((size_t)(BM + BN) * pitch4(p.D) + (size_t)BN * pitch4(p.Dv) + (size_t)BM * PP);
  auto kern = attn_fwd_generic_kernel<T, NCOL, RT>;
  if (smem > 48 * 1024) {
    int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                        "cudaFuncSetAttribute(generic fwd)");
    if (rc) return rc;
  }
  dim3 grid((p.Lq + BM - 1) / BM, p.Hq, p.B);
  kern<<<grid, NT, smem, stream>>>(p);
  count_launch();
  return check_cuda(cudaGetLastError(), "generic forward launch");
}

// Tiles of 32 queries while 64-query tiles would not give every SM two CTAs.
template <typename T, int NCOL>
int launch_rows(const FwdParams& p, cudaStream_t stream) {
  const int64_t ctas = (int64_t)((p.Lq + 63) / 64) * p.Hq * p.B;
  return ctas < 296 ? launch_t<T, NCOL, 2>(p, stream) : launch_t<T, NCOL, 4>(p, stream);
}

template <typename T>
int launch_d(const FwdParams& p, cudaStream_t stream) {
  if (p.Dv <= 64) return launch_rows<T, 1>(p, stream);
  if (p.Dv <= 128) return launch_rows<T, 2>(p, stream);
  return launch_rows<T, 4>(p, stream);
}

}  // namespace

int launch_fwd_generic(const FwdParams& p, int dtype, cudaStream_t stream) {
  if (p.D > 256 || p.Dv > 256) return fail(PJX_ERR_UNSUPPORTED, "head dims above 256 are not supported (D=%d, Dv=%d)", p.D, p.Dv);
  if (p.B == 0 || p.Lq == 0 || p.Hq == 0) return PJX_OK;
  switch (dtype) {
    case PJX_F32: return launch_d<float>(p, stream);
    case PJX_BF16: return launch_d<__nv_bfloat16>(p, stream);
    case PJX_F16: return launch_d<__half>(p, stream);
  }
  return fail(PJX_ERR_BAD_ARG, "unknown dtype %d", dtype);
}

}  // namespace pjx
