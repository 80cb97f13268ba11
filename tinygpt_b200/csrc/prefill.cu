// prefill.cu — the small kernels around the tcgen05 GEMM in the batched PREFILL path (S prompt tokens at once):
//   q/k per-head RMSNorm + RoPE + in-place KV-cache write for all S tokens, and causal attention of the chunk against the cache on
//   the CUDA cores (one CTA per query row and head, online softmax over 128-key chunks; B200_PREFILL_ATTN=cuda — the
//   tensor-core kernel is prefill_attn.cu).
//   [ref: src/layer/Attention.h:71-112,156-163; TT/Operation/OpLinalg.cpp:273-275;
//    TT/Operation/OpNNLayerCuda.cuh:252-299,412-440; TFA/mma/kernel.cuh:18-203 (causal prefill)]
// Decode never comes here.
#include "common.cuh"
#include "ops.cuh"

namespace b200 {

namespace {

// y[r, j] = bf16(y[r, j] + b[j]): a bias that cannot ride on the GEMM's store (not 16-byte aligned)
__global__ void __launch_bounds__(256) bias_add_kernel(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ b,
                                                       int64_t rows, int64_t n) {
  const int64_t total = rows * n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = __hadd(y[i], b[i % n]);
}

// q and k heads of the merged qkv rows [S, qdim + 2 kvdim]: optional per-head RMSNorm, RoPE at position p0 + t, q written back in
// place, k and v written to the cache row.  HD / 16 lanes per (token, head): a lane holds 8 neighbouring elements of the
// head's lower half and their 8 rotation partners of the upper half, so every access is a 16-byte vector and the norm's sum
// goes over the head's lanes; a v head is a copy.  A lane takes G heads of its token: their rows are all asked for before the first is worked on.
// EARLY: the token's rotation is read ahead of the wait for the kernel in front, for sixteen registers more.
template <int HD, int G, bool EARLY>
__global__ void __launch_bounds__(256) prefill_qk_kernel(__nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ q_norm,
                                                         const __nv_bfloat16* __restrict__ k_norm, float eps,
                                                         const float* __restrict__ rope, __nv_bfloat16* __restrict__ kcache,
                                                         __nv_bfloat16* __restrict__ vcache, int S, int Hq, int Hkv, int p0) {
  constexpr int L = HD / 16;   // lanes per head
  const int heads = Hq + 2 * Hkv;
  const unsigned groups = (unsigned)(heads + G - 1) / G;
  const unsigned item = (blockIdx.x * blockDim.x + threadIdx.x) / L;
  const int part = threadIdx.x % L;
  const bool live = item < (unsigned)S * groups;
  const int t = live ? (int)(item / groups) : 0, h0 = live ? (int)(item % groups) * G : 0;
  const float* const row = rope + (size_t)(p0 + t) * HD * 2 + part * 16;
  float cs[16];
  auto load_cs = [&]() {
    if ((reinterpret_cast<uintptr_t>(rope) & 15) == 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) reinterpret_cast<float4*>(cs)[e] = reinterpret_cast<const float4*>(row)[e];
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e) cs[e] = row[e];
    }
  };
  if (EARLY && h0 < Hq + Hkv) load_cs();
  pdl_wait();
  pdl_trigger();
  uint4* const src = reinterpret_cast<uint4*>(qkv + ((int64_t)t * heads + h0) * HD);
  uint4 los[G], his[G];
#pragma unroll
  for (int i = 0; i < G; ++i)
    if (h0 + i < heads) {
      los[i] = src[i * 2 * L + part];
      his[i] = src[i * 2 * L + part + L];
    }
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int h = h0 + i;
    if (h >= heads) break;
    uint4 lo = los[i], hi = his[i];
    if (h < Hq + Hkv) {   // uniform among the lanes of a head
      const __nv_bfloat16* nw = h < Hq ? q_norm : k_norm;
      float a[8], b[8];
      unpack8(lo, a);
      unpack8(hi, b);
      if (nw != nullptr) {
        // The sum's order is that of one warp per head, where lane l adds elements l, l + 32, … before a butterfly over the lanes: a lane of
        // the head's lower half gathers what belongs to its eight such lanes from its partner, the butterfly's first steps go
        // over lanes, its last three over the eight sums.
        const unsigned mask = ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
        float s8[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if constexpr (HD == 128) {   // elements i, i + 32, i + 64, i + 96 with i = 8·(part & 3) + e
            const float oa = __shfl_xor_sync(mask, a[e], 4), ob = __shfl_xor_sync(mask, b[e], 4);
            const bool low = part < 4;
            const float x0 = low ? a[e] : oa, x1 = low ? oa : a[e], x2 = low ? b[e] : ob, x3 = low ? ob : b[e];
            s8[e] = __fmaf_rn(x3, x3, __fmaf_rn(x2, x2, __fmaf_rn(x1, x1, __fmul_rn(x0, x0))));
          } else {                     // elements i, i + 32 with i = 8·part + e
            s8[e] = __fmaf_rn(b[e], b[e], __fmul_rn(a[e], a[e]));
          }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) s8[e] += __shfl_xor_sync(mask, s8[e], 2);
#pragma unroll
        for (int e = 0; e < 8; ++e) s8[e] += __shfl_xor_sync(mask, s8[e], 1);
        const float ss = ((s8[0] + s8[4]) + (s8[2] + s8[6])) + ((s8[1] + s8[5]) + (s8[3] + s8[7]));
        const float inv = rsqrtf(ss / (float)HD + eps);
        float wa[8], wb[8];
        if ((reinterpret_cast<uintptr_t>(nw) & 15) == 0) {
          unpack8(reinterpret_cast<const uint4*>(nw)[part], wa);
          unpack8(reinterpret_cast<const uint4*>(nw)[part + L], wb);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            wa[e] = bf16_to_f(nw[part * 8 + e]);
            wb[e] = bf16_to_f(nw[(part + L) * 8 + e]);
          }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          a[e] = round_bf16(a[e] * inv * wa[e]);
          b[e] = round_bf16(b[e] * inv * wb[e]);
        }
      }
      if (!EARLY && i == 0) load_cs();
      float x[8], y[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float c = cs[2 * e], sn = cs[2 * e + 1];   // the roundings of each product are part of the result: spelled out
        x[e] = __fmaf_rn(a[e], c, -__fmul_rn(b[e], sn));
        y[e] = __fmaf_rn(a[e], sn, __fmul_rn(b[e], c));
      }
      lo = make_uint4(pack2(x[0], x[1]), pack2(x[2], x[3]), pack2(x[4], x[5]), pack2(x[6], x[7]));
      hi = make_uint4(pack2(y[0], y[1]), pack2(y[2], y[3]), pack2(y[4], y[5]), pack2(y[6], y[7]));
    }
    if (!live) continue;
    uint4* const dst = h < Hq ? src + i * 2 * L
                              : reinterpret_cast<uint4*>((h < Hq + Hkv ? kcache : vcache) + ((size_t)(p0 + t) * Hkv + (h - Hq) % Hkv) * HD);
    dst[part] = lo;
    dst[part + L] = hi;
  }
}

template <int HD>
struct InvSqrtHdP;
template <>
struct InvSqrtHdP<64> {
  static constexpr float value = 0.125f;
};
template <>
struct InvSqrtHdP<128> {
  static constexpr float value = 0.08838834764831845f;
};

// Causal attention of S query rows (positions p0 … p0+S-1) against cache rows 0 … p0+row: one CTA per (row, head).
template <int HD>
__global__ void __launch_bounds__(128) attn_prefill_kernel(__nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ qkv,
                                                           const __nv_bfloat16* __restrict__ kcache,
                                                           const __nv_bfloat16* __restrict__ vcache, int Hq, int Hkv,
                                                           int p0) {
  constexpr float kScale = InvSqrtHdP<HD>::value * 1.4426950408889634f;
  __shared__ float qs[HD];
  __shared__ float ps[128];
  __shared__ float red[4];
  const int row = blockIdx.x, h = blockIdx.y;
  const int kvh = h / (Hq / Hkv);
  const int tid = threadIdx.x;
  const int qdim = Hq * HD, kvdim = Hkv * HD;
  const __nv_bfloat16* qp = qkv + (size_t)row * (qdim + 2 * kvdim) + h * HD;
  for (int d = tid; d < HD; d += 128) qs[d] = bf16_to_f(qp[d]);
  __syncthreads();
  const int nkeys = p0 + row + 1;
  float m_run = -INFINITY, l_run = 0.f, acc = 0.f;
  for (int c0 = 0; c0 < nkeys; c0 += 128) {
    const int j = c0 + tid;
    float s = -INFINITY;
    if (j < nkeys) {
      const uint4* kp = reinterpret_cast<const uint4*>(kcache + ((size_t)j * Hkv + kvh) * HD);
      float d = 0.f;
#pragma unroll
      for (int piece = 0; piece < HD / 8; ++piece) {
        float qf[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) qf[e] = qs[piece * 8 + e];
        d = dot8(kp[piece], qf, d);
      }
      s = d;
    }
    float cm = warp_max(s);
    if ((tid & 31) == 0) red[tid >> 5] = cm;
    __syncthreads();
    cm = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    __syncthreads();
    const float m_new = fmaxf(m_run, cm);
    const float corr = (m_run == -INFINITY) ? 0.f : exp2f((m_run - m_new) * kScale);
    const float e = (j < nkeys) ? exp2f(s * kScale - m_new * kScale) : 0.f;
    ps[tid] = e;
    float cs = warp_sum(e);
    if ((tid & 31) == 0) red[tid >> 5] = cs;
    __syncthreads();
    cs = red[0] + red[1] + red[2] + red[3];
    l_run = l_run * corr + cs;
    m_run = m_new;
    if (tid < HD) {
      acc *= corr;
      const int n = min(128, nkeys - c0);
      for (int jj = 0; jj < n; ++jj)
        acc = fmaf(ps[jj], bf16_to_f(vcache[((size_t)(c0 + jj) * Hkv + kvh) * HD + tid]), acc);
    }
    __syncthreads();
  }
  if (tid < HD) o[(size_t)row * qdim + h * HD + tid] = f_to_bf16(acc * (l_run > 0.f ? 1.f / l_run : 0.f));
}

}  // namespace

int launch_bias_add(void* y, const void* b, int64_t rows, int64_t n, cudaStream_t st) {
  B200_CHECK_ARG(y && b && rows > 0 && n > 0, "bias_add: bad arguments");
  int64_t g = (rows * n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  g_launches.fetch_add(1);
  bias_add_kernel<<<(unsigned)g, 256, 0, st>>>((__nv_bfloat16*)y, (const __nv_bfloat16*)b, rows, n);
  B200_CUDA(cudaGetLastError());
  return B200_OK;
}

int launch_prefill_qk(void* qkv, const void* q_norm, const void* k_norm, float eps, const float* rope, void* kcache,
                      void* vcache, int S, int Hq, int Hkv, int hd, int p0, cudaStream_t st) {
  B200_CHECK_ARG(hd == 64 || hd == 128, "prefill: head_dim %d not built", hd);
  B200_CHECK_ARG(aligned16(qkv, kcache, vcache), "prefill: rows and caches must be 16-byte aligned");   // the engine's own
  B200_CHECK_ARG((int64_t)S * (Hq + 2 * Hkv) * (hd / 16) < (1ll << 31), "prefill: too many rows at a time");
  // Two heads a lane where heads of 64 fill more than one CTA per SM: prompts of the 0.5B model with one / two, 300 rows 1.59 / 1.59 ms, 700 2.16 / 2.14,
  // 2 048 3.44 / 3.31.  Heads of 128 (1.7B, 60 rows 1.92 / 1.94, 1 200 4.82 / 4.87) and four heads a lane (2 048 rows 3.41) gain nothing.  The rotation
  // ahead of the wait pays while all CTAs are on the chip at once, four of 64 registers on each SM (1.7B behind → ahead: 9 rows 1.864 → 1.842, 300
  // 2.479 → 2.426, but 1 200 4.78 → 4.82); heads of 64 are past that line with two heads a lane, where it pays too.
  const int heads = Hq + 2 * Hkv;
  const int64_t lanes = (int64_t)S * heads * (hd / 16);
  const bool two = hd == 64 && lanes > 148 * 256;
  const unsigned grid = (unsigned)(((two ? (int64_t)S * ((heads + 1) / 2) * (hd / 16) : lanes) + 255) / 256);
  auto* const kernel = hd == 128 ? (grid <= 4 * 148 ? prefill_qk_kernel<128, 1, true> : prefill_qk_kernel<128, 1, false>)
                                 : two ? prefill_qk_kernel<64, 2, true> : prefill_qk_kernel<64, 1, true>;
  B200_CUDA(launch_pdl(kernel, dim3(grid), dim3(256), 0, st, pdl_scope(), (__nv_bfloat16*)qkv, (const __nv_bfloat16*)q_norm,
                       (const __nv_bfloat16*)k_norm, eps, rope, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, S, Hq, Hkv, p0));
  return B200_OK;
}

int launch_attn_prefill(void* o, const void* qkv, const void* kcache, const void* vcache, int S, int Hq, int Hkv, int hd,
                        int p0, cudaStream_t st) {
  B200_CHECK_ARG(hd == 64 || hd == 128, "prefill: head_dim %d not built", hd);
  if (prefill_attn_mma_enabled()) return launch_attn_prefill_mma(o, qkv, kcache, vcache, S, Hq, Hkv, hd, p0, st);
  dim3 grid((unsigned)S, (unsigned)Hq);
  g_launches.fetch_add(1);
  if (hd == 64)
    attn_prefill_kernel<64><<<grid, 128, 0, st>>>((__nv_bfloat16*)o, (const __nv_bfloat16*)qkv,
                                                  (const __nv_bfloat16*)kcache, (const __nv_bfloat16*)vcache, Hq, Hkv, p0);
  else
    attn_prefill_kernel<128><<<grid, 128, 0, st>>>((__nv_bfloat16*)o, (const __nv_bfloat16*)qkv,
                                                   (const __nv_bfloat16*)kcache, (const __nv_bfloat16*)vcache, Hq, Hkv, p0);
  B200_CUDA(cudaGetLastError());
  return B200_OK;
}

}  // namespace b200
