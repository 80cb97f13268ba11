// attn.cu — decode attention for sm_100a: one launch per layer does what the reference does with
//   split (3 memcpy) + [Qwen3 q/k RMSNorm ×2] + RoPE ×2 + KV concat (4 memcpy, O(ctx) re-copy) + TinyFA flash-attn
//   [ref: src/layer/Attention.h:71-112,156-163; src/engine/CacheManager.h:24-42;
//    TT/Operation/OpNNLayerCuda.cuh:252-299 (norm), :412-440 (rope);
//    TFA/mma/kernel.cuh:18-203, TFA/mma/softmax.cuh:67-131 (online softmax, base-2 exponent)]
//
// Why not the reference's shape: TinyFA launches one CTA per Q head with a 128-row Q tile of which one row is live
// and re-reads K/V once per Q head.  Here a CTA owns (KV head, KV split): the G = Hq/Hkv query heads that share the
// KV head are processed together so K/V are read once, the context is split across `nsplit` CTAs so the whole GPU
// works on one token, and the last CTA of a KV head (atomic ticket) merges the split partials — no second launch.
// The KV cache is a pre-allocated [max_ctx, Hkv, hd] buffer written in place at position *pos.
//
// Numerics: q·k and P·V accumulate in fp32 over bf16 inputs; rounding points of q/k (after norm, after RoPE) are the
// reference's.  Probabilities stay fp32 (the reference rounds P to bf16 before P·V, TFA/mma/layout.cuh:88-97); the
// oracle models the reference's rounding and the parity tests bound the difference.
#include "gemv.cuh"
#include "key_range.cuh"
#include "ops.cuh"
#include "tc.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kAttnThreads = 256;
constexpr int kAttnWarps = 8;
constexpr float kLog2e = 1.4426950408889634f;

template <int HD>
struct InvSqrtHd;
template <>
struct InvSqrtHd<64> {
  static constexpr float value = 0.125f;
};
template <>
struct InvSqrtHd<128> {
  static constexpr float value = 0.08838834764831845f;
};


// keys per split: fixed by the shared-memory staging buffers (K and V of one split = 64 KB for both head dims)
template <int HD>
struct SplitKeys {
  static constexpr int value = (HD == 64) ? 256 : 128;
};

// ------------------------------------------------------------------------------------------------- decode kernel
// CTA = (KV split, group of G query heads that share one KV head).  A first version staged K/V of the split in shared memory
// (cp.async) and ran scores / softmax / P·V as three barrier-separated phases: 2.0 µs per launch at ctx ≈ 80 for 69 KB
// of traffic (in-kernel stamps: q/k/v staging 0.54, scores 0.54, softmax 0.64, P·V 0.3).  This kernel keeps everything
// a thread needs in registers (measured against the staged kernel on B200: 409 vs 415 µs per Qwen2.5-0.5B token,
// 1 425 vs 1 445 µs for Llama-3.2-3B, 1 106 vs 1 131 µs at ctx 2 048 for Qwen3-1.7B):
//   * thread = (key group, 16-byte piece): the K and V pieces of up to 8 cached rows per thread are loaded into
//     REGISTERS before griddepcontrol.wait (the rows were written by earlier tokens), no shared-memory staging;
//   * after the wait: q/k RMSNorm + RoPE by one warp per head as before, ONE barrier, then every thread runs an online
//     softmax over its own ≤ 8 keys (scores never leave registers), the key groups of a warp merge by xor-shuffle, the
//     8 warps through 5 KB of shared memory: two more barriers per query head, none for scores / softmax / P·V.
// The new K/V row is written in place to the cache and handed to the owning thread through shared memory.
template <int HD>
__global__ void __launch_bounds__(kAttnThreads) attn_decode_reg_kernel(const AttnDecodeParams p_in, const int G) {
  constexpr int LPK = HD / 8;             // lanes per key row
  constexpr int NG = kAttnThreads / LPK;  // key rows per pass
  constexpr int KPT = 8;                  // key rows per thread
  constexpr int CHUNK = NG * KPT;         // = SplitKeys<HD>: 256 (hd 64) / 128 (hd 128)
  static_assert(CHUNK == SplitKeys<HD>::value, "split size is shared with the host-side nsplit");
  constexpr int EPL = HD / 32;
  constexpr float kScale = InvSqrtHd<HD>::value * kLog2e;
  __shared__ float q_s[8 * HD];
  __shared__ __align__(16) __nv_bfloat16 knew[HD];
  __shared__ __align__(16) __nv_bfloat16 vnew[HD];
  __shared__ float ared[kAttnWarps * 16 * 10];
  __shared__ int is_last;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hg = blockIdx.y, split = blockIdx.x;
  AttnDecodeParams p = p_in;
  {  // batched decode: this CTA's sequence
    const long long b = blockIdx.z;
    p.qkv += b * p.qkv_bstride;
    p.out += b * p.out_bstride;
    p.kcache += b * p.cache_bstride;
    p.vcache += b * p.cache_bstride;
    p.ws += b * p.ws_bstride;
    p.tickets += b * p.tick_bstride;
  }
  const int h0 = hg * G;
  const int group = p.Hq / p.Hkv;
  const int kvh = h0 / group;
  const bool kv_leader = (h0 % group) == 0;
  if (p.trace != nullptr && hg == 0 && split == 0 && blockIdx.z == 0 && tid == 0) p.trace[0] = global_timer_ns();
  pdl_trigger();
  const bool append = (p.pos != nullptr);
  const int pos = append ? *p.pos : p.fixed_len - 1;   // stable since before the producer kernel started (engine.cu)
  const int L = pos + 1;
  const int nact = (L + CHUNK - 1) / CHUNK;
  if (split >= nact) {
    pdl_wait();
    return;
  }
  const int start = split * CHUNK;
  const int end = min(L, start + CHUNK);
  const int n_old_end = append ? min(end, pos) : end;    // rows [start, n_old_end) are already in the cache
  const bool owns_new = append && pos >= start && pos < end;
  const int grp = tid / LPK, part = tid % LPK;
  const int imax = (end - start + NG - 1) / NG;   // key slots per thread that this split can fill (CTA-uniform)

  uint4 kreg[KPT], vreg[KPT];
#pragma unroll
  for (int i = 0; i < KPT; ++i) {
    const int row = start + grp + NG * i;
    kreg[i] = make_uint4(0, 0, 0, 0);
    vreg[i] = make_uint4(0, 0, 0, 0);
    if (i < imax && row < n_old_end) {
      const size_t g = ((size_t)row * p.Hkv + kvh) * HD + part * 8;
      kreg[i] = *reinterpret_cast<const uint4*>(p.kcache + g);
      vreg[i] = *reinterpret_cast<const uint4*>(p.vcache + g);
    }
  }
  float rc[EPL / 2], rs[EPL / 2];
  if (p.rope != nullptr) {
    const float* row = p.rope + (size_t)pos * HD * 2;
#pragma unroll
    for (int j = 0; j < EPL / 2; ++j) {
      rc[j] = row[(lane + 32 * j) * 2];
      rs[j] = row[(lane + 32 * j) * 2 + 1];
    }
  }
  pdl_wait();   // qkv of this token is complete and visible from here on
  if (p.trace != nullptr && hg == 0 && split == 0 && tid == 0) p.trace[1] = global_timer_ns();
  const int qdim = p.Hq * HD, kvdim = p.Hkv * HD;
  for (int h = warp; h < G + 1; h += kAttnWarps) {
    const bool is_k = (h == G);
    if (is_k && !owns_new) break;
    const __nv_bfloat16* src = is_k ? p.qkv + qdim + kvh * HD : p.qkv + (h0 + h) * HD;
    const __nv_bfloat16* nw = is_k ? p.k_norm : p.q_norm;
    float x[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) x[j] = bf16_to_f(src[lane + 32 * j]);
    if (nw != nullptr) {
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < EPL; ++j) ss += x[j] * x[j];
      ss = warp_sum(ss);
      const float inv = rsqrtf(ss / (float)HD + p.eps);
#pragma unroll
      for (int j = 0; j < EPL; ++j) x[j] = round_bf16(x[j] * inv * bf16_to_f(nw[lane + 32 * j]));
    }
    if (p.rope != nullptr) {
#pragma unroll
      for (int j = 0; j < EPL / 2; ++j) {
        const float x1 = x[j], x2 = x[j + EPL / 2];
        x[j] = round_bf16(x1 * rc[j] - x2 * rs[j]);
        x[j + EPL / 2] = round_bf16(x2 * rc[j] + x1 * rs[j]);
      }
    }
    if (is_k) {
      __nv_bfloat16* kg = p.kcache + ((size_t)pos * p.Hkv + kvh) * HD;
      __nv_bfloat16* vg = p.vcache + ((size_t)pos * p.Hkv + kvh) * HD;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const __nv_bfloat16 kk = f_to_bf16(x[j]);
        const __nv_bfloat16 vv = p.qkv[qdim + kvdim + kvh * HD + lane + 32 * j];
        knew[lane + 32 * j] = kk;
        vnew[lane + 32 * j] = vv;
        if (kv_leader) {
          kg[lane + 32 * j] = kk;
          vg[lane + 32 * j] = vv;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < EPL; ++j) q_s[h * HD + lane + 32 * j] = x[j];
    }
  }
  __syncthreads();
  if (p.trace != nullptr && hg == 0 && split == 0 && tid == 0) p.trace[3] = global_timer_ns();
  if (owns_new) {
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      if (start + grp + NG * i == pos) {
        kreg[i] = reinterpret_cast<const uint4*>(knew)[part];
        vreg[i] = reinterpret_cast<const uint4*>(vnew)[part];
      }
    }
  }
  for (int g = 0; g < G; ++g) {
    float qf[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) qf[e] = q_s[g * HD + part * 8 + e];
    float sc[KPT];
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      sc[i] = -INFINITY;
      if (i < imax) {   // uniform: unused slots cost one branch
        float d = dot8(kreg[i], qf, 0.f);
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if ((start + grp + NG * i) < end) sc[i] = d;
        m = fmaxf(m, sc[i]);
      }
    }
    float l = 0.f, acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    const float m_scaled = m * kScale;
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      if (i < imax) {
        const float pr = (sc[i] == -INFINITY) ? 0.f : exp2f(sc[i] * kScale - m_scaled);
        l += pr;
        float vf[8];
        unpack8(vreg[i], vf);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(pr, vf[e], acc[e]);
      }
    }
#pragma unroll
    for (int o = LPK; o < 32; o <<= 1) {   // key groups that live in the same warp
      const float mo = __shfl_xor_sync(0xffffffffu, m, o);
      const float lo = __shfl_xor_sync(0xffffffffu, l, o);
      const float mn = fmaxf(m, mo);
      const float a = (m == -INFINITY) ? 0.f : exp2f((m - mn) * kScale);
      const float b = (mo == -INFINITY) ? 0.f : exp2f((mo - mn) * kScale);
      l = l * a + lo * b;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float ao = __shfl_xor_sync(0xffffffffu, acc[e], o);
        acc[e] = acc[e] * a + ao * b;
      }
      m = mn;
    }
    if (lane < LPK) {
      float* r = ared + (warp * 16 + lane) * 10;
      r[0] = m;
      r[1] = l;
#pragma unroll
      for (int e = 0; e < 8; ++e) r[2 + e] = acc[e];
    }
    __syncthreads();
    if (tid < HD) {
      const int d = tid, pt = d >> 3, e = d & 7;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < kAttnWarps; ++w) M = fmaxf(M, ared[(w * 16 + pt) * 10]);
      float num = 0.f, den = 0.f;
#pragma unroll
      for (int w = 0; w < kAttnWarps; ++w) {
        const float* r = ared + (w * 16 + pt) * 10;
        const float wgt = (r[0] == -INFINITY) ? 0.f : exp2f((r[0] - M) * kScale);
        num = fmaf(wgt, r[2 + e], num);
        den = fmaf(wgt, r[1], den);
      }
      if (nact == 1) {
        p.out[(h0 + g) * HD + d] = f_to_bf16(num * (den > 0.f ? 1.f / den : 0.f));
      } else {
        float* wsr = p.ws + ((size_t)(h0 + g) * p.nsplit + split) * (HD + 2);
        wsr[d] = num;
        if (d == 0) {
          wsr[HD] = M;
          wsr[HD + 1] = den;
        }
      }
    }
    __syncthreads();
  }
  if (p.trace != nullptr && hg == 0 && split == 0 && tid == 0) p.trace[2] = global_timer_ns();
  if (nact == 1) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned int t = atomicAdd(&p.tickets[hg], 1u);
    is_last = (t == (unsigned int)nact - 1) ? 1 : 0;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  for (int idx = tid; idx < G * HD; idx += kAttnThreads) {
    const int g = idx / HD, d = idx % HD;
    const float* base = p.ws + (size_t)(h0 + g) * p.nsplit * (HD + 2);
    float M = -INFINITY;
    for (int s = 0; s < nact; ++s) M = fmaxf(M, __ldcg(base + (size_t)s * (HD + 2) + HD));
    float num = 0.f, den = 0.f;
    for (int s = 0; s < nact; ++s) {
      const float* r = base + (size_t)s * (HD + 2);
      const float w = exp2f((__ldcg(r + HD) - M) * kScale);
      num = fmaf(w, __ldcg(r + d), num);
      den = fmaf(w, __ldcg(r + HD + 1), den);
    }
    p.out[(h0 + g) * HD + d] = f_to_bf16(num * (den > 0.f ? 1.f / den : 0.f));
  }
  if (tid == 0) p.tickets[hg] = 0;
}

// ------------------------------------------------------------------------------- one query row over many keys
// One new row against every key, probabilities in fp32, as (a) o = softmax(q·kᵀ)·v for Sq = 1 through the operator boundary and (b) the fused decode
// attention over long contexts (q/k norm, rotation and the in-place append as in attn_decode_reg_kernel).
// A cluster shares a (sequence, group of up to eight query heads of one KV head): its CTAs take neighbouring ranges of the keys, so that a key
// and a value are read once for all of the group's heads.  A CTA walks its range in units of 128 keys, sixteen a warp; the K and V rows come
// through a ring in shared memory (cp.async, 96 KB, all of it asked for at once and, for cached rows, before the kernel in front has ended).
// Inside its sixteen keys a warp works alone, without a barrier:
//   scores  K·qᵀ on mma.sync, the heads as its eight columns: exact products of bf16, summed in fp32
//   softmax online, from the score fragments
//   P·V     fp32 multiply-adds, a lane four columns, the probabilities broadcast from shared memory
// The warps merge through shared memory, and every CTA sends each of the others its share of the result through distributed shared memory:
// one cluster barrier, no workspace, no tickets, one launch.  Bound by launch, one round trip of loads and the merge.
//
// Against eight CTAs per one or two heads, which read K and V once per head in eight dependent rounds of register loads: device µs, rotating caches of 4 096
// tokens, positions 100 / 1 000 / 2 000 / 4 000: 16 / 8 heads of 128 5.1 / 6.6 / 8.7 / 12.2 → 5.4 / 5.8 / 6.7 / 9.9, 24 / 8 heads 5.3 / 6.8 / 9.2 / 13.0 →
// 5.8 / 6.0 / 7.3 / 10.9, 14 / 2 heads of 64 4.6 / 5.3 / 5.9 / 7.2 → 5.2 / 5.2 / 5.6 / 6.9.  Inside a token the loads run beside the
// kernel in front: µs a token at positions 100 / 1 000 / 3 900, caches for 4 096, 28 layers, 2 048 wide 804 / 869 / 1 035 → 826 / 834 / 913, 24 layers, 896 wide
// 452 / 461 / 509 → 432 / 437 / 465.  Eight CTAs at most instead of sixteen: 0.3 µs less at short positions, 0.7 … 2 more at long ones, and long
// tokens behind (4 000: 1 021).  Barriers over the whole CTA in every unit: 6.9 µs at position 100.
struct AttnRow {
  AttnDecodeParams d;               // decode: everything; row: qkv = q [B, Hq, HD], out, kcache / vcache and the strides
  int nkeys;                        // row: keys to see (decode reads the position)
  long long kv_bstride;             // elements from one batch element's keys to the next
  int G, per_kv;                    // query heads of a CTA; CTAs (clusters) per KV head
  int log_splits;
};
constexpr int kUnit = 128, kMaxSplits = 16;
template <int HD>
struct KeyRing {
  static constexpr int RB = HD * 2, SLOT = kUnit * RB, NS = HD == 128 ? 3 : 6;   // bytes of a row and of a unit's K or V; slots
  static constexpr int smem = NS * SLOT;
};
template <bool DECODE>
__device__ __forceinline__ void row_stamp(const AttnDecodeParams& p, int i) {   // nothing that has to stay in a register
  if (DECODE && p.trace != nullptr && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) p.trace[i] = global_timer_ns();
}
template <int HD, int GM, bool DECODE>
__global__ void __launch_bounds__(kAttnThreads, 2) attn_row_kernel(const AttnRow a) {
  using R = KeyRing<HD>;
  constexpr int LQ = HD / 4;   // column quads
  constexpr int EPL = HD / 32, QP = HD + 8;
  constexpr float kScale = InvSqrtHd<HD>::value * kLog2e;
  static_assert(kAttnWarps * GM * HD * 4 <= R::smem, "the warps' sums fit where the keys were");
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ __align__(16) __nv_bfloat16 q_s[8][QP];
  __shared__ __align__(16) __nv_bfloat16 knew[HD];
  __shared__ __align__(16) __nv_bfloat16 vnew[HD];
  __shared__ __align__(16) float ps[kUnit][GM];
  __shared__ __align__(16) float2 w_ml[kAttnWarps][8];
  __shared__ __align__(16) float4 part[GM * LQ + kMaxSplits];   // [CTA][its share of this CTA's columns]
  __shared__ __align__(16) float2 part_ml[kMaxSplits][GM];
  const AttnDecodeParams& p = a.d;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3, G = a.G;
  const int h0 = blockIdx.y * G, kvh = a.per_kv == 1 ? blockIdx.y : blockIdx.y / a.per_kv;
  const long long b = blockIdx.z;
  const int rank = (int)cluster_rank(), splits = 1 << a.log_splits;
  row_stamp<DECODE>(p, 0);
  pdl_trigger();
  if (!DECODE || p.late) pdl_wait();
  cluster_arrive_relaxed();                // this CTA runs: the others may write to it once they have waited for that
  const bool append = DECODE && p.pos != nullptr;
  int pos = append ? *p.pos : p.fixed_len - 1;   // where q is rotated; stable since before the producer kernel started
  if (append && (unsigned)pos >= (unsigned)p.max_ctx) pos = -1;   // outside the caches: no keys, and none of the ranges has the new one
  const int cached = append ? pos : DECODE ? p.fixed_len : a.nkeys;   // rows that are in the cache already
  const KeyRange keys = key_range(cached, append, rank, a.log_splits);
  const int k0 = keys.first, n = keys.n, n_cached = keys.n_cached;   // this CTA's keys
  const int units = (n - warp * 16 + kUnit - 1) / kUnit;   // with a key for this warp
  constexpr int PC = HD / 8, RP = 32 / PC;   // 16-byte pieces of a row; rows that a warp copies at once
  constexpr uint32_t WB = 16 * R::RB;        // a warp's part of a slot
  const int c0 = lane % PC, r0 = lane / PC;
  const int64_t ks = (int64_t)p.Hkv * HD, first = (int64_t)b * a.kv_bstride + kvh * HD + (k0 + warp * 16 + r0) * ks + c0 * 8;
  const __nv_bfloat16 *k_src = p.kcache + first, *v_src = p.vcache + first;
  const uint32_t ring_u = smem_u32(ring) + warp * WB;
  // place of 16-byte piece c of row r: pieces of eight rows change places, so that both ways of reading spread over the banks
  auto piece_at = [&](int r, int c) { return (uint32_t)(r * R::RB + ((c ^ (r & 7)) << 4)); };
  auto load = [&](int s) {   // K (even) or V (odd) of this warp's keys of unit s / 2, zeros behind the last; always one commit group
    const int rows = n_cached - (s >> 1) * kUnit - warp * 16 - r0;
    if (rows + r0 > 0) {
      const __nv_bfloat16* src = ((s & 1) ? v_src : k_src) + (int64_t)(s >> 1) * kUnit * ks;
      const uint32_t dst = ring_u + (uint32_t)(s % R::NS) * R::SLOT;
#pragma unroll
      for (int r = 0; r < 16; r += RP)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     ::"r"(dst + piece_at(r + r0, c0)), "l"(r < rows ? src + r * ks : p.kcache), "r"(r < rows ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float q_in[DECODE ? 1 : GM * HD / kAttnThreads + 1];
  if constexpr (!DECODE) {
#pragma unroll
    for (int i = 0; i < GM * HD / kAttnThreads + 1; ++i) {
      const int e = i * kAttnThreads + tid;
      q_in[i] = e < G * HD ? bf16_to_f(p.qkv[b * p.qkv_bstride + h0 * HD + e]) : 0.f;
    }
  }
#pragma unroll
  for (int s = 0; s < R::NS; ++s) load(s);   // rows of earlier tokens: nothing that the producer kernel writes
  [[maybe_unused]] const __nv_bfloat16* qkv = p.qkv + b * p.qkv_bstride;
  const bool owns_new = keys.owns_new;
  for (int i = G * (QP / 2) + tid; i < 8 * (QP / 2); i += kAttnThreads) reinterpret_cast<uint32_t*>(&q_s[0][0])[i] = 0;   // columns without a head
  if constexpr (DECODE) {
    float rc[EPL / 2], rs[EPL / 2];
    if (p.rope != nullptr) {
      const float* row = p.rope + (size_t)max(pos, 0) * HD * 2;
#pragma unroll
      for (int j = 0; j < EPL / 2; ++j) {
        rc[j] = row[(lane + 32 * j) * 2];
        rs[j] = row[(lane + 32 * j) * 2 + 1];
      }
    }
    pdl_wait();                            // qkv of this token is complete and visible from here on
    row_stamp<DECODE>(p, 1);
    const int qdim = p.Hq * HD, kvdim = p.Hkv * HD;
    for (int h = warp; h < G + 1; h += kAttnWarps) {
      const bool is_k = h == G;
      if (is_k && !owns_new) break;
      const __nv_bfloat16* src = is_k ? qkv + qdim + kvh * HD : qkv + (h0 + h) * HD;
      const __nv_bfloat16* nw = is_k ? p.k_norm : p.q_norm;
      float x[EPL];
#pragma unroll
      for (int j = 0; j < EPL; ++j) x[j] = bf16_to_f(src[lane + 32 * j]);
      if (nw != nullptr) {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) ss += x[j] * x[j];
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss / (float)HD + p.eps);
#pragma unroll
        for (int j = 0; j < EPL; ++j) x[j] = round_bf16(x[j] * inv * bf16_to_f(nw[lane + 32 * j]));
      }
      if (p.rope != nullptr) {
#pragma unroll
        for (int j = 0; j < EPL / 2; ++j) {
          const float x1 = x[j], x2 = x[j + EPL / 2];
          x[j] = round_bf16(x1 * rc[j] - x2 * rs[j]);
          x[j + EPL / 2] = round_bf16(x2 * rc[j] + x1 * rs[j]);
        }
      }
      if (is_k) {
        const size_t at = (size_t)(b * a.kv_bstride) + ((size_t)pos * p.Hkv + kvh) * HD;
        const bool leader = (int)blockIdx.y == kvh * a.per_kv;   // one CTA writes the new cache row
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          const __nv_bfloat16 kk = f_to_bf16(x[j]), vv = qkv[qdim + kvdim + kvh * HD + lane + 32 * j];
          knew[lane + 32 * j] = kk;
          vnew[lane + 32 * j] = vv;
          if (leader) {
            p.kcache[at + lane + 32 * j] = kk;
            p.vcache[at + lane + 32 * j] = vv;
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < EPL; ++j) q_s[h][lane + 32 * j] = f_to_bf16(x[j]);   // rounded before: exact
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < GM * HD / kAttnThreads + 1; ++i) {
      const int e = i * kAttnThreads + tid;
      if (e < G * HD) q_s[e / HD][e % HD] = f_to_bf16(q_in[i]);
    }
  }
  __syncthreads();
  row_stamp<DECODE>(p, 3);
  uint32_t qb[HD / 16][2];   // q as the B operand: column g = head, rows of two neighbouring channels
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk) {
    qb[kk][0] = *reinterpret_cast<const uint32_t*>(&q_s[g][kk * 16 + tq * 2]);
    qb[kk][1] = *reinterpret_cast<const uint32_t*>(&q_s[g][kk * 16 + tq * 2 + 8]);
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};   // of heads 2·tq and 2·tq + 1; l: this lane's keys
  const int dq = lane % LQ, kg = lane / LQ;                 // P·V: this lane's columns, and (heads of 64) its half of the keys
  float acc[GM][4];
#pragma unroll
  for (int h = 0; h < GM; ++h)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[h][e] = 0.f;
  float(*const pw)[GM] = ps + warp * 16;
  for (int u = 0; u < units; ++u) {
    const int nv = min(16, n - u * kUnit - warp * 16);
    const bool has_new = owns_new && u * kUnit + warp * 16 + nv == n;
    const uint32_t kslot = (uint32_t)(2 * u % R::NS) * R::SLOT, vslot = (uint32_t)((2 * u + 1) % R::NS) * R::SLOT;
    auto put_new = [&](uint32_t slot, const __nv_bfloat16* row) {
      __syncwarp();   // a lane has waited for its own copies only: the zeros of this row are another's at most places
      if (nv == 1 && n_cached == n - 1 && u * kUnit + warp * 16 == n_cached) {   // a warp without a cached key has not cleared its rows
        for (int e = lane; e < (int)WB / 16; e += 32) reinterpret_cast<uint4*>(ring + warp * WB + slot)[e] = make_uint4(0, 0, 0, 0);
        __syncwarp();
      }
      if (lane < HD / 8) *reinterpret_cast<uint4*>(ring + warp * WB + slot + piece_at(nv - 1, lane)) = reinterpret_cast<const uint4*>(row)[lane];
    };
    asm volatile("cp.async.wait_group %0;" ::"n"(R::NS - 1) : "memory");
    if (has_new) put_new(kslot, knew);
    __syncwarp();
    float c[2][4] = {};   // keys g and g + 8 of the warp's sixteen, heads 2·tq and 2·tq + 1; two chains
#pragma unroll
    for (int kk = 0; kk < HD / 16; ++kk) {
      uint32_t ka[4];
      float(&d)[4] = c[kk & 1];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(ka[0]), "=r"(ka[1]), "=r"(ka[2]), "=r"(ka[3]) : "r"(ring_u + kslot + piece_at(lane & 15, 2 * kk + (lane >> 4))) : "memory");
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                   : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                   : "r"(ka[0]), "r"(ka[1]), "r"(ka[2]), "r"(ka[3]), "r"(qb[kk][0]), "r"(qb[kk][1]));
    }
    __syncwarp();   // every lane's rows of K have been read
    load(2 * u + R::NS);
    float pr[4], alpha[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float s0 = g < nv ? c[0][e] + c[1][e] : -INFINITY, s1 = g + 8 < nv ? c[0][2 + e] + c[1][2 + e] : -INFINITY;
      float t = fmaxf(s0, s1);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
      t = fmaxf(t, m[e]);
      const float ts = t == -INFINITY ? 0.f : t * kScale;
      alpha[e] = u == 0 || m[e] == -INFINITY ? 0.f : exp2f(m[e] * kScale - ts);
      m[e] = t;
      pr[e] = g < nv ? exp2f(s0 * kScale - ts) : 0.f;
      pr[2 + e] = g + 8 < nv ? exp2f(s1 * kScale - ts) : 0.f;
      l[e] = l[e] * alpha[e] + (pr[e] + pr[2 + e]);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (2 * tq + e < GM) {
        pw[g][2 * tq + e] = pr[e];
        pw[g + 8][2 * tq + e] = pr[2 + e];
      }
    if (u > 0) {
#pragma unroll
      for (int h = 0; h < GM; ++h) {
        const float f = __shfl_sync(0xffffffffu, alpha[h & 1], h >> 1);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[h][e] *= f;
      }
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(R::NS - 1) : "memory");
    if (has_new) put_new(vslot, vnew);
    __syncwarp();
    const uint8_t* const vt = ring + warp * WB + vslot + (dq & 1) * 8;
#pragma unroll 4
    for (int k = kg; k < 16; k += 32 / LQ) {   // keys behind the last: a weight of 0 and rows of zeros
      const uint2 w = *reinterpret_cast<const uint2*>(vt + piece_at(k, dq >> 1));
      const float v[4] = {__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u)};
      float pk[GM];
      if constexpr (GM >= 4) {
#pragma unroll
        for (int h = 0; h < GM; h += 4) *reinterpret_cast<float4*>(&pk[h]) = *reinterpret_cast<const float4*>(&pw[k][h]);
      } else {
#pragma unroll
        for (int h = 0; h < GM; ++h) pk[h] = pw[k][h];
      }
#pragma unroll
      for (int h = 0; h < GM; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[h][e] = fmaf(pk[h], v[e], acc[h][e]);
    }
    __syncwarp();
    load(2 * u + 1 + R::NS);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");   // only empty groups are left
#pragma unroll
  for (int e = 0; e < 2; ++e)
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l[e] += __shfl_xor_sync(0xffffffffu, l[e], o);
  if (g == 0) {
    w_ml[warp][2 * tq] = make_float2(m[0], l[0]);
    w_ml[warp][2 * tq + 1] = make_float2(m[1], l[1]);
  }
  __syncthreads();                                     // every warp's keys are read: the ring takes the sums
  float4* const sums = reinterpret_cast<float4*>(ring);   // [warp][GM][LQ]
#pragma unroll
  for (int h = 0; h < GM; ++h) {
    if constexpr (LQ == 16) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[h][e] += __shfl_xor_sync(0xffffffffu, acc[h][e], 16);
    }
    if (kg == 0) sums[(warp * GM + h) * LQ + dq] = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
  }
  __syncthreads();
  cluster_wait();                                      // every CTA runs
  const int share = (G * LQ + splits - 1) / splits;    // column quads that a CTA finishes
  for (int i = tid; i < G * LQ; i += kAttnThreads) {
    const int h = i / LQ, to = i / share;
    float2 ml[kAttnWarps];
    float4 x[kAttnWarps];
    float top = -INFINITY, den = 0.f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      ml[w] = w_ml[w][h];
      x[w] = sums[(w * GM + h) * LQ + i % LQ];
      top = fmaxf(top, ml[w].x);
    }
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float f = ml[w].x == -INFINITY ? 0.f : exp2f((ml[w].x - top) * kScale);
      den = fmaf(f, ml[w].y, den);
      t.x = fmaf(f, x[w].x, t.x);
      t.y = fmaf(f, x[w].y, t.y);
      t.z = fmaf(f, x[w].z, t.z);
      t.w = fmaf(f, x[w].w, t.w);
    }
    st_cluster_f4(mapa_u32(smem_u32(&part[rank * share + i - to * share]), to), t);
    // with the first of this head's columns that go there, the maximum and the sum
    if (i == max(h * LQ, to * share)) st_cluster_f2(mapa_u32(smem_u32(&part_ml[rank][h]), to), make_float2(top, den));
  }
  cluster_sync_all();                                  // every CTA's parts are in place
  const int r = tid & (splits - 1), j = tid >> a.log_splits, i = rank * share + j;   // a lane per CTA and four neighbouring outputs
  const bool live = j < share && i < G * LQ;
  const unsigned mask = __ballot_sync(0xffffffffu, live);   // the lanes that sum below: all of a CTA's parts of an output, or none
  if (live) {
    const float2 ml = part_ml[r][i / LQ];
    const float4 x = part[r * share + j];
    float top = ml.x;
    for (int o = splits >> 1; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(mask, top, o));
    const float f = ml.x == -INFINITY ? 0.f : exp2f((ml.x - top) * kScale);
    float den = f * ml.y, num[4] = {f * x.x, f * x.y, f * x.z, f * x.w};
    for (int o = splits >> 1; o > 0; o >>= 1) {
      den += __shfl_xor_sync(mask, den, o);
#pragma unroll
      for (int e = 0; e < 4; ++e) num[e] += __shfl_xor_sync(mask, num[e], o);
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
    __nv_bfloat16* o = p.out + b * p.out_bstride + h0 * HD + i * 4;
    if (r == 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = f_to_bf16(num[e] * inv);
    }
  }
  row_stamp<DECODE>(p, 2);
}

// ------------------------------------------------------------------------------------------ general attention
// One CTA per (q row, head, batch); keys in chunks of 128 with online softmax.  For what the other kernels do not take: several
// query rows that are not a causal prompt, and tensors off a 16-byte boundary (k_wide = 0: keys read two bytes at a time).
template <int HD>
__global__ void __launch_bounds__(128) attn_general_kernel(__nv_bfloat16* __restrict__ o,
                                                           const __nv_bfloat16* __restrict__ q,
                                                           const __nv_bfloat16* __restrict__ k,
                                                           const __nv_bfloat16* __restrict__ v, int Sq, int Skv, int Hq,
                                                           int Hkv, int causal, int k_wide) {
  constexpr float kScale = InvSqrtHd<HD>::value * kLog2e;
  __shared__ float qs[HD];
  __shared__ float ps[128];
  __shared__ float red[4];
  const int row = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int kvh = h / (Hq / Hkv);
  const int tid = threadIdx.x;
  const __nv_bfloat16* qp = q + (((size_t)b * Sq + row) * Hq + h) * HD;
  for (int d = tid; d < HD; d += 128) qs[d] = bf16_to_f(qp[d]);
  __syncthreads();
  const int nkeys = causal ? min(Skv, row + 1) : Skv;
  float m_run = -INFINITY, l_run = 0.f, acc = 0.f;  // thread d < HD owns output column d
  for (int c0 = 0; c0 < nkeys; c0 += 128) {
    const int j = c0 + tid;
    float s = -INFINITY;
    if (j < nkeys) {
      const __nv_bfloat16* kp = k + (((size_t)b * Skv + j) * Hkv + kvh) * HD;
      float d = 0.f;
#pragma unroll
      for (int piece = 0; piece < HD / 8; ++piece) {
        float qf[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) qf[e] = qs[piece * 8 + e];
        uint4 kv;
        if (k_wide) {
          kv = reinterpret_cast<const uint4*>(kp)[piece];
        } else {
          const unsigned short* e = reinterpret_cast<const unsigned short*>(kp) + piece * 8;
          kv = make_uint4(e[0] | (uint32_t)e[1] << 16, e[2] | (uint32_t)e[3] << 16, e[4] | (uint32_t)e[5] << 16, e[6] | (uint32_t)e[7] << 16);
        }
        d = dot8(kv, qf, d);
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
        acc = fmaf(ps[jj], bf16_to_f(v[(((size_t)b * Skv + c0 + jj) * Hkv + kvh) * HD + tid]), acc);
    }
    __syncthreads();
  }
  if (tid < HD) o[(((size_t)b * Sq + row) * Hq + h) * HD + tid] = f_to_bf16(acc * (l_run > 0.f ? 1.f / l_run : 0.f));
}

}  // namespace

// Caches from which the cluster kernel takes over: more splits than this (1 024 tokens for heads of 128, 2 048 for heads of 64).  The choice is
// by the cache, since a captured graph serves every position.  Device µs with caches for 4 096 tokens, one CTA per
// split / cluster, at positions 20, 300, 2 000 and 4 000: 16 heads of 128 5.9 / 5.5, 9.3 / 5.6, 11.4 / 6.7, 21.5 / 9.9; 32 heads of
// 128 7.8 / 5.9, 13.8 / 5.9, 17.4 / 7.3, 33.2 / 10.9; 14 heads of 64 9.5 / 5.1, 17.4 / 5.2, 17.7 / 5.6, 21.1 / 6.9.
constexpr int kLongSplits = 8;

int64_t attn_decode_ws_floats(int Hq, int Hkv, int hd, int nsplit) {
  (void)Hkv;
  if (nsplit > kLongSplits) return 0;      // the cluster kernel keeps its partials in shared memory
  return (int64_t)Hq * nsplit * (hd + 2);  // same size whatever the head grouping
}

// Query heads per CTA: the whole GQA group once the context is long enough for K/V re-reads to matter, else one.
// The kernel takes any G ≤ 8 that divides the GQA group (the reference accepts every Hq % Hkv == 0): the largest such
// divisor (6 → 6, 5 → 5, 16 → 8, 12 → 6).
int attn_heads_per_cta(int Hq, int Hkv, int max_ctx) {
  if (max_ctx <= 1024) return 1;
  const int group = Hq / Hkv;
  for (int g = 8; g > 1; --g)
    if (group % g == 0) return g;
  return 1;
}

int attn_setup_attributes() { return B200_OK; }   // attn_decode_reg_kernel has static shared memory only; launch_row_t sets attn_row_kernel's

int attn_decode_nsplit(int hd, int max_ctx) {
  const int chunk = (hd == 64) ? SplitKeys<64>::value : SplitKeys<128>::value;
  return std::max(1, (max_ctx + chunk - 1) / chunk);
}

template <int HD, int GM, bool DECODE>
static int launch_row_t(const AttnRow& a, int splits, int B, cudaStream_t st, bool pdl) {
  static PerDevice attrs;
  B200_CUDA(attrs([] {
    const cudaError_t e = cudaFuncSetAttribute(attn_row_kernel<HD, GM, DECODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, KeyRing<HD>::smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attn_row_kernel<HD, GM, DECODE>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)splits, (unsigned)(a.d.Hq / a.G), (unsigned)B);
  cfg.blockDim = dim3(kAttnThreads);
  cfg.dynamicSmemBytes = KeyRing<HD>::smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  g_launches.fetch_add(1);
  B200_CUDA(cudaLaunchKernelEx(&cfg, attn_row_kernel<HD, GM, DECODE>, a));
  return B200_OK;
}
template <int HD, bool DECODE>
static int launch_row_g(const AttnRow& a, int splits, int B, cudaStream_t st, bool pdl) {
  if (a.G == 1) return launch_row_t<HD, 1, DECODE>(a, splits, B, st, pdl);
  if (a.G == 2) return launch_row_t<HD, 2, DECODE>(a, splits, B, st, pdl);
  return a.G <= 4 ? launch_row_t<HD, 4, DECODE>(a, splits, B, st, pdl) : launch_row_t<HD, 8, DECODE>(a, splits, B, st, pdl);
}
// The heads of a CTA: the largest divisor of the group up to eight.  The CTAs of a cluster: as many (a power of two up to 16) as the SMs hold
// clusters of at once, two CTAs to an SM (14 of 16 CTAs, 33 of 8, 71 of 4, 148 of 2), while each keeps 64 of `keys` keys.  Every CTA is a range of keys
// with a maximum and sums of its own, so their number is part of a sequence's bits: a decoded batch takes what the largest one would, whatever
// its size, and the limits are constants, not the chip's.  µs a token at positions 100 / 1 000 / 3 900, caches for 4 096, CTAs by the batch's own size → by
// the largest: 28 layers, 8 KV heads of 128, two sequences 884 / 930 / 1 137 → 876 / 991 / 1 405, four 1 032 / 1 102 / 1 431 → 906 / 1 027 / 1 445, eight
// the same; 24 layers, 2 KV heads of 64, two 577 / 579 / 628 → 576 / 589 / 709.  Sixteen ranges for every batch, several to a CTA with the same sums: four
// sequences 1 039 / 1 315 / 1 629, the merges of the ranges cost more than the waves they save.
static int launch_row(AttnRow& a, int hd, int64_t keys, int B, bool decode, cudaStream_t st, bool pdl) {
  const int group = a.d.Hq / a.d.Hkv;
  a.G = 1;
  for (int g = 2; g <= 8; ++g)
    if (group % g == 0) a.G = g;
  const int64_t clusters = (int64_t)(a.d.Hq / a.G) * (decode && B > 1 ? std::max(B, kMaxBatch) : B);
  const int most = clusters <= 14 ? 16 : clusters <= 33 ? 8 : clusters <= 71 ? 4 : clusters <= 148 ? 2 : 1;
  int splits = 1;
  while (splits < most && keys >= 128 * splits) splits *= 2, ++a.log_splits;
  a.per_kv = group / a.G;
  if (hd == 64) return decode ? launch_row_g<64, true>(a, splits, B, st, pdl) : launch_row_g<64, false>(a, splits, B, st, pdl);
  return decode ? launch_row_g<128, true>(a, splits, B, st, pdl) : launch_row_g<128, false>(a, splits, B, st, pdl);
}
static int launch_attn_row(void* o, const void* q, const void* k, const void* v, int64_t B, int64_t Skv, int64_t Hq, int64_t Hkv, int64_t hd,
                           int causal, cudaStream_t st) {
  B200_CHECK_ARG(hd == 64 || hd == 128, "attention: head_dim %lld not built (64 and 128 are)", (long long)hd);
  B200_CHECK_ARG(B > 0 && Skv > 0 && Hkv > 0 && Hq % Hkv == 0 && Hq < 65536 && B < 65536, "attention: bad shape");
  B200_CHECK_ARG(Skv < (1ll << 30), "attention: too many keys");
  AttnRow a{};
  a.d.qkv = (const __nv_bfloat16*)q;
  a.d.out = (__nv_bfloat16*)o;
  a.d.kcache = const_cast<__nv_bfloat16*>((const __nv_bfloat16*)k);   // read only
  a.d.vcache = const_cast<__nv_bfloat16*>((const __nv_bfloat16*)v);
  a.d.Hq = (int)Hq;
  a.d.Hkv = (int)Hkv;
  a.d.qkv_bstride = a.d.out_bstride = Hq * hd;
  a.kv_bstride = Skv * Hkv * hd;
  a.nkeys = causal ? 1 : (int)Skv;   // causal: the mask is top-left aligned, row 0 sees key 0
  return launch_row(a, (int)hd, a.nkeys, (int)B, false, st, op_pdl(st));
}

int launch_attn_decode(const AttnDecodeParams& p, int hd, cudaStream_t st, bool pdl) {
  B200_CHECK_ARG(hd == 64 || hd == 128, "attention: head_dim %d not built (64 and 128 are, like the reference)", hd);
  B200_CHECK_ARG(p.Hkv > 0 && p.Hq % p.Hkv == 0, "attention: Hq=%d must be a multiple of Hkv=%d", p.Hq, p.Hkv);
  const int G = p.heads_per_cta > 0 ? p.heads_per_cta : attn_heads_per_cta(p.Hq, p.Hkv, p.max_ctx);
  B200_CHECK_ARG((p.Hq / p.Hkv) % G == 0, "attention: heads per CTA %d must divide the GQA group %d", G, p.Hq / p.Hkv);
  B200_CHECK_ARG(p.max_ctx >= 1 && p.nsplit == attn_decode_nsplit(hd, p.max_ctx),
                 "attention: nsplit %d does not match max_ctx %d (need %d)", p.nsplit, p.max_ctx,
                 attn_decode_nsplit(hd, p.max_ctx));
  B200_CHECK_ARG(p.nsplit <= 65535, "attention: context too long");
  B200_CHECK_ARG(G >= 1 && G <= 8, "attention: at most 8 query heads per CTA (got %d)", G);
  const unsigned nb = (unsigned)std::max(1, p.batch);
  // The operator takes the cluster kernel at any length: no tickets to be zeroed by a launch of their own, which cost it more than its attention (µs a call,
  // 16 / 8 heads of 128, caches for 256 / 1 024: 19.8 / 19.8, with a native call 12.1 / 17.4, here 5.4 / 5.5).  The engines' steps stay with the
  // other kernel up to kLongSplits, whose bits theirs are.
  if (p.nsplit > kLongSplits || p.late) {
    AttnRow a{p, 0, p.cache_bstride, 1, 1, 0};
    return launch_row(a, hd, p.max_ctx, (int)nb, true, st, pdl);
  }
  if (hd == 64)
    B200_CUDA(launch_pdl(attn_decode_reg_kernel<64>, dim3(p.nsplit, p.Hq / G, nb), dim3(kAttnThreads), 0, st, pdl, p, G));
  else
    B200_CUDA(launch_pdl(attn_decode_reg_kernel<128>, dim3(p.nsplit, p.Hq / G, nb), dim3(kAttnThreads), 0, st, pdl, p, G));
  return B200_OK;
}

int launch_attn_general(void* o, const void* q, const void* k, const void* v, int64_t B, int64_t Sq, int64_t Skv,
                        int64_t Hq, int64_t Hkv, int64_t hd, int causal, cudaStream_t st) {
  B200_CHECK_ARG(hd == 64 || hd == 128, "attention: head_dim %lld not built (64 and 128 are)", (long long)hd);
  B200_CHECK_ARG(B > 0 && Sq > 0 && Skv > 0 && Hkv > 0 && Hq % Hkv == 0 && Hq < 65536 && B < 65536,
                 "attention: bad shape");
  dim3 grid((unsigned)Sq, (unsigned)Hq, (unsigned)B);
  const int k_wide = aligned16(k) ? 1 : 0;
  g_launches.fetch_add(1);
  if (hd == 64)
    attn_general_kernel<64><<<grid, 128, 0, st>>>((__nv_bfloat16*)o, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k,
                                                  (const __nv_bfloat16*)v, (int)Sq, (int)Skv, (int)Hq, (int)Hkv, causal, k_wide);
  else
    attn_general_kernel<128><<<grid, 128, 0, st>>>((__nv_bfloat16*)o, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k,
                                                   (const __nv_bfloat16*)v, (int)Sq, (int)Skv, (int)Hq, (int)Hkv,
                                                   causal, k_wide);
  B200_CUDA(cudaGetLastError());
  return B200_OK;
}

}  // namespace b200

extern "C" int b200_attn_bf16(void* o, const void* q, const void* k, const void* v, int64_t B, int64_t Sq, int64_t Skv,
                              int64_t Hq, int64_t Hkv, int64_t hd, int causal, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(o && q && k && v, "attention: null pointer");
  if (int bad = op_wait_check()) return bad;
  // A contiguous view may start anywhere: the prompt kernels read q, k and v 16 bytes at a time and store o in words, the row kernel reads k
  // and v 16 bytes at a time; what is not aligned for them goes to the general kernel.
  if (causal && Sq == Skv && Sq > 1 && prefill_attn_mma_enabled() && aligned16(q, k, v) && (reinterpret_cast<uintptr_t>(o) & 3) == 0)
    return launch_attn_causal_mma(o, q, k, v, B, Sq, Hq, Hkv, hd, (cudaStream_t)stream);
  if (Sq == 1 && aligned16(k, v)) return launch_attn_row(o, q, k, v, B, Skv, Hq, Hkv, hd, causal, (cudaStream_t)stream);
  return launch_attn_general(o, q, k, v, B, Sq, Skv, Hq, Hkv, hd, causal, (cudaStream_t)stream);
}
