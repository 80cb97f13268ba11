// prefill_attn_tc.cu — causal flash attention of a PREFILL chunk on the 5th-generation tensor cores (tcgen05, TMEM, TMA) for head
// sizes 64 and 128, sm_100a.  Same arithmetic as prefill_attn.cu (bf16 Q·Kᵀ products summed in fp32, base-2 online softmax in
// fp32, P rounded to bf16, bf16 P·V products summed in fp32), same masks (causal over a cached prefix, sliding window with
// kept first keys), sink and per-head gate.
//
// Shape of the work: a CTA takes 128 query rows of one query head, keys in tiles of 64 in ascending order, two CTAs per SM
// (96 KB of shared memory, 256 TMEM columns each) so that one CTA's softmax runs beside the other's products:
//   warp 0    TMA producer: the Q block once, then K and V tiles (128-byte swizzle; rows past the sequence are zero-filled)
//   warp 1    MMA issuer (one thread): S = Q·Kᵀ of the next tile goes out before P·V of this one, so the tensor pipe works
//             while the softmax warps hold a tile; S is double-buffered in TMEM, O stays in TMEM
//   warps 2-5 softmax, one row per thread: S from TMEM, row maximum and sum without shuffles, P (bf16) back into the TMEM columns
//             of S as the A operand of P·V; O is rescaled in TMEM where a row's maximum grew (nearly every tile of 32 rows), behind the
//             exponentials: by then the product before is over and S's registers are free for two loads of O in flight
//             (16 heads of 128 over 2 048 rows 51.1 → 48.1 µs)
// Late query blocks (most keys) of all heads are scheduled first.
//
// A key that a row does not see has P = 0, and 0 · V is 0 only for finite V: tiles that some row of the block sees in part are looked
// through, and a block that meets an infinity or a NaN there is computed again key by key (see_alone), so that nothing a row
// does not see reaches it.
//
// Bound by the chain of tiles that a late block waits for: about 1.1 µs each, most of it the latency of TMEM loads, maxima, 64
// exponentials and TMEM stores of one warp (issue slots 26 %, tensor pipe 20 % busy).  µs, mma.sync → here, same error against 64 bits:
// 16 heads of 128 over 2 048 rows 112 → 48, 24 heads 146 → 53; 14 heads of 64 over 2 048 rows 51 → 41; 16 heads of 128 over 512
// rows 17.8 → 18.2, which is where the dispatch stops (prefill_attn_tc_wins).
#include "ops.cuh"
#include "tc.cuh"

#include <algorithm>
#include <mutex>

namespace b200 {

namespace {

constexpr int kTBM = 128, kTBN = 64, kTThreads = 192;
constexpr unsigned kAttnWaitCode = 0xa7000000u;

struct TcAttn {
  __nv_bfloat16* o;
  const __nv_bfloat16* gate;
  int64_t o_rs, o_bs, q_rs, q_bs;
  int S, Hq, Hkv, p0;
  float scale_log2;
  int window, keep_first, sink;
  unsigned* err;
  const __nv_bfloat16 *qp, *kp, *vp;   // see_alone
  int64_t kv_rs, kv_bs;
};

template <int HD>
struct TcCfg {
  static constexpr int NB = HD / 64;                 // 64-column blocks of a row (one swizzle atom wide)
  static constexpr int ST = HD == 64 ? 4 : 2;        // K and V stages
  static constexpr int QB = NB * kTBM * 128, TB = NB * kTBN * 128;
  static constexpr int smem = QB + 2 * ST * TB + 1024 /*align*/ + 256 /*barriers*/;
};

// weights below 2⁻¹²⁶ of a row's largest count as zero (with subnormals 16 heads over 2 048 rows take 53.9 instead of 51.6 µs)
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 at a time
__device__ __forceinline__ uint64_t pack_f2(float a, float b) { return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32); }
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_f2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float lo_f2(uint64_t a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float hi_f2(uint64_t a) { return __uint_as_float((uint32_t)(a >> 32)); }
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int32_t c0, int32_t c1, int32_t c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// D[tmem] (+)= A[tmem]·B[smem]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
      "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// [keys][64 columns] rows of 128 bytes, 128-byte swizzle, as a B operand whose N runs along the columns (MN-major): 64-column blocks
// `blk` bytes apart (bits 16-29), groups of 8 keys 1 024 bytes apart (bits 32-45)
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t smem_addr, uint32_t blk) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(blk >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// One row, the keys it sees one after another (P rounded to bf16 like above): the way out for a block whose partly visible tiles hold
// infinities or NaNs in V.  Slow and rare.
template <int HD>
__device__ __noinline__ void see_alone(const TcAttn& p, int b, int h, int kvh, int r, float (&ml)[2], int c, float (&acc)[32]) {
  const __nv_bfloat16* q = p.qp + (size_t)b * p.q_bs + (size_t)r * p.q_rs + (size_t)h * HD;
  const int rpos = p.p0 + r;
  for (int j = 0; j <= rpos; ++j) {
    if (p.window > 0 && rpos - j >= p.window && j >= p.keep_first) continue;
    const size_t row = (size_t)b * p.kv_bs + (size_t)j * p.kv_rs + (size_t)kvh * HD;
    float s = 0.f;
    for (int d = 0; d < HD; ++d) s = fmaf(bf16_to_f(q[d]), bf16_to_f(p.kp[row + d]), s);
    if (c < 0) {   // first walk: maximum and sum
      const float top = fmaxf(ml[0], s);
      ml[1] = ml[1] * (ml[0] == -INFINITY ? 0.f : ex2f((ml[0] - top) * p.scale_log2)) + ex2f((s - top) * p.scale_log2);
      ml[0] = top;
    } else {
      const float w = round_bf16(ex2f((s - ml[0]) * p.scale_log2));
      for (int e = 0; e < 32; ++e) acc[e] = fmaf(w, bf16_to_f(p.vp[row + c + e]), acc[e]);
    }
  }
}

template <int HD>
__global__ void __launch_bounds__(kTThreads, 2)
attn_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
               const TcAttn p) {
  using C = TcCfg<HD>;
  constexpr int NB = C::NB, ST = C::ST;
  constexpr uint32_t kIdescS = umma_idesc(kTBM, kTBN), kIdescO = umma_idesc(kTBM, HD, true);
  constexpr int kCols = 256, kColO = 128;   // S at columns 0 and 64, O from column 128 on
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                      // [NB][128 rows × 128 bytes]
  uint8_t* sK = sQ + C::QB;                // [ST][NB][64 keys × 128 bytes]
  uint8_t* sV = sK + ST * C::TB;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sV + ST * C::TB);
  uint64_t* k_full = q_full + 1;           // [ST]
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint64_t* s_full = v_empty + ST;         // [2]
  uint64_t* p_full = s_full + 2;           // [2], one arrival per softmax warp
  uint64_t* pv_done = p_full + 2;          // one phase per tile but the last
  uint64_t* o_full = pv_done + 1;          // the last tile's product, and so all of them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  int* not_finite = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, qb = (int)gridDim.y - 1 - (int)blockIdx.y, b = blockIdx.z;
  const int kvh = h / (p.Hq / p.Hkv);
  const int q0 = qb * kTBM;
  const int rows_valid = min(kTBM, p.S - q0);
  const int first_pos = p.p0 + q0, last_pos = first_pos + rows_valid - 1;
  const int T = last_pos / kTBN + 1;
  // tiles to visit: with a window those of the kept first keys, then from the first row's window edge up to the diagonal
  const int t_lo = p.window > 0 ? max(0, first_pos - p.window + 1) / kTBN : 0;
  const int n_keep = p.window > 0 ? min(t_lo, (p.keep_first + kTBN - 1) / kTBN) : 0;
  const int n_tiles = T - t_lo + n_keep;
  auto tile_of = [&](int it) { return it < n_keep ? it : t_lo + (it - n_keep); };
  bool ok = true;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
    mbar_init(q_full, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 4);
    }
    mbar_init(pv_done, 1);
    mbar_init(o_full, 1);
    *not_finite = 0;
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc<1>(tmem_slot, kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, C::QB);
#pragma unroll
      for (int c = 0; c < NB; ++c) tma_load_3d(sQ + c * kTBM * 128, &tq, h * HD + c * 64, q0, b, q_full);
      int s = 0;
      uint32_t ph = 1;
      for (int it = 0; it < n_tiles; ++it) {
        const int k0 = tile_of(it) * kTBN;
        if (!(ok = mbar_wait_limited(&k_empty[s], ph, p.err, kAttnWaitCode | 1))) break;
        mbar_arrive_expect_tx(&k_full[s], C::TB);
#pragma unroll
        for (int c = 0; c < NB; ++c) tma_load_3d(sK + s * C::TB + c * kTBN * 128, &tk, kvh * HD + c * 64, k0, b, &k_full[s]);
        if (!(ok = mbar_wait_limited(&v_empty[s], ph, p.err, kAttnWaitCode | 2))) break;
        mbar_arrive_expect_tx(&v_full[s], C::TB);
#pragma unroll
        for (int c = 0; c < NB; ++c) tma_load_3d(sV + s * C::TB + c * kTBN * 128, &tv, kvh * HD + c * 64, k0, b, &v_full[s]);
        if (++s == ST) {
          s = 0;
          ph ^= 1;
        }
      }
      if (!ok) drain_async();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t q_u = smem_u32(sQ), k_u = smem_u32(sK), v_u = smem_u32(sV);
      auto scores = [&](int it) -> bool {   // S[it & 1] = Q·Kᵀ of tile it
        const int s = it % ST;
        if (!mbar_wait_limited(&k_full[s], (uint32_t)((it / ST) & 1), p.err, kAttnWaitCode | 3)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          umma_bf16(tmem + (uint32_t)((it & 1) * 64), umma_desc(q_u + (kk / 4) * kTBM * 128 + (kk % 4) * 32),
                    umma_desc(k_u + s * C::TB + (kk / 4) * kTBN * 128 + (kk % 4) * 32), kIdescS, kk > 0 ? 1u : 0u);
        umma_commit(&k_empty[s]);
        umma_commit(&s_full[it & 1]);
        return true;
      };
      ok = mbar_wait_limited(q_full, 0, p.err, kAttnWaitCode | 4) && scores(0);
      for (int it = 0; it < n_tiles && ok; ++it) {
        // the buffer that tile it + 1 overwrites held P of tile it - 1: its product went out before, and products run in order
        if (it + 1 < n_tiles && !(ok = scores(it + 1))) break;
        const int s = it % ST;
        if (!(ok = mbar_wait_limited(&p_full[it & 1], (uint32_t)((it >> 1) & 1), p.err, kAttnWaitCode | 5))) break;
        if (!(ok = mbar_wait_limited(&v_full[s], (uint32_t)((it / ST) & 1), p.err, kAttnWaitCode | 6))) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < kTBN / 16; ++kk)   // 16 keys: 8 columns of P, 2 048 bytes further down V's rows
          umma_bf16_ts(tmem + kColO, tmem + (uint32_t)((it & 1) * 64 + kk * 8), umma_desc_mn(v_u + s * C::TB + kk * 2048, kTBN * 128), kIdescO,
                       (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&v_empty[s]);
        umma_commit(it + 1 < n_tiles ? pv_done : o_full);
      }
      if (!ok) drain_async();
    }
  } else {
    // ---------------------------------------------------------------------------------------------- softmax
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const int rpos = first_pos + min(row, rows_valid - 1);   // padding rows behave like the last valid row
    const float k_scale = p.scale_log2;
    const uint64_t scale2 = pack_f2(k_scale, k_scale);
    float m = -INFINITY, l = 0.f;
    for (int it = 0; it < n_tiles; ++it) {
      ok = __all_sync(0xffffffffu, mbar_wait_limited(&s_full[it & 1], (uint32_t)((it >> 1) & 1), p.err, kAttnWaitCode | 7));
      if (!ok) break;
      tc_fence_after();
      uint32_t s0[32], s1[32];
      const uint32_t sbuf = lane_base + (uint32_t)((it & 1) * 64);
      tmem_ld32(sbuf, s0);
      tmem_ld32(sbuf + 32, s1);
      tmem_wait_ld();
      const int kbase = tile_of(it) * kTBN;
      if (kbase + kTBN - 1 > first_pos || (p.window > 0 && last_pos - kbase >= p.window)) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int j0 = kbase + j, j1 = kbase + 32 + j;
          if (j0 > rpos || (p.window > 0 && rpos - j0 >= p.window && j0 >= p.keep_first)) s0[j] = 0xff800000u;
          if (j1 > rpos || (p.window > 0 && rpos - j1 >= p.window && j1 >= p.keep_first)) s1[j] = 0xff800000u;
        }
        const int vs = it % ST;
        ok = __all_sync(0xffffffffu, mbar_wait_limited(&v_full[vs], (uint32_t)((it / ST) & 1), p.err, kAttnWaitCode | 10));
        if (!ok) break;
        const uint4* vt = reinterpret_cast<const uint4*>(sV + vs * C::TB);
        bool bad = false;
#pragma unroll
        for (int j = 0; j < C::TB / 16 / 128; ++j) {
          const uint4 w = vt[j * 128 + row];
          const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) bad = bad || (x[e] & 0x7f80u) == 0x7f80u || (x[e] & 0x7f800000u) == 0x7f800000u;
        }
        if (bad) *not_finite = 1;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(s0[j + e]), __uint_as_float(s1[j + e])));
      }
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const bool grow = top > m;
      const bool rescale = it > 0 && __any_sync(0xffffffffu, grow);
      const float alpha = grow && it > 0 ? ex2f((m - top) * k_scale) : 1.f;
      if (grow) m = top;
      l *= alpha;
      const float ms = m == -INFINITY ? 0.f : m * k_scale;
      const uint64_t neg = pack_f2(-ms, -ms);
      uint64_t sum[2] = {0, 0};
      uint32_t pk[32];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const uint64_t za = fma_f2(pack_f2(__uint_as_float(s0[2 * j]), __uint_as_float(s0[2 * j + 1])), scale2, neg);
        const uint64_t zb = fma_f2(pack_f2(__uint_as_float(s1[2 * j]), __uint_as_float(s1[2 * j + 1])), scale2, neg);
        const float a0 = ex2f(lo_f2(za)), a1 = ex2f(hi_f2(za)), b0 = ex2f(lo_f2(zb)), b1 = ex2f(hi_f2(zb));
        sum[0] = add_f2(sum[0], pack_f2(a0, a1));
        sum[1] = add_f2(sum[1], pack_f2(b0, b1));
        pk[j] = pack2(a0, a1);
        pk[16 + j] = pack2(b0, b1);
      }
      sum[0] = add_f2(sum[0], sum[1]);
      l += lo_f2(sum[0]) + hi_f2(sum[0]);
      tmem_st32(sbuf, pk);
      if (rescale) {
        ok = __all_sync(0xffffffffu, mbar_wait_limited(pv_done, (uint32_t)((it - 1) & 1), p.err, kAttnWaitCode | 8));
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD; c += 64) {
          uint32_t o0[32], o1[32];
          tmem_ld32(lane_base + kColO + c, o0);
          tmem_ld32(lane_base + kColO + c + 32, o1);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            o0[j] = __float_as_uint(__uint_as_float(o0[j]) * alpha);
            o1[j] = __float_as_uint(__uint_as_float(o1[j]) * alpha);
          }
          tmem_st32(lane_base + kColO + c, o0);
          tmem_st32(lane_base + kColO + c + 32, o1);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[it & 1]);
    }
    // ---- normalise and store.  The end has a barrier of its own: a parity tells a phase from its neighbours only, and here the products
    // of the last two tiles may both be running (inside the loop S of tile it says that the product of tile it - 2 is over).
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait_limited(o_full, 0, p.err, kAttnWaitCode | 9));
    named_bar_sync(1, 128);
    const bool alone = *not_finite != 0;   // the same for all softmax threads
    if (ok) {
      tc_fence_after();
      if (alone) {
        float ml[2] = {-INFINITY, 0.f}, none[32];
        see_alone<HD>(p, b, h, kvh, q0 + min(row, rows_valid - 1), ml, -1, none);
        m = ml[0];
        l = ml[1];
      }
      if (p.sink && m != -INFINITY) l += ex2f(-m * k_scale);
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (p.gate != nullptr && row < rows_valid)
        inv *= 1.f / (1.f + expf(-bf16_to_f(p.gate[(size_t)b * p.q_bs + (size_t)(q0 + row) * p.q_rs + h])));
      __nv_bfloat16* dst = p.o + (size_t)b * p.o_bs + (size_t)(q0 + min(row, rows_valid - 1)) * p.o_rs + (size_t)h * HD;
#pragma unroll 1
      for (int c = 0; c < HD; c += 32) {
        uint32_t o[32];
        tmem_ld32(lane_base + kColO + c, o);
        tmem_wait_ld();
        if (alone) {
          float ml[2] = {m, l}, acc[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j] = 0.f;
          see_alone<HD>(p, b, h, kvh, q0 + min(row, rows_valid - 1), ml, c, acc);
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(acc[j]);
        }
        if (row < rows_valid) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 v;
            v.x = pack2(__uint_as_float(o[8 * j]) * inv, __uint_as_float(o[8 * j + 1]) * inv);
            v.y = pack2(__uint_as_float(o[8 * j + 2]) * inv, __uint_as_float(o[8 * j + 3]) * inv);
            v.z = pack2(__uint_as_float(o[8 * j + 4]) * inv, __uint_as_float(o[8 * j + 5]) * inv);
            v.w = pack2(__uint_as_float(o[8 * j + 6]) * inv, __uint_as_float(o[8 * j + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c + 8 * j) = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_free<1>(tmem, kCols);
  }
}

template <int HD>
int launch_tc(const TcPrefillAttn& a, cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(attn_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<HD>::smem);
  });
  B200_CUDA(attr_err);
  TcAttn p{};
  int rc;
  if ((rc = wait_word(&p.err)) != B200_OK) return rc;
  p.o = a.o; p.gate = a.gate; p.o_rs = a.o_rs; p.o_bs = a.o_bs; p.q_rs = a.q_rs; p.q_bs = a.q_bs;
  p.S = a.S; p.Hq = a.Hq; p.Hkv = a.Hkv; p.p0 = a.p0;
  p.scale_log2 = a.scale_log2; p.window = a.window; p.keep_first = a.keep_first; p.sink = a.sink;
  p.qp = a.q; p.kp = a.k; p.vp = a.v; p.kv_rs = a.kv_rs; p.kv_bs = a.kv_bs;
  const int64_t keys = (int64_t)a.p0 + a.S;
  CUtensorMap tq, tk, tv;
  if ((rc = make_tmap_sw128(&tq, 3, a.q, a.B, a.S, (int64_t)a.Hq * HD, a.q_bs, a.q_rs, kTBM)) != B200_OK) return rc;
  if ((rc = make_tmap_sw128(&tk, 3, a.k, a.B, keys, (int64_t)a.Hkv * HD, a.kv_bs, a.kv_rs, kTBN)) != B200_OK) return rc;
  if ((rc = make_tmap_sw128(&tv, 3, a.v, a.B, keys, (int64_t)a.Hkv * HD, a.kv_bs, a.kv_rs, kTBN)) != B200_OK) return rc;
  const dim3 grid((unsigned)a.Hq, (unsigned)((a.S + kTBM - 1) / kTBM), (unsigned)a.B);
  g_launches.fetch_add(1);
  attn_tc_kernel<HD><<<grid, kTThreads, TcCfg<HD>::smem, st>>>(tq, tk, tv, p);
  B200_CUDA(cudaGetLastError());
  return B200_OK;
}

}  // namespace

bool prefill_attn_tc_ok(const TcPrefillAttn& a, int hd) {
  return (hd == 64 || hd == 128) && (a.S + kTBM - 1) / kTBM < 65536 && a.B < 65536 && aligned16(a.o, a.q, a.k, a.v) && a.q_rs % 8 == 0 &&
         a.q_bs % 8 == 0 && a.kv_rs % 8 == 0 && a.kv_bs % 8 == 0 && a.o_rs % 8 == 0 && a.o_bs % 8 == 0;
}
// Whether this kernel beats the mma.sync one, by fits (µs) to both over 128 … 2 048 rows, 14 … 64 (head, sequence) pairs: this one takes a launch
// and pipeline fill of 9.6 and the longest block's tiles one after another; that one the larger of its longest block's tiles and all
// of its 64 × 64 tiles on the tensor cores, and a third of the smaller.
bool prefill_attn_tc_wins(const TcPrefillAttn& a, int hd, int rows) {
  double all = 0, longest = 0;
  for (int r = 0; r < rows; r += 64) {
    const int last = std::min(rows, r + 64) - 1, edge = a.window > 0 ? std::max(0, r - a.window + 1) / 64 : 0;
    const double tiles = last / 64 + 1 - edge + (a.window > 0 ? std::min(edge, (a.keep_first + 63) / 64) : 0);
    all += tiles;
    longest = std::max(longest, tiles);
  }
  all *= (double)a.B * a.Hq;
  const double chain = (hd == 64 ? 1.0 : 1.75) * longest, work = (hd == 64 ? 0.0066 : 0.0133) * all;
  const double mma = 3.3 + std::max(chain, work) + 0.3 * std::min(chain, work);
  const double here = std::max(9.6 + (hd == 64 ? 0.98 : 1.1) * longest, 5.0 + 0.0038 * all);
  return here < mma;
}
int launch_prefill_attn_tc(const TcPrefillAttn& a, int hd, cudaStream_t st) { return hd == 64 ? launch_tc<64>(a, st) : launch_tc<128>(a, st); }

}  // namespace b200
