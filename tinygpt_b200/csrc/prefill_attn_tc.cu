// prefill_attn_tc.cu — causal flash attention of a PREFILL chunk on the 5th-generation tensor cores (tcgen05, TMEM, TMA) for head
// sizes 64 and 128, sm_100a.  Same arithmetic as prefill_attn.cu (bf16 Q·Kᵀ products summed in fp32, base-2 online softmax in
// fp32, P rounded to bf16, bf16 P·V products summed in fp32), same masks (causal over a cached prefix, sliding window with
// kept first keys), sink and per-head gate.
//
// Shape of the work: 128 query rows of one query head against keys in tiles of 64 in ascending order, by one CTA or by a cluster of two that
// share the tiles by parity (attn_tc_halves), two CTAs per SM (96 KB of shared memory, 256 TMEM columns each) so that one CTA's softmax
// runs beside the other's products:
//   warp 0    TMA producer: the Q block once, then K and V tiles (128-byte swizzle; rows past the sequence are zero-filled)
//   warp 1    MMA issuer (one thread): S = Q·Kᵀ of the next tile goes out before P·V of this one, so the tensor pipe works
//             while the softmax warps hold a tile; S is double-buffered in TMEM, O stays in TMEM
//   warps 2-5 softmax, one row per thread: S from TMEM, row maximum and sum without shuffles, P (bf16) back into the TMEM columns
//             of S as the A operand of P·V; O is rescaled in TMEM where a row's maximum grew (nearly every tile of 32 rows), behind the
//             exponentials: by then the product before is over and S's registers are free for two loads of O in flight
// Late query blocks (most keys) of all heads are scheduled first.  Two CTAs of a cluster end with a maximum, a sum and 128 columns of O per row
// each: one hands the other half of its columns through distributed shared memory, and each finishes its own half.
//
// A key that a row does not see has P = 0, and 0 · V is 0 only for finite V: tiles that some row of the block sees in part are looked
// through, and a block that meets an infinity or a NaN there is computed again key by key (see_alone), so that nothing a row
// does not see reaches it.
//
// Bound by the chain of a block's tiles, S → softmax → P·V in turn, and by how long and short blocks come to lie on the SMs: 16 heads of 128 over 2 048
// rows keep the tensor pipe 28 % and the issue slots 30 % busy (a tile's products take 640 cycles, those of N = 64 three quarters of what
// N = 128 takes: 48 and 64 cycles).  Small calls by what a CTA does once: barriers, TMEM and the first loads, the merge and the stores.  128-key tiles
// (P then shares the only S buffer) and eight softmax warps of 64 keys were no faster: 43 and 40 µs where this form took 38.
// Masks as bits (two comparisons per key took longer than whole tiles), results stored in whole rows through shared memory
// (straight from the lanes a store touches 32 rows), the first loads in front of the TMEM allocation, waits whose first look is inline.
// µs, mma.sync / here at first / now, same error against 64 bits: 16 heads of 128 over 2 048 rows 64 / 51 / 34.6, 24 heads
// 98 / 53 / 41.4, 32 heads 123 / 71 / 52.5; 16 heads over 512 rows 14.2 / 18.2 / 10.6; 14 heads of 64 over 2 048 rows 48 / 41 / 29.2,
// four sequences of 333 rows 12.1 / - / 9.9.
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
  int pdl;
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
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
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
// D[tmem] (+)= A[tmem]·B[smem], B's descriptor by its lower half: the address and, from bit 16 on, the distance of 64-column blocks of an operand
// whose N runs along the columns (V's [keys][64 columns] rows of 128 bytes, MN-major)
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}" ::"r"(d), "r"(a), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
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
// A wait that gave up says so to the whole CTA and sets `dead`: its role goes on without waiting (what follows neither hangs nor leaves
// the buffers), and nothing is stored.  The first look is inline and has no loop around it.
__device__ __noinline__ bool wait_slow(uint64_t* bar, uint32_t parity, unsigned* err, unsigned code, volatile int* gave_up) {
  if (mbar_wait_limited(bar, parity, err, code)) return false;
  *gave_up = 1;
  __threadfence_block();
  return true;
}
__device__ __forceinline__ uint32_t bits_below(int n) { return n >= 32 ? ~0u : n <= 0 ? 0u : (1u << n) - 1; }

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

template <int HD, int SPLIT>
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
  int* gave_up = not_finite + 1;
  float4* part = reinterpret_cast<float4*>(sQ);   // [128 rows]: maximum, sum, V is not finite, gave up
  float4* give = reinterpret_cast<float4*>(sK);   // [HD / 8][128 rows]: the columns that the other CTA finishes

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = SPLIT == 2 ? (int)cluster_rank() : 0;
  const int h = blockIdx.x / SPLIT, qb = (int)gridDim.y - 1 - (int)blockIdx.y, b = blockIdx.z;
  const int kvh = h / (p.Hq / p.Hkv);
  const int q0 = qb * kTBM;
  const int rows_valid = min(kTBM, p.S - q0);
  const int first_pos = p.p0 + q0, last_pos = first_pos + rows_valid - 1;
  const int T = last_pos / kTBN + 1;
  // tiles to visit: with a window those of the kept first keys, then from the first row's window edge up to the diagonal
  const int t_lo = p.window > 0 ? max(0, first_pos - p.window + 1) / kTBN : 0;
  const int n_keep = p.window > 0 ? min(t_lo, (p.keep_first + kTBN - 1) / kTBN) : 0;
  // this CTA's share of them: all, or the tiles of its parity.  By the tile's place in the cache, so that a row's sums are the same however
  // its prompt is cut
  const int own_keep = SPLIT == 2 ? (n_keep + 1 - half) >> 1 : n_keep, own_lo = SPLIT == 2 ? t_lo + ((t_lo ^ half) & 1) : t_lo;
  const int n_tiles = own_keep + (max(T - own_lo, 0) + SPLIT - 1) / SPLIT;
  auto tile_of = [&](int it) { return it < own_keep ? half + SPLIT * it : own_lo + SPLIT * (it - own_keep); };
  bool dead = false;
  auto wait_for = [&](uint64_t* bar, uint32_t parity, unsigned code) {
    if (!mbar_try_wait(bar, parity) && !dead) dead = wait_slow(bar, parity, p.err, code, gave_up);
  };

  auto load_k = [&](int it, int s) {
    mbar_arrive_expect_tx(&k_full[s], C::TB);
#pragma unroll
    for (int c = 0; c < NB; ++c) tma_load_3d(sK + s * C::TB + c * kTBN * 128, &tk, kvh * HD + c * 64, tile_of(it) * kTBN, b, &k_full[s]);
  };
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
    *gave_up = 0;
    fence_mbar_init();
    if (p.pdl) pdl_wait();
    if (n_tiles > 0) {   // on their way while TMEM is allocated
      load_k(0, 0);
      mbar_arrive_expect_tx(q_full, C::QB);
#pragma unroll
      for (int c = 0; c < NB; ++c) tma_load_3d(sQ + c * kTBM * 128, &tq, h * HD + c * 64, q0, b, q_full);
    }
  }
  if (warp == 2) tmem_alloc<1>(tmem_slot, kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (p.pdl) pdl_wait();

  float4 mine{};   // of a row: maximum, sum, V is not finite, gave up
  if (warp == 0) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 1;
      for (int it = 0; it < n_tiles; ++it) {
        if (it > 0) {
          wait_for(&k_empty[s], ph, kAttnWaitCode | 1);
          load_k(it, s);
        }
        wait_for(&v_empty[s], ph, kAttnWaitCode | 2);
        mbar_arrive_expect_tx(&v_full[s], C::TB);
#pragma unroll
        for (int c = 0; c < NB; ++c) tma_load_3d(sV + s * C::TB + c * kTBN * 128, &tv, kvh * HD + c * 64, tile_of(it) * kTBN, b, &v_full[s]);
        if (++s == ST) {
          s = 0;
          ph ^= 1;
        }
      }
      if (dead) drain_async();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------------- MMA issuer
    if (n_tiles > 0 && elect_one()) {
      const uint32_t q_u = desc_lo(smem_u32(sQ)), k_u = desc_lo(smem_u32(sK)), v_u = desc_lo(smem_u32(sV));
      bool k_ready = false;   // of the tile after the next, looked at before the products of this one go out
      auto scores = [&](int it) {   // S[it & 1] = Q·Kᵀ of tile it
        const int s = it % ST;
        if (!k_ready) wait_for(&k_full[s], (uint32_t)((it / ST) & 1), kAttnWaitCode | 3);
        tc_fence_after();
        const uint32_t ks = k_u + s * (C::TB >> 4), d = tmem + (uint32_t)((it & 1) * 64);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          umma_lo<1>(d, q_u + (((kk / 4) * kTBM * 128 + (kk % 4) * 32) >> 4), ks + (((kk / 4) * kTBN * 128 + (kk % 4) * 32) >> 4), kIdescS,
                     kk > 0 ? 1u : 0u);
        umma_commit(&k_empty[s]);
        umma_commit(&s_full[it & 1]);
      };
      wait_for(q_full, 0, kAttnWaitCode | 4);
      scores(0);
      for (int it = 0; it < n_tiles; ++it) {
        // the buffer that tile it + 1 overwrites held P of tile it - 1: its product went out before, and products run in order
        if (it + 1 < n_tiles) scores(it + 1);
        const int s = it % ST, next = it + 2;
        wait_for(&v_full[s], (uint32_t)((it / ST) & 1), kAttnWaitCode | 6);
        wait_for(&p_full[it & 1], (uint32_t)((it >> 1) & 1), kAttnWaitCode | 5);
        tc_fence_after();
        k_ready = mbar_test(&k_full[next % ST], (uint32_t)((next / ST) & 1));
        const uint32_t vs = v_u + s * (C::TB >> 4), ps = tmem + (uint32_t)((it & 1) * 64);
#pragma unroll
        for (int kk = 0; kk < kTBN / 16; ++kk)   // 16 keys: 8 columns of P, 2 048 bytes further down V's rows
          umma_ts(tmem + kColO, ps + kk * 8, vs + (kk * 2048 >> 4) + ((kTBN * 128 >> 4) << 16), kIdescO, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&v_empty[s]);
        umma_commit(it + 1 < n_tiles ? pv_done : o_full);
      }
      if (dead) drain_async();
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
      wait_for(&s_full[it & 1], (uint32_t)((it >> 1) & 1), kAttnWaitCode | 7);
      __syncwarp();
      tc_fence_after();
      uint32_t s[2][32];
      const uint32_t sbuf = lane_base + (uint32_t)((it & 1) * 64);
      tmem_ld32(sbuf, s[0]);
      tmem_ld32(sbuf + 32, s[1]);
      tmem_wait_ld();
      const int kbase = tile_of(it) * kTBN;
      if (kbase + kTBN - 1 > first_pos || (p.window > 0 && last_pos - kbase >= p.window)) {
        // the keys this row sees, a bit each (comparing them one by one took longer than a whole tile)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int k0 = kbase + i * 32;
          const uint32_t seen = bits_below(rpos + 1 - k0) &
                                (p.window > 0 ? ~bits_below(rpos + 1 - p.window - k0) | bits_below(p.keep_first - k0) : ~0u);
#pragma unroll
          for (int j = 0; j < 32; ++j) s[i][j] = seen & (1u << j) ? s[i][j] : 0xff800000u;
        }
        const int vs = it % ST;
        wait_for(&v_full[vs], (uint32_t)((it / ST) & 1), kAttnWaitCode | 10);
        const uint4* vt = reinterpret_cast<const uint4*>(sV + vs * C::TB);
        bool bad = false;
#pragma unroll
        for (int j = 0; j < C::TB / 16 / 128; ++j) {
          const uint4 w = vt[j * 128 + row];
          const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) bad |= (x[e] & 0x7f80u) == 0x7f80u | (x[e] & 0x7f800000u) == 0x7f800000u;
        }
        if (bad) *not_finite = 1;
        __syncwarp();
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(s[0][j + e]), __uint_as_float(s[1][j + e])));
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
        const uint64_t za = fma_f2(pack_f2(__uint_as_float(s[0][2 * j]), __uint_as_float(s[0][2 * j + 1])), scale2, neg);
        const uint64_t zb = fma_f2(pack_f2(__uint_as_float(s[1][2 * j]), __uint_as_float(s[1][2 * j + 1])), scale2, neg);
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
        wait_for(pv_done, (uint32_t)((it - 1) & 1), kAttnWaitCode | 8);
        __syncwarp();
        tc_fence_after();
        const uint64_t alpha2 = pack_f2(alpha, alpha);
#pragma unroll 1
        for (int c = 0; c < HD; c += 64) {
          uint32_t o[2][32];
          tmem_ld32(lane_base + kColO + c, o[0]);
          tmem_ld32(lane_base + kColO + c + 32, o[1]);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const uint64_t y = mul_f2(pack_f2(__uint_as_float(o[i][j]), __uint_as_float(o[i][j + 1])), alpha2);
              o[i][j] = (uint32_t)y;
              o[i][j + 1] = (uint32_t)(y >> 32);
            }
          tmem_st32(lane_base + kColO + c, o[0]);
          tmem_st32(lane_base + kColO + c + 32, o[1]);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[it & 1]);
    }
    // ---- the end has a barrier of its own: a parity tells a phase from its neighbours only, and here the products of the last two tiles may
    // both be running (inside the loop S of tile it says that the product of tile it - 2 is over).
    if (n_tiles > 0) wait_for(o_full, 0, kAttnWaitCode | 9);
    __syncwarp();
    tc_fence_after();
    named_bar_sync(1, 128);   // every load and product of this CTA is over
    mine = make_float4(m, l, *not_finite != 0 ? 1.f : 0.f, dead || *gave_up != 0 ? 1.f : 0.f);
    if constexpr (SPLIT == 2) {   // the other CTA's columns, the maxima and the sums go where Q and K were
      part[row] = mine;
      if (n_tiles > 0) {
#pragma unroll 1
        for (int c = 0; c < HD / 2; c += 32) {
          uint32_t o[32];
          tmem_ld32(lane_base + kColO + (half ^ 1) * (HD / 2) + c, o);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            give[(c / 4 + j) * kTBM + row] = make_float4(__uint_as_float(o[4 * j]), __uint_as_float(o[4 * j + 1]), __uint_as_float(o[4 * j + 2]),
                                                         __uint_as_float(o[4 * j + 3]));
        }
      }
    }
  }
  // The next launch may come in only now: started with this one, its blocks, the longest first, would take the places that free up early, two long
  // ones to an SM (16 heads of 128 over 2 048 rows, calls behind each other: 42.2 µs)
  if (p.pdl) pdl_trigger();
  __syncwarp();
  if constexpr (SPLIT == 2) cluster_sync_all();   // both halves have written
  if (warp >= 2) {
    // ---- merge, normalise and store this CTA's columns
    constexpr int W = HD / SPLIT, CH = W / 8;   // columns; 16-byte pieces of a row of results
    const int q = warp & 3, row = q * 32 + lane;
    const int r = q0 + min(row, rows_valid - 1);
    const uint32_t o_at = tmem + ((uint32_t)(q * 32) << 16) + kColO + half * W;
    const float k_scale = p.scale_log2;
    float4 other = make_float4(-INFINITY, 0.f, 0.f, 0.f), y[SPLIT == 2 ? W / 4 : 1];
    if constexpr (SPLIT == 2) {
      const uint32_t take = mapa_u32(smem_u32(&give[row]), (uint32_t)(half ^ 1));
      other = ld_cluster_f4(mapa_u32(smem_u32(&part[row]), (uint32_t)(half ^ 1)));
#pragma unroll
      for (int j = 0; j < W / 4; ++j) y[j] = ld_cluster_f4(take + j * kTBM * 16);
      cluster_arrive();   // the other half may leave; its wait lies behind the store
    }
    const bool alone = __any_sync(0xffffffffu, mine.z + other.z != 0.f);
    float m = fmaxf(mine.x, other.x);
    // a half whose tiles the row does not see has no maximum and a sum of 0, or of NaN where its scores were
    const float fm = SPLIT == 1 ? 1.f : mine.x == -INFINITY ? mine.y : ex2f((mine.x - m) * k_scale);
    const float fo = SPLIT == 1 ? 0.f : other.x == -INFINITY ? other.y : ex2f((other.x - m) * k_scale);
    float l = SPLIT == 1 ? mine.y : mine.y * fm + other.y * fo;
    if (__all_sync(0xffffffffu, mine.w + other.w == 0.f)) {
      if (alone) {
        float ml[2] = {-INFINITY, 0.f}, none[32];
        see_alone<HD>(p, b, h, kvh, r, ml, -1, none);
        m = ml[0];
        l = ml[1];
      }
      if (p.sink && m != -INFINITY) l += ex2f(-m * k_scale);
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (p.gate != nullptr && row < rows_valid)
        inv *= 1.f / (1.f + expf(-bf16_to_f(p.gate[(size_t)b * p.q_bs + (size_t)(q0 + row) * p.q_rs + h])));
      // through shared memory (where V was), so that a store covers whole rows: straight from the lanes it touches 32 of them
      uint8_t* const mid = sV + q * (32 * W * 2);
      auto place = [&](int rw, int c) { return mid + rw * (W * 2) + (c ^ ((CH >= 8 ? rw : rw >> 1) & (CH >= 8 ? 7 : 3))) * 16; };
      const uint32_t km = fm != 0.f ? ~0u : 0u, ko = fo != 0.f ? ~0u : 0u;   // what a half of weight 0 holds is not looked at
      const float wm = fm * inv, wo = fo * inv;
      auto mix = [&](uint32_t a, float b) {
        if constexpr (SPLIT == 1) return __uint_as_float(a) * inv;
        return __uint_as_float(a & km) * wm + __uint_as_float(__float_as_uint(b) & ko) * wo;
      };
#pragma unroll
      for (int c = 0; c < W; c += 32) {
        uint32_t o[32];
        tmem_ld32(o_at + c, o);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 ya = y[SPLIT == 2 ? c / 4 + 2 * j : 0], yb = y[SPLIT == 2 ? c / 4 + 2 * j + 1 : 0];
          uint4 v;
          v.x = pack2(mix(o[8 * j], ya.x), mix(o[8 * j + 1], ya.y));
          v.y = pack2(mix(o[8 * j + 2], ya.z), mix(o[8 * j + 3], ya.w));
          v.z = pack2(mix(o[8 * j + 4], yb.x), mix(o[8 * j + 5], yb.y));
          v.w = pack2(mix(o[8 * j + 6], yb.z), mix(o[8 * j + 7], yb.w));
          *reinterpret_cast<uint4*>(place(lane, c / 8 + j)) = v;
        }
      }
      if (alone) {
#pragma unroll 1
        for (int c = 0; c < W; c += 32) {
          float ml[2] = {m, l}, x[32];
          for (int e = 0; e < 32; ++e) x[e] = 0.f;
          see_alone<HD>(p, b, h, kvh, r, ml, half * W + c, x);
          for (int e = 0; e < 32; ++e) reinterpret_cast<__nv_bfloat16*>(place(lane, (c + e) / 8))[e & 7] = f_to_bf16(x[e] * inv);
        }
      }
      __syncwarp();
      __nv_bfloat16* const dst = p.o + (size_t)b * p.o_bs + (size_t)h * HD + half * W + (lane % CH) * 8;
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int rw = i * (32 / CH) + lane / CH;
        if (q * 32 + rw < rows_valid)
          *reinterpret_cast<uint4*>(dst + (size_t)(q0 + q * 32 + rw) * p.o_rs) = *reinterpret_cast<const uint4*>(place(rw, lane % CH));
      }
    }
    tc_fence_before();
    __syncwarp();
  } else if constexpr (SPLIT == 2) {
    cluster_arrive();
  }
  if constexpr (SPLIT == 2) cluster_wait();   // neither half leaves while the other still reads
  __syncthreads();                            // nor frees its TMEM before its own warps have read
  if (warp == 2) {
    tc_fence_after();
    tmem_free<1>(tmem, kCols);
  }
}

template <int HD, int SPLIT>
int launch_tc(const TcPrefillAttn& a, cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(attn_tc_kernel<HD, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<HD>::smem);
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
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)a.Hq * SPLIT, (unsigned)((a.S + kTBM - 1) / kTBM), (unsigned)a.B);
  cfg.blockDim = dim3(kTThreads);
  cfg.dynamicSmemBytes = TcCfg<HD>::smem;
  cfg.stream = st;
  // Behind another launch's end the blocks find some SMs still busy and the longest ones pair up on the others: where two CTAs an SM hold the whole
  // grid and the chains are long, that costs more than the launch (16 heads of 128 over 2 048 rows 40.3 against 37.9 µs; four sequences of 14
  // heads of 64 over 333 rows, six tiles, 10.0 against 12.1; 32 heads of 128 over 2 048 rows, two rounds, 48.2 against 54).
  const int64_t blocks = (int64_t)a.B * a.Hq * ((a.S + kTBM - 1) / kTBM);
  p.pdl = a.pdl && (SPLIT == 2 || blocks <= 148 || blocks > 296 || keys < 16 * kTBN);
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = p.pdl;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = SPLIT == 2 ? 2 : 1;
  g_launches.fetch_add(1);
  B200_CUDA(cudaLaunchKernelEx(&cfg, attn_tc_kernel<HD, SPLIT>, tq, tk, tv, p));
  return B200_OK;
}

}  // namespace

bool prefill_attn_tc_ok(const TcPrefillAttn& a, int hd) {
  return (hd == 64 || hd == 128) && (a.S + kTBM - 1) / kTBM < 65536 && a.B < 65536 && aligned16(a.o, a.q, a.k, a.v) && a.q_rs % 8 == 0 &&
         a.q_bs % 8 == 0 && a.kv_rs % 8 == 0 && a.kv_bs % 8 == 0 && a.o_rs % 8 == 0 && a.o_bs % 8 == 0;
}
// Whether this kernel beats the mma.sync one: where the longest block walks enough tiles of 64 keys, or a few of them in more blocks than that one
// runs at once.  µs here / there: 16 heads of 128, one sequence 192 rows (three tiles) 8.5 / 7.3, 256 rows 8.5 / 8.6, 320 rows (five)
// 9.3 / 10.0, two sequences 11.9 / 11.2, four 12.9 / 14.2; four sequences of 32 heads 128 rows (256 blocks of 64) 8.1 / 8.2, 160 rows
// (384) 10.0 / 12.1, of 24 heads 160 rows (288) 9.9 / 9.8, 256 rows (384) 12.3 / 15.5; 14 heads of 64, one, two and four sequences: 320 rows (five)
// 7.4 / 7.1, 8.9 / 7.3, 9.8 / 9.5, 333 rows (six) 7.4 / 7.8, 8.9 / 9.0, 10.1 / 12.1.
bool prefill_attn_tc_wins(const TcPrefillAttn& a, int hd, int rows) {
  const int last = (rows - 1) / 64 * 64;   // first row of the last block
  const int edge = a.window > 0 ? std::max(0, last - a.window + 1) / 64 : 0;
  const int tiles = last / 64 + 1 - edge + (a.window > 0 ? std::min(edge, (a.keep_first + 63) / 64) : 0);
  return tiles >= (hd == 64 ? 6 : 5) || (hd == 128 && tiles >= 3 && (int64_t)a.B * a.Hq * (last / 64 + 1) > 296);
}
// Two CTAs per 128 rows of a head while all of them still run at once (two to an SM; a constant, since the two forms sum in other orders): the longest chain of tiles is half as long.  Beyond that the
// second CTA's start and end cost more than the chain.  µs, one / two: 16 heads of 128 512 rows 12.9 / 10.6, 1 024 rows (128 blocks)
// 20.5 / 15.7, 1 536 rows (192) 27.2 / 27.0, 2 048 rows 34.6 / 35.5; 32 heads 512 rows (128) 13.4 / 12.7, 768 rows (192) 17.7 / 22.0; a single
// tile or two of them per block 5.7 / 7.4.
static bool attn_tc_halves(const TcPrefillAttn& a, int rows) {
  return rows > kTBM && (int64_t)a.B * a.Hq * ((rows + kTBM - 1) / kTBM) <= 148;
}
int launch_prefill_attn_tc(const TcPrefillAttn& a, int hd, int rows, cudaStream_t st) {
  const bool two = attn_tc_halves(a, rows);
  if (hd == 64) return two ? launch_tc<64, 2>(a, st) : launch_tc<64, 1>(a, st);
  return two ? launch_tc<128, 2>(a, st) : launch_tc<128, 1>(a, st);
}

}  // namespace b200
