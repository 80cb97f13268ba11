// prefill_attn_tc.cu — causal flash attention of a PREFILL chunk on the 5th-generation tensor cores (tcgen05, TMEM, TMA) for head
// sizes 64 and 128, sm_100a.  Same arithmetic as prefill_attn.cu (bf16 Q·Kᵀ products summed in fp32, base-2 online softmax in
// fp32, P rounded to bf16, bf16 P·V products summed in fp32), same masks (causal over a cached prefix, sliding window with
// kept first keys), sink and per-head gate.
//
// Shape of the work: blocks of 128 query rows of a head, long ones first, shared out over one CTA per SM that runs through several; a block visits its keys
// in tiles of 128 in ascending order.  TMEM holds three S and one O of 128 columns:
//   warps 0-7    softmax, two groups of four warps, which take the tiles by the parity of their place in the cache (so that a row's sums are the same
//                however its prompt is cut); one row per thread: S from TMEM, row maximum and sum without shuffles, P (bf16) back into the TMEM columns of S
//                as the A operand of P·V.  Both groups' P go into the same O, so each hands its running maximum on to the other, with the tile's
//                number, through shared memory
//   warps 8-11   rescale O where a row's maximum grew, beside the exponentials; at a block's end they normalise and store (TMA), while the
//                groups are at the next block
//   warp 12      TMA producer: Q blocks, K and V tiles (128-byte swizzle; rows past the sequence are zero-filled)
//   warp 13      MMA issuer (one thread): P·V of a tile and right behind it S of the tile three further on, also across blocks
//
// A key that a row does not see has P = 0, and 0 · V is 0 only for finite V.  So where a result is not finite, V of the tiles that some row of the
// block sees in part is looked at, and if it holds infinities or NaNs those rows go over the keys that they see, one after another, behind the CTA's last
// block: what a row does not see never reaches it.
//
// Bound by the chain S → softmax → P·V of three tiles in flight: a group takes some 2 400 cycles a tile (1 024 of them the exponentials' pipe) and 800 until it
// begins the next one; tensor pipe and exponentials 40 % of the active cycles at 16 heads of 128 over 2 048 rows.  Small calls by what is done once: barriers, TMEM,
// first loads, code that is not in the caches yet, results (some 5 µs in all; up to 128 keys a kernel of its own, below, takes less).  Slower, at 16 heads of
// 128 over 2 048 rows, were two O of which each group has one (26 µs where this form takes 21.5: S, whose columns P shares, then waits for P·V), three groups
// of softmax warps (28), tiles read twice from TMEM in loops (23), the exponentials ahead of the maximum (22), 64-key tiles in two CTAs per SM (36).  A
// maximum that moves only where weights grow beyond 2^8 needs hardly a rescale (20.5), but the largest weight is then no longer 1, and rounded: 5 % more
// error against 64 bits, not taken.
// µs, mma.sync / 64-key tiles in two CTAs per SM / here: 16 heads of 128 over 2 048 rows 63 / 36.2 / 21.5, 24 heads 99 / 42.3 / 32.6, 32 heads
// 123 / 47.8 / 38.8; 16 heads over 512 rows 15.4 / 9.2 / 9.1, 1 024 rows 33.6 / 16.3 / 13.1; four sequences of 32 heads, 512 rows 43 / 26.2 / 19.9; 14 heads
// of 64 over 2 048 rows 56 / 30.6 / 18.5, four sequences of 333 rows 11.9 / 9.7 / 7.5.  Errors against 64 bits within 1 % of each other.
#include "ops.cuh"
#include "tc.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kTBM = 128, kTBN = 128, kTThreads = 512;
constexpr unsigned kAttnWaitCode = 0xa7000000u;

// n / d for n below 2³¹ (Granlund and Montgomery 1994)
struct Div {
  uint32_t m, s1, s2;
  Div() = default;
  explicit Div(uint32_t d) {
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;
    m = (uint32_t)(((1ull << 32) * ((1ull << l) - d)) / d + 1);
    s1 = l < 1 ? l : 1;
    s2 = l < 1 ? 0 : l - 1;
  }
  __device__ __forceinline__ int operator()(int n) const {
    const uint32_t t = __umulhi(m, (uint32_t)n);
    return (int)((t + (((uint32_t)n - t) >> s1)) >> s2);
  }
};

struct TcAttn {
  __nv_bfloat16* o;
  const __nv_bfloat16* gate;
  int64_t o_rs, o_bs, q_rs, q_bs;
  int S, Hq, p0;
  float scale_log2;
  int window, keep_first, sink;
  unsigned* err;
  int pdl;
  int blocks, heads, last;             // blocks of 128 rows in all; heads of all sequences; the last block of a head
  Div by_heads, by_hq, by_group;       // by heads, by Hq, by Hq / Hkv
  const __nv_bfloat16 *qp, *kp, *vp;   // see_alone
  int64_t kv_rs, kv_bs;
};

template <int HD>
struct TcCfg {
  static constexpr int NB = HD / 64;                 // 64-column blocks of a row (one swizzle atom wide)
  static constexpr int KST = HD == 64 ? 4 : 2, VST = HD == 64 ? 4 : 3;   // K and V stages
  static constexpr int TB = NB * 128 * 128;          // 128 rows of Q, K or V
  static constexpr int stage = 128 * 128;            // 64 columns of results of 128 rows
  static constexpr int small = 384 /*barriers*/ + 4 * 1024 /*m_row*/ + 2 * 2 * 1024 /*ml*/;
  static constexpr int smem_one = 3 * TB + 64 /*barriers*/ + 1024 /*align*/;
  static constexpr int smem = (1 + KST + VST) * TB + stage + small + 1024 /*align*/;
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
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* smem_src, int32_t c0, int32_t c1, int32_t c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }   // this thread's copies have left shared memory
__device__ __forceinline__ void bulk_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }        // and lie in global memory
// D[tmem] (+)= A[tmem]·B[smem], B's descriptor by its lower half: the address and, from bit 16 on, the distance of 64-column blocks of an operand
// whose N runs along the columns (V's [keys][64 columns] rows of 128 bytes, MN-major)
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}" ::"r"(d), "r"(a), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15])
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
// what has been loaded may be read behind this, and not before
template <int N>
__device__ __forceinline__ void tmem_loaded(uint32_t (&r)[N]) {
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
// waits for some 20 µs at most without taking issue slots from the warps that work
__device__ __forceinline__ bool mbar_sleep(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(20000u) : "memory");
  return ok != 0;
}
// A wait that gave up says so to the whole CTA and sets `dead`: its role goes on without waiting (what follows neither hangs nor leaves
// the buffers), and nothing is stored.  The first look is inline and has no loop around it.
__device__ __forceinline__ bool wait_slow(uint64_t* bar, uint32_t parity, unsigned* err, unsigned code, volatile int* gave_up) {
  const unsigned long long t0 = global_timer_ns();
  while (!mbar_sleep(bar, parity)) {
    if (global_timer_ns() - t0 > 2000000000ull) {
      *reinterpret_cast<volatile unsigned*>(err) = code;
      *gave_up = 1;
      __threadfence_system();
      return true;
    }
  }
  return false;
}
__device__ __forceinline__ uint32_t bits_below(int n) { return n >= 32 ? ~0u : n <= 0 ? 0u : (1u << n) - 1; }

__device__ __forceinline__ float max3f(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
// A row's maximum and the number of the tile that it is from (as a float's bits), which says whether it is there: one access of 64 bits, so that no reader sees
// a new number beside an old maximum (a vector access may be carried out element by element).
__device__ __forceinline__ float2 ld_max(const float2* p) {
  float2 v;
  asm volatile("{\n\t.reg .b64 t;\n\tld.volatile.shared.b64 t, [%2];\n\tmov.b64 {%0, %1}, t;\n\t}" : "=f"(v.x), "=f"(v.y) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_max(float2* p, float2 v) {
  asm volatile("{\n\t.reg .b64 t;\n\tmov.b64 t, {%1, %2};\n\tst.volatile.shared.b64 [%0], t;\n\t}" ::"r"(smem_u32(p)), "f"(v.x), "f"(v.y) : "memory");
}
constexpr int kTCtas = 148;   // one per SM; which CTA has a block changes no bit

// What a block of 128 query rows of a head has to visit: tiles of 128 keys in ascending order
struct Block {
  int b, h, kvh, q0, rows_valid, first_pos, last_pos, n_keep, t_lo, n;
  __device__ __forceinline__ Block(const TcAttn& p, int i) {
    const int late = p.by_heads(i), hb = i - late * p.heads;
    b = p.by_hq(hb);
    h = hb - b * p.Hq;
    kvh = p.by_group(h);
    q0 = (p.last - late) * kTBM;   // late blocks (most keys) first
    rows_valid = min(kTBM, p.S - q0);
    first_pos = p.p0 + q0;
    last_pos = first_pos + rows_valid - 1;
    // with a window the tiles of the kept first keys, then from the first row's window edge up to the diagonal
    t_lo = p.window > 0 ? max(0, first_pos - p.window + 1) / kTBN : 0;
    n_keep = p.window > 0 ? min(t_lo, (p.keep_first + kTBN - 1) / kTBN) : 0;
    n = n_keep + last_pos / kTBN + 1 - t_lo;
  }
  // some row does not see some key of the tile
  __device__ __forceinline__ bool in_part(const TcAttn& p, int kbase) const {
    return kbase + kTBN - 1 > first_pos || (p.window > 0 && last_pos - kbase >= p.window);
  }
  __device__ __forceinline__ int tile(int it) const { return it < n_keep ? it : t_lo + it - n_keep; }   // its place in the cache
};

// Whether V holds infinities or NaNs in a tile that some row of the block sees in part; one warp
template <int HD>
__device__ __forceinline__ bool part_not_finite(const TcAttn& p, const Block& w, int lane) {
  bool bad = false;
  for (int it = 0; it < w.n; ++it) {
    const int kbase = w.tile(it) * kTBN;
    if (!w.in_part(p, kbase)) continue;
    const __nv_bfloat16* const v = p.vp + (size_t)w.b * p.kv_bs + (size_t)kbase * p.kv_rs + (size_t)w.kvh * HD;
    const int rows = min(kTBN, p.p0 + p.S - kbase);
#pragma unroll 1
    for (int e = lane; e < rows * (HD / 8); e += 32) {
      const uint4 x4 = *reinterpret_cast<const uint4*>(v + (size_t)(e / (HD / 8)) * p.kv_rs + e % (HD / 8) * 8);
      const uint32_t x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) bad |= (((x[k] & 0x7f807f80u) + 0x00800080u) & 0x80008000u) != 0;
    }
  }
  return __any_sync(0xffffffffu, bad);
}

// The way out for such a block: this warp's 32 rows, each over the keys that it sees and no others (weights rounded to bf16 like above).  A row's scores go to
// the lanes, 32 keys at a time, its columns to the lanes, key after key.  Slow and rare: 32 rows over 300 000 keys take 1.6 s (heads of 64: 0.92 s), bound by the
// latency of loads; kept small, since a call also pays for code that it only jumps over.
template <int HD>
__device__ __forceinline__ void see_alone(const TcAttn& p, const Block& w, int quarter, int lane) {
  constexpr int E = HD / 32;   // columns of a lane
  const int end = min(w.rows_valid, quarter * 32 + 32);
#pragma unroll 1
  for (int row = quarter * 32; row < end; ++row) {
    const int r = w.q0 + row, rpos = p.p0 + r;
    const __nv_bfloat16* const q = p.qp + (size_t)w.b * p.q_bs + (size_t)r * p.q_rs + (size_t)w.h * HD;
    const size_t kv = (size_t)w.b * p.kv_bs + (size_t)w.kvh * HD;
    auto score = [&](int j, float& s) {   // whether the row sees key j; its score
      if (j > rpos || (p.window > 0 && rpos - j >= p.window && j >= p.keep_first)) return false;
      const __nv_bfloat16* const k = p.kp + kv + (size_t)j * p.kv_rs;
      s = 0.f;
#pragma unroll 2
      for (int d = 0; d < HD; d += 8) {
        float x[8];
        unpack8(*reinterpret_cast<const uint4*>(q + d), x);
        s = dot8(*reinterpret_cast<const uint4*>(k + d), x, s);
      }
      return true;
    };
    // the keys behind the kept ones and in front of the window are passed over, 32 at a time
    const int edge = p.window > 0 ? max(0, rpos - p.window + 1) & ~31 : 0, from = p.keep_first > 0 ? 0 : edge;
    float m = -INFINITY, l = 0.f, acc[E];   // the maximum so far; of this lane's keys; of its columns
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = 0.f;
#pragma unroll 1
    for (int j0 = from; j0 <= rpos; j0 = j0 + 32 >= p.keep_first && j0 + 32 < edge ? edge : j0 + 32) {
      float s = -INFINITY;
      const bool sees = score(j0 + lane, s);
      float top = fmaxf(m, s);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      if (top != m) {
        const float f = m == -INFINITY ? 1.f : ex2f((m - top) * p.scale_log2);
        l *= f;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] *= f;
        m = top;
      }
      const float weight = sees ? ex2f(fmaf(s, p.scale_log2, m == -INFINITY ? 0.f : -m * p.scale_log2)) : 0.f;
      l += weight;
      const float rounded = round_bf16(weight);
      const unsigned seen = __ballot_sync(0xffffffffu, sees);
      const __nv_bfloat16* const v = p.vp + kv + (size_t)j0 * p.kv_rs + lane * E;
      auto add = [&](int j) {
        const float x = __shfl_sync(0xffffffffu, rounded, j);
        uint32_t y[E / 2];
        if constexpr (E == 4) *reinterpret_cast<uint2*>(y) = *reinterpret_cast<const uint2*>(v + (size_t)j * p.kv_rs);
        else y[0] = *reinterpret_cast<const uint32_t*>(v + (size_t)j * p.kv_rs);
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = fmaf(x, __uint_as_float(e & 1 ? y[e / 2] & 0xffff0000u : y[e / 2] << 16), acc[e]);
      };
      if (seen == 0xffffffffu) {
#pragma unroll 8
        for (int j = 0; j < 32; ++j) add(j);
      } else {
#pragma unroll 1
        for (unsigned left = seen; left != 0; left &= left - 1) add(__ffs(left) - 1);
      }
    }
    l = warp_sum(l);
    if (p.sink && m != -INFINITY) l += ex2f(-m * p.scale_log2);
    const float gate = p.gate != nullptr ? 1.f / (1.f + expf(-bf16_to_f(p.gate[(size_t)w.b * p.q_bs + (size_t)r * p.q_rs + w.h]))) : 1.f;
    const float inv = (l > 0.f ? 1.f / l : 0.f) * gate;
    __nv_bfloat16* const o = p.o + (size_t)w.b * p.o_bs + (size_t)r * p.o_rs + (size_t)w.h * HD + lane * E;
#pragma unroll
    for (int e = 0; e < E; e += 2) *reinterpret_cast<uint32_t*>(o + e) = pack2(acc[e] * inv, acc[e + 1] * inv);
  }
}

// the weights of 32 keys of a row, rounded to bf16, to TMEM; their sums in fp32
__device__ __forceinline__ void weights32(const uint32_t (&s)[32], uint64_t scale2, uint64_t neg, uint64_t (&sum)[2], uint32_t at) {
  uint32_t pk[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const uint64_t z = fma_f2(pack_f2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), scale2, neg);
    const float a0 = ex2f(lo_f2(z)), a1 = ex2f(hi_f2(z));
    sum[e & 1] = add_f2(sum[e & 1], pack_f2(a0, a1));
    pk[e] = pack2(a0, a1);
  }
  tmem_st16(at, pk);
}

// 32 rows of a block from O in TMEM, this lane's with maximum m and sum l: normalised, through shared memory (64 columns at `mid`, the next 64 `step`
// bytes further on) into the result.  has_read is called behind the last look at O.  Whether some result is not finite, which is what 0 · V may have left
// where V is not.
template <int HD, typename F>
__device__ __forceinline__ bool store_rows(const TcAttn& p, const CUtensorMap* to, const Block& w, uint32_t o_at, int row, float m, float l, uint8_t* mid,
                                           int step, bool lost, F has_read) {
  const int lane = row & 31, rr = w.q0 + min(row, w.rows_valid - 1);
  const float k_scale = p.scale_log2;
  if (p.sink && m != -INFINITY) l += ex2f(-m * k_scale);
  const float gate = p.gate != nullptr ? 1.f / (1.f + expf(-bf16_to_f(p.gate[(size_t)w.b * p.q_bs + (size_t)rr * p.q_rs + w.h]))) : 1.f;
  const float inv = (l > 0.f ? 1.f / l : 0.f) * gate;
  uint32_t odd = 0;   // the sign bits of halves whose exponent is all ones
#pragma unroll 1
  for (int c = 0; c < HD; c += 64, mid += step) {
    if (step == 0) {
      if (lane == 0) bulk_read();   // the copy before has read
      __syncwarp();
    }
#pragma unroll 1
    for (int k = 0; k < 64; k += 32) {
      uint32_t o[32], y[16];
      tmem_ld32(o_at + c + k, o);
      tmem_loaded(o);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        y[e] = pack2(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv);
        odd |= (y[e] & 0x7f807f80u) + 0x00800080u;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)   // in the tensor map's 128-byte swizzle
        *reinterpret_cast<uint4*>(mid + lane * 128 + ((k / 8 + e) ^ (lane & 7)) * 16) = make_uint4(y[4 * e], y[4 * e + 1], y[4 * e + 2], y[4 * e + 3]);
    }
    if (c + 64 == HD) has_read();
    fence_proxy_async();
    __syncwarp();
    if (lane == 0 && !lost && row < w.rows_valid) {
      tma_store_3d(to, mid, w.h * HD + c, w.q0 + row, w.b);   // rows past the sequence are not written
      bulk_commit();
    }
  }
  return __any_sync(0xffffffffu, (odd & 0x80008000u) != 0);
}

// The same for 128 keys at most, one tile: nothing is shared out and nothing runs ahead, so four warps do everything one after another, on as many
// keys as there are (P of those behind is zero, and adding their products changes no bit).
template <int HD>
__global__ void __launch_bounds__(128)
attn_tc_one_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                   const __grid_constant__ CUtensorMap to, const __grid_constant__ TcAttn p) {
  using C = TcCfg<HD>;
  constexpr int kColO = 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sQ = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sK = sQ + C::TB;
  uint8_t* sV = sK + C::TB;
  uint64_t* qk_full = reinterpret_cast<uint64_t*>(sV + C::TB);
  uint64_t* v_full = qk_full + 1;
  uint64_t* s_full = v_full + 1;
  uint64_t* o_full = s_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  int* gave_up = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = threadIdx.x;
  bool dead = false;
  auto wait_for = [&](uint64_t* bar, unsigned code) {
    if (!mbar_try_wait(bar, 0) && !dead) dead = wait_slow(bar, 0, p.err, code, gave_up);
  };
  const Block w(p, (int)blockIdx.x);
  const int keys = p.p0 + p.S, steps = (keys + 15) / 16;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tv);
    tma_prefetch_desc(&to);
    for (int i = 0; i < 4; ++i) mbar_init(qk_full + i, 1);
    *gave_up = 0;
    fence_mbar_init();
    if (p.pdl) pdl_wait();
    mbar_arrive_expect_tx(qk_full, 2 * C::TB);
#pragma unroll
    for (int c = 0; c < C::NB; ++c) {
      tma_load_3d(sK + c * kTBN * 128, &tk, w.kvh * HD + c * 64, 0, w.b, qk_full);
      tma_load_3d(sQ + c * kTBM * 128, &tq, w.h * HD + c * 64, 0, w.b, qk_full);
    }
    mbar_arrive_expect_tx(v_full, C::TB);
#pragma unroll
    for (int c = 0; c < C::NB; ++c) tma_load_3d(sV + c * kTBN * 128, &tv, w.kvh * HD + c * 64, 0, w.b, v_full);
  }
  if (warp == 1) tmem_alloc<1>(tmem_slot, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (p.pdl) {
    pdl_wait();
    pdl_trigger();
  }
  if (warp == 0 && elect_one()) {
    const uint32_t q_u = desc_lo(smem_u32(sQ)), k_u = desc_lo(smem_u32(sK)), idesc = umma_idesc(kTBM, steps * 16);
    wait_for(qk_full, kAttnWaitCode | 17);
    tc_fence_after();
#pragma unroll
    for (int kk = 0; kk < HD / 16; ++kk) {
      const uint32_t at = ((kk / 4) * 128 * 128 + (kk % 4) * 32) >> 4;
      umma_lo<1>(tmem, q_u + at, k_u + at, idesc, kk > 0 ? 1u : 0u);
    }
    umma_commit(s_full);
  }
  __syncwarp();
  const uint32_t s_at = tmem + ((uint32_t)(warp * 32) << 16);
  const int rpos = w.first_pos + min(row, w.rows_valid - 1);   // padding rows behave like the last valid row
  const float k_scale = p.scale_log2;
  const uint64_t scale2 = pack_f2(k_scale, k_scale);
  wait_for(s_full, kAttnWaitCode | 18);
  __syncwarp();
  tc_fence_after();
  float m = -INFINITY, l = 0.f;
  {
    uint32_t s[4][32];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k * 32 < keys) tmem_ld32(s_at + k * 32, s[k]);
    tmem_wait_ld();
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k * 32 >= keys) continue;
      const int k0 = k * 32;
      const uint32_t seen = bits_below(rpos + 1 - k0) & (p.window > 0 ? ~bits_below(rpos + 1 - p.window - k0) | bits_below(p.keep_first - k0) : ~0u);
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        asm volatile("" : "+r"(s[k][e]));
        s[k][e] = seen & (1u << e) ? s[k][e] : 0xff800000u;
      }
#pragma unroll
      for (int e = 0; e < 32; e += 2) mx[e / 2 % 4] = max3f(mx[e / 2 % 4], __uint_as_float(s[k][e]), __uint_as_float(s[k][e + 1]));
    }
    m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
    const float ms = m == -INFINITY ? 0.f : m * k_scale;
    const uint64_t neg = pack_f2(-ms, -ms);
    uint64_t sum[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k * 32 >= keys) continue;
      weights32(s[k], scale2, neg, sum, s_at + k * 16);
    }
    sum[0] = add_f2(sum[0], sum[1]);
    l = lo_f2(sum[0]) + hi_f2(sum[0]);
  }
  tmem_wait_st();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0 && elect_one()) {
    const uint32_t v_u = desc_lo(smem_u32(sV));
    wait_for(v_full, kAttnWaitCode | 19);
    tc_fence_after();
    for (int kk = 0; kk < steps; ++kk)
      umma_ts(tmem + kColO, tmem + kk * 8, v_u + (kk * 2048 >> 4) + ((kTBN * 128 >> 4) << 16), umma_idesc(kTBM, HD, true), kk > 0 ? 1u : 0u);
    umma_commit(o_full);
  }
  __syncwarp();
  wait_for(o_full, kAttnWaitCode | 20);
  __syncwarp();
  tc_fence_after();
  const bool lost = __any_sync(0xffffffffu, dead || *reinterpret_cast<volatile int*>(gave_up) != 0);
  // results on their way out take Q's place: its product is over
  const bool odd = store_rows<HD>(p, &to, w, s_at + kColO, row, m, l, sQ + warp * (32 * 128), 128 * 128, lost, [&] {});
  if (__builtin_expect(odd, 0) && !lost && part_not_finite<HD>(p, w, lane)) {
    if (lane == 0) bulk_done();   // the stores that these rows write over
    __syncwarp();
    see_alone<HD>(p, w, warp, lane);
  }
  if (lane == 0) bulk_read();
  if (dead) drain_async();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_free<1>(tmem, 256);
  }
}

template <int HD>
__global__ void __launch_bounds__(kTThreads, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
               const __grid_constant__ CUtensorMap to, const __grid_constant__ TcAttn p) {
  using C = TcCfg<HD>;
  constexpr int NB = C::NB, KST = C::KST, VST = C::VST;
  constexpr uint32_t kIdescS = umma_idesc(kTBM, kTBN), kIdescO = umma_idesc(kTBM, HD, true);
  constexpr int kCols = 512, kColO = 384;   // three S, and P in them, at columns 0, 128 and 256, O behind them
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                      // [NB][128 rows × 128 bytes]
  uint8_t* sK = sQ + C::TB;                // [KST][NB][128 keys × 128 bytes]
  uint8_t* sV = sK + KST * C::TB;          // [VST]
  uint8_t* sO = sV + VST * C::TB;          // [4 warps][32 rows × 128 bytes]
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sO + C::stage);
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_empty + 1;          // [KST]
  uint64_t* k_empty = k_full + KST;
  uint64_t* v_full = k_empty + KST;        // [VST]
  uint64_t* v_empty = v_full + VST;
  uint64_t* s_full = v_empty + VST;        // [2 groups][3]: a group that has no tile for a while skips no phase of its own barriers
  uint64_t* p_full = s_full + 6;           // [3], one arrival per warp of the group that has the tile
  uint64_t* pv_done = p_full + 3;          // [3]: P has been read
  uint64_t* m_full = pv_done + 3;          // [3], one arrival per warp of the group that has the tile: its maxima are in m_row
  uint64_t* o_ready = m_full + 3;          // [3], one arrival per correcting warp: O goes by the tile's maxima
  uint64_t* o_full = o_ready + 3;          // all products of a block are over
  uint64_t* o_empty = o_full + 1;          // one arrival per storing warp: it has read O
  uint64_t* ml_full = o_empty + 1;         // [2], one arrival per softmax warp
  uint64_t* ml_empty = ml_full + 2;        // [2], one arrival per storing warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ml_empty + 2);
  int* gave_up = reinterpret_cast<int*>(tmem_slot + 1);
  float2* m_row = reinterpret_cast<float2*>(sO + C::stage + 384);   // [4][128]: a row's maximum on its way to the group with the next tile, and the
                                                                      // tile's number.  Tile c + 4 overwrites what c + 1 has read: its S comes behind P of c + 1.
  float2* ml = m_row + 4 * kTBM;               // [2][2 groups][128]: a block's maxima and sums

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool dead = false;
  auto wait_for = [&](uint64_t* bar, uint32_t parity, unsigned code) {
    if (__builtin_expect(!mbar_try_wait(bar, parity), 0) && !dead) dead = wait_slow(bar, parity, p.err, code, gave_up);
  };
  auto wait_passed = [&](const float2* at, int tile, float2& v) {   // the row's maximum behind this tile; limited like every wait
    unsigned long long t0 = 0;
    for (unsigned spins = 1; __float_as_int(v.y) != tile && !dead; ++spins) {
      v = ld_max(at);
      if ((spins & 0x3ffu) == 0) {
        const unsigned long long now = global_timer_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > 2000000000ull) {
          dead = true;
          *reinterpret_cast<volatile unsigned*>(p.err) = kAttnWaitCode | 15;
          *reinterpret_cast<volatile int*>(gave_up) = 1;
          __threadfence_system();
        }
      }
    }
    __syncwarp();
  };
  // round r's block of this CTA: forwards and backwards in turn, so that who has had a long one gets a short one
  const int grid = (int)gridDim.x, cta = (int)blockIdx.x;
  auto block_of = [&](int r) { return r * grid + (r & 1 ? grid - 1 - cta : cta); };

  auto load_q = [&](const Block& w) {
    mbar_arrive_expect_tx(q_full, C::TB);
#pragma unroll
    for (int c = 0; c < NB; ++c) tma_load_3d(sQ + c * kTBM * 128, &tq, w.h * HD + c * 64, w.q0, w.b, q_full);
  };
  auto load_k = [&](const Block& w, int key, int s) {
    mbar_arrive_expect_tx(&k_full[s], C::TB);
#pragma unroll
    for (int c = 0; c < NB; ++c) tma_load_3d(sK + s * C::TB + c * kTBN * 128, &tk, w.kvh * HD + c * 64, key, w.b, &k_full[s]);
  };
  auto load_v = [&](const Block& w, int key, int s) {
    mbar_arrive_expect_tx(&v_full[s], C::TB);
#pragma unroll
    for (int c = 0; c < NB; ++c) tma_load_3d(sV + s * C::TB + c * kTBN * 128, &tv, w.kvh * HD + c * 64, key, w.b, &v_full[s]);
  };
  if (warp == 12) {
    if (lane == 0) {
      tma_prefetch_desc(&tk);
      tma_prefetch_desc(&tq);
      tma_prefetch_desc(&tv);
      tma_prefetch_desc(&to);
      *gave_up = 0;
    }
    const int bars = (int)(ml_empty + 2 - q_full);
    for (int i = lane; i < bars; i += 32) {
      const uint64_t* const bar = q_full + i;
      mbar_init(q_full + i, bar >= p_full && bar < pv_done || bar >= m_full && bar < o_full ? 4 : bar == o_empty || bar >= ml_empty ? 4 : bar >= ml_full ? 8 : 1);
    }
    fence_mbar_init();
    __syncwarp();
    if (lane == 0) {
      const Block w(p, cta);
      if (p.pdl) pdl_wait();
      load_k(w, w.tile(0) * kTBN, 0);   // on their way while TMEM is allocated
      load_q(w);
    }
  }
  if (warp == 13) tmem_alloc<1>(tmem_slot, kCols);
  m_row[threadIdx.x] = make_float2(0.f, __int_as_float(-1));
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (p.pdl) {
    pdl_wait();
    pdl_trigger();
  }

  // Registers: 2 × 184 + 88 + 56 are the 4 × 128 that a quarter of the SM has been launched with
  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 12 && lane == 0) {
      // ---------------------------------------------------------------------------------------- TMA producer
      int ks = 1, vs = 0;          // the first K tile and the first Q have gone out
      uint32_t kph = 1, vph = 1;
      bool first = true;
      static_assert(KST > 1, "a second K stage");
      for (int r = 0, i; (i = block_of(r)) < p.blocks; ++r) {
        const Block w(p, i);
        if (r > 0) {
          wait_for(q_empty, (uint32_t)((r - 1) & 1), kAttnWaitCode | 1);
          load_q(w);
        }
        auto next_k = [&](int it) {
          if (it >= w.n) return;
          if (first) {
            first = false;
            return;
          }
          wait_for(&k_empty[ks], kph, kAttnWaitCode | 2);
          load_k(w, w.tile(it) * kTBN, ks);
          if (++ks == KST) {
            ks = 0;
            kph ^= 1;
          }
        };
        next_k(0);
        next_k(1);
        for (int it = 0; it < w.n; ++it) {
          next_k(it + 2);
          wait_for(&v_empty[vs], vph, kAttnWaitCode | 3);
          load_v(w, w.tile(it) * kTBN, vs);
          if (++vs == VST) {
            vs = 0;
            vph ^= 1;
          }
        }
      }
      if (dead) drain_async();
    } else if (warp == 13 && elect_one()) {
      // ----------------------------------------------------------------------------------------- MMA issuer
      // Two streams of products that run in the order in which they go out: P·V of a tile as soon as P is there and, right behind it, S of the tile three
      // further on, those of the next block among them, into the buffer that P has left.  What does not depend on P has been found out by then.
      const uint32_t q_u = desc_lo(smem_u32(sQ)), k_u = desc_lo(smem_u32(sK)), v_u = desc_lo(smem_u32(sV));
      int ks = 0, vs = 0, sbuf = 0, pbuf = 0, ahead = 0, sr = 0, s_it = 0, pr = 0, p_it = 0;
      uint32_t kph = 0, vph = 0, pph = 0;
      Block sw(p, cta);
      int p_n = sw.n;
      bool s_left = true, k_ok = false, v_ok = false;
      unsigned spins = 0;
      unsigned long long t0 = 0;
      for (;;) {
        if (!k_ok & s_left) k_ok = mbar_test(&k_full[ks], kph) & (s_it > 0 || mbar_test(q_full, (uint32_t)(sr & 1)));
        if (!v_ok) v_ok = mbar_test(&v_full[vs], vph) & (p_it > 0 || pr == 0 || mbar_test(o_empty, (uint32_t)((pr - 1) & 1)));
        bool do_p = false;
        if (ahead > 0) {   // with nothing else to be done the thread sleeps until P is there
          const bool sleep = v_ok & (!s_left | (k_ok & (ahead == 3)));
          do_p = sleep ? mbar_sleep(&p_full[pbuf], pph) : mbar_test(&p_full[pbuf], pph);
          if (do_p) do_p = mbar_try_wait(&o_ready[pbuf], pph) || mbar_sleep(&o_ready[pbuf], pph);
        }
        do_p &= v_ok;
        if (dead) {   // nothing is waited for any more, and nothing leaves the buffers
          do_p = ahead > 0;
          k_ok = true;
        }
        const bool do_s = s_left & k_ok & (ahead - (int)do_p < 3);
        if (!do_p & !do_s) {
          if ((++spins & 0xffu) == 0) {
            const unsigned long long now = global_timer_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > 2000000000ull && !dead) {
              dead = true;
              *reinterpret_cast<volatile unsigned*>(p.err) = kAttnWaitCode | 4;
              *reinterpret_cast<volatile int*>(gave_up) = 1;
              __threadfence_system();
            }
          }
          continue;
        }
        t0 = 0;
        tc_fence_after();
        const bool p_last = do_p && p_it + 1 == p_n;
        if (do_p) {
          const uint32_t vt = v_u + vs * (C::TB >> 4), more = p_it > 0;
#pragma unroll
          for (int kk = 0; kk < kTBN / 16; ++kk)   // 16 keys: 8 columns of P, 2 048 bytes further down V's rows
            umma_ts(tmem + kColO, tmem + pbuf * 128 + kk * 8, vt + (kk * 2048 >> 4) + ((kTBN * 128 >> 4) << 16), kIdescO, kk > 0 ? 1u : more);
          umma_commit(&pv_done[pbuf]);   // O may be rescaled while S is on
          if (p_last) umma_commit(o_full);
        }
        if (do_s) {
          const uint32_t kt = k_u + ks * (C::TB >> 4), d = tmem + sbuf * 128;
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            const uint32_t at = ((kk / 4) * 128 * 128 + (kk % 4) * 32) >> 4;
            umma_lo<1>(d, q_u + at, kt + at, kIdescS, kk > 0 ? 1u : 0u);
          }
          umma_commit(&s_full[(sw.tile(s_it) & 1) * 3 + sbuf]);
          umma_commit(&k_empty[ks]);
          if (++ks == KST) {
            ks = 0;
            kph ^= 1;
          }
          if (++sbuf == 3) sbuf = 0;
          ++ahead;
          k_ok = false;
          if (++s_it == sw.n) {
            umma_commit(q_empty);
            const int i = block_of(++sr);
            s_it = 0;
            s_left = i < p.blocks;
            if (s_left) sw = Block(p, i);
          }
        }
        if (do_p) {
          umma_commit(&v_empty[vs]);
          if (++vs == VST) {
            vs = 0;
            vph ^= 1;
          }
          if (++pbuf == 3) {
            pbuf = 0;
            pph ^= 1;
          }
          --ahead;
          ++p_it;
          v_ok = false;
          if (p_last) {
            const int i = block_of(++pr);
            if (i >= p.blocks) break;
            p_it = 0;
            p_n = Block(p, i).n;
          }
        }
      }
      if (dead) drain_async();
    }
  } else if (warp < 8) {
    // ---------------------------------------------------------------------------------------------- softmax
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    const int g = warp >> 2, q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const float k_scale = p.scale_log2;
    const uint64_t scale2 = pack_f2(k_scale, k_scale);
    int c = -1, buf = 2;   // the tile's number, its S buffer
    uint32_t s_ph = 0;
    for (int r = 0, i; (i = block_of(r)) < p.blocks; ++r) {
      const Block w(p, i);
      const int rpos = w.first_pos + min(row, w.rows_valid - 1);   // padding rows behave like the last valid row
      float held = -INFINITY;         // the maximum of the tiles before, where this group has had the last of them
      float m = -INFINITY, l = 0.f;   // of this group's tiles: the maximum that the weights were last taken against, their sum
      for (int it = 0, prev = -1; it < w.n; ++it) {
        const int tile = w.tile(it), mine = tile & 1;
        ++c;
        if (++buf == 3) buf = 0;
        const bool from_other = it > 0 && prev != g;
        prev = mine;
        if (mine != g) continue;
        const int kbase = tile * kTBN;
        const uint32_t s_at = lane_base + buf * 128;
        const bool part = w.in_part(p, kbase);
        wait_for(&s_full[g * 3 + buf], s_ph >> buf & 1, kAttnWaitCode | 10);
        s_ph ^= 1u << buf;
        __syncwarp();
        tc_fence_after();
        const float2* const from = &m_row[((c - 1) & 3) * kTBM + row];
        float2 passed = ld_max(from);
        uint32_t s[4][32];
        tmem_ld32(s_at, s[0]);
        tmem_ld32(s_at + 32, s[1]);
        // the maximum of the tiles before, from the group that had the last of them
        if (from_other) {
          if (__builtin_expect(__any_sync(0xffffffffu, __float_as_int(passed.y) != c - 1), 0)) wait_passed(from, c - 1, passed);
          held = passed.x;
        }
        tmem_loaded(s[0]);
        tmem_loaded(s[1]);
        tmem_ld32(s_at + 64, s[2]);
        tmem_ld32(s_at + 96, s[3]);
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        auto look = [&](int k) {
#pragma unroll
          for (int e = 0; e < 32; e += 2) mx[e / 2 % 4] = max3f(mx[e / 2 % 4], __uint_as_float(s[k][e]), __uint_as_float(s[k][e + 1]));
        };
        if (__builtin_expect(part, 0)) {   // the keys this row sees, a bit each (comparing them one by one took longer than a whole tile)
          tmem_loaded(s[2]);
          tmem_loaded(s[3]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int k0 = kbase + k * 32;
            const uint32_t seen = bits_below(rpos + 1 - k0) &
                                  (p.window > 0 ? ~bits_below(rpos + 1 - p.window - k0) | bits_below(p.keep_first - k0) : ~0u);
#pragma unroll
            for (int e = 0; e < 32; ++e) s[k][e] = seen & (1u << e) ? s[k][e] : 0xff800000u;
          }
          asm volatile("" ::: "memory");   // a branch, and not two selections per key of every tile
        }
        look(0);
        look(1);
        tmem_loaded(s[2]);
        tmem_loaded(s[3]);
        look(2);
        look(3);
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        const float next = fmaxf(held, top);
        st_max(&m_row[(c & 3) * kTBM + row], make_float2(next, __int_as_float(c)));
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_full[buf]);
        held = next;
        const float ms = next == -INFINITY ? 0.f : next * k_scale;
        const uint64_t neg = pack_f2(-ms, -ms);
        uint64_t sum[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < 4; ++k) weights32(s[k], scale2, neg, sum, s_at + k * 16);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[buf]);
        if (top != -INFINITY) {   // a tile of which the row sees nothing leaves its sums as they are, however its prompt is cut
          l *= m == -INFINITY ? 1.f : ex2f((m - held) * k_scale);
          m = held;
        }
        sum[0] = add_f2(sum[0], sum[1]);
        l += lo_f2(sum[0]) + hi_f2(sum[0]);
      }
      wait_for(&ml_empty[r & 1], (uint32_t)(((r >> 1) & 1) ^ 1), kAttnWaitCode | 12);
      ml[((r & 1) * 2 + g) * kTBM + row] = make_float2(m, l);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ml_full[r & 1]);
    }
  } else {
    // ----------------------------------------------------------------------------- O: rescaled, in the end normalised and stored
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t o_at = tmem + ((uint32_t)(q * 32) << 16) + kColO;
    const float k_scale = p.scale_log2;
    int c = -1, buf = 2;   // the tile's number, its S buffer
    uint32_t ph = 1;
    bool odd = false;   // in the blocks so far
    for (int r = 0, i; (i = block_of(r)) < p.blocks; ++r) {
      const Block w(p, i);
      float was = -INFINITY;
      for (int it = 0; it < w.n; ++it) {
        ++c;
        const int before = buf;
        const uint32_t before_ph = ph;
        if (++buf == 3) {
          buf = 0;
          ph ^= 1;
        }
        wait_for(&m_full[buf], ph, kAttnWaitCode | 11);
        __syncwarp();
        const float now = ld_max(&m_row[(c & 3) * kTBM + row]).x;
        if (it > 0 && __any_sync(0xffffffffu, now != was)) {
          const float alpha = now != was ? ex2f((was - now) * k_scale) : 1.f;
          const uint64_t alpha2 = pack_f2(alpha, alpha);
          wait_for(&pv_done[before], before_ph, kAttnWaitCode | 21);
          __syncwarp();
          tc_fence_after();
#pragma unroll 1
          for (int k = 0; k < HD; k += 64) {
            uint32_t o[2][32];
            tmem_ld32(o_at + k, o[0]);
            tmem_ld32(o_at + k + 32, o[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              tmem_loaded(o[i]);
#pragma unroll
              for (int e = 0; e < 32; e += 2) {
                const uint64_t y = mul_f2(pack_f2(__uint_as_float(o[i][e]), __uint_as_float(o[i][e + 1])), alpha2);
                o[i][e] = (uint32_t)y;
                o[i][e + 1] = (uint32_t)(y >> 32);
              }
              tmem_st32(o_at + k + i * 32, o[i]);
            }
          }
          tmem_wait_st();
          tc_fence_before();
        }
        was = now;
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_ready[buf]);
      }
      wait_for(&ml_full[r & 1], (uint32_t)((r >> 1) & 1), kAttnWaitCode | 13);
      __syncwarp();
      float2 part[2];
#pragma unroll
      for (int g = 0; g < 2; ++g) part[g] = ml[((r & 1) * 2 + g) * kTBM + row];
      float m = fmaxf(part[0].x, part[1].x), l = 0.f;
#pragma unroll
      for (int g = 0; g < 2; ++g)   // a group whose tiles the row does not see has no maximum and a sum of 0, or of NaN where its scores were
        l = __fadd_rn(l, part[g].x == -INFINITY ? part[g].y : __fmul_rn(part[g].y, ex2f((part[g].x - m) * k_scale)));
      wait_for(o_full, (uint32_t)(r & 1), kAttnWaitCode | 14);
      __syncwarp();
      tc_fence_after();
      const bool lost = __any_sync(0xffffffffu, dead || *reinterpret_cast<volatile int*>(gave_up) != 0);
      odd |= store_rows<HD>(p, &to, w, o_at, row, m, l, sO + q * (32 * 128), 0, lost, [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(o_empty);
      });
      if (lane == 0) mbar_arrive(&ml_empty[r & 1]);
    }
    // Rows that go over their keys one after another do so here, where nobody waits for this warp any more: over a long cache they take longer than
    // a wait lasts.  A block whose results are all finite has no such V in the tiles that are looked at, so which ones were not need not be kept.
    if (__builtin_expect(odd, 0) && !__any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(gave_up) != 0)) {
      if (lane == 0) bulk_done();   // the stores that these rows write over
      __syncwarp();
#pragma unroll 1
      for (int r = 0, i; (i = block_of(r)) < p.blocks; ++r) {
        const Block w(p, i);
        if (part_not_finite<HD>(p, w, lane)) see_alone<HD>(p, w, q, lane);
      }
    }
    if (lane == 0) bulk_read();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_free<1>(tmem, kCols);
  }
}

template <int HD>
int launch_tc(const TcPrefillAttn& a, cudaStream_t st) {
  static PerDevice attrs;
  B200_CUDA(attrs([] {
    const cudaError_t e = cudaFuncSetAttribute(attn_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<HD>::smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attn_tc_one_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<HD>::smem_one);
  }));
  TcAttn p{};
  int rc;
  if ((rc = wait_word(&p.err)) != B200_OK) return rc;
  p.o = a.o; p.gate = a.gate; p.o_rs = a.o_rs; p.o_bs = a.o_bs; p.q_rs = a.q_rs; p.q_bs = a.q_bs;
  p.S = a.S; p.Hq = a.Hq; p.p0 = a.p0;
  p.scale_log2 = a.scale_log2; p.window = a.window; p.keep_first = a.keep_first; p.sink = a.sink;
  p.qp = a.q; p.kp = a.k; p.vp = a.v; p.kv_rs = a.kv_rs; p.kv_bs = a.kv_bs;
  p.heads = a.B * a.Hq;
  p.last = (a.S - 1) / kTBM;
  p.blocks = p.heads * (p.last + 1);
  p.by_heads = Div((uint32_t)p.heads);
  p.by_hq = Div((uint32_t)a.Hq);
  p.by_group = Div((uint32_t)(a.Hq / a.Hkv));
  p.pdl = a.pdl;
  const int64_t keys = (int64_t)a.p0 + a.S;
  CUtensorMap tq, tk, tv, to;
  if ((rc = make_tmap_sw128(&tq, 3, a.q, a.B, a.S, (int64_t)a.Hq * HD, a.q_bs, a.q_rs, kTBM)) != B200_OK) return rc;
  if ((rc = make_tmap_sw128(&tk, 3, a.k, a.B, keys, (int64_t)a.Hkv * HD, a.kv_bs, a.kv_rs, kTBN)) != B200_OK) return rc;
  if ((rc = make_tmap_sw128(&tv, 3, a.v, a.B, keys, (int64_t)a.Hkv * HD, a.kv_bs, a.kv_rs, kTBN)) != B200_OK) return rc;
  if ((rc = make_tmap_sw128(&to, 3, a.o, a.B, a.S, (int64_t)a.Hq * HD, a.o_bs, a.o_rs, 32)) != B200_OK) return rc;
  if (keys <= kTBN) {
    B200_CUDA(launch_pdl(attn_tc_one_kernel<HD>, dim3((unsigned)p.blocks), dim3(128), (size_t)TcCfg<HD>::smem_one, st, p.pdl != 0, tq, tk, tv, to, p));
    return B200_OK;
  }
  B200_CUDA(launch_pdl(attn_tc_kernel<HD>, dim3((unsigned)std::min(p.blocks, kTCtas)), dim3(kTThreads), (size_t)TcCfg<HD>::smem, st, p.pdl != 0, tq, tk, tv, to, p));
  return B200_OK;
}

}  // namespace

bool prefill_attn_tc_ok(const TcPrefillAttn& a, int hd) {
  return (hd == 64 || hd == 128) && (int64_t)a.B * a.Hq * ((a.S + kTBM - 1) / kTBM) < (1ll << 31) && aligned16(a.o, a.q, a.k, a.v) && a.q_rs % 8 == 0 &&
         a.q_bs % 8 == 0 && a.kv_rs % 8 == 0 && a.kv_bs % 8 == 0 && a.o_rs % 8 == 0 && a.o_bs % 8 == 0;
}
// Whether this kernel beats the mma.sync one: where a block of 64 rows, that one's, walks enough tiles of 64 keys, or fewer in more blocks than that one
// runs at once.  µs here / there, calls back to back:
//   heads of 128  one sequence of 16: 64 rows 4.9 / 4.0, 100 rows (two tiles, 32 blocks) 5.1 / 5.1, 128 rows 5.2 / 5.4, 160 rows 6.3 / 6.4, 192 rows 6.4 / 6.8, 256 rows
//                 6.7 / 8.1; two of 32, 100 rows (128 blocks) 5.2 / 6.9
//   heads of 64   14 heads, one, two, four and eight sequences: 160 rows (three tiles) 5.3 / 4.6, 5.4 / 5.1, 6.0 / 6.5 (168 blocks), 7.6 / 7.3 (336 blocks), 192 rows
//                 5.4 / 4.9, 5.5 / 5.3, 6.1 / 6.9, 7.7 / 7.9, 200 rows (four) 5.4 / 5.3, 5.6 / 6.7, 6.1 / 8.3, 7.7 / 8.7; 32 heads, four sequences: 128 rows (256
//                 blocks) 4.9 / 6.0, 160 rows (384) 7.7 / 7.3, 192 rows 7.8 / 7.7
// In a captured graph, where nothing overlaps, short prompts lose up to 0.6 µs here (14 heads of 64 over 200 rows 6.0 / 5.4, 16 of 128 over 160 6.8 / 6.6): a call has the same bits
// either way, so the rule does not ask.
// With a window, heads of 64 stay with the other kernel where a block there walks as few tiles, of half as many keys, or where its blocks just fill the SMs and those here
// begin a second round (µs a layer of such heads, here / there: window of 64, 24 heads over 1 024 rows 42.8 / 40.0, 14 over 2 048 43.7 / 42.7, 8 over 2 048 35.0 /
// 33.9; of 64 behind 4 kept keys 14 over 2 048 46.7 / 42.9; of 100 behind 4, 384 blocks 44.0 / 44.2, 448 blocks 46.5 / 45.0,
// 512 blocks 47.1 / 50.1; of 130 behind 64, 384 blocks 44.0 / 46.1, 448 blocks 49.0 / 46.7).  From six tiles on there is hardly a
// loss: a window of 256, 448 blocks 49.5 / 49.1, 384 blocks 43.8 / 48.2.  Heads of 128, window of 16: 512 blocks 52.5 / 56.7, 128 blocks 33.5 / 34.5 and 39.9 / 38.9.
bool prefill_attn_tc_wins(const TcPrefillAttn& a, int hd, int rows) {
  auto tiles_of = [&](int n) {   // of the last block of n rows, n keys each
    const int last = (rows - 1) / n * n, edge = a.window > 0 ? std::max(0, last - a.window + 1) / n : 0;
    return last / n + 1 - edge + (a.window > 0 ? std::min(edge, (a.keep_first + n - 1) / n) : 0);
  };
  const int tiles = tiles_of(64);
  const int64_t blocks = (int64_t)a.B * a.Hq * ((rows - 1) / 64 + 1);
  if (hd == 128) return tiles >= 3 || (tiles == 2 && blocks > 74);
  const bool enough = tiles >= 4 || (tiles >= 2 && blocks > 148 && (tiles == 2 || blocks <= 296));
  return enough && (a.window == 0 || tiles >= 6 || (tiles > tiles_of(128) && (blocks <= 384 || blocks > 448)));
}
int launch_prefill_attn_tc(const TcPrefillAttn& a, int hd, cudaStream_t st) {
  return hd == 64 ? launch_tc<64>(a, st) : launch_tc<128>(a, st);
}

}  // namespace b200
