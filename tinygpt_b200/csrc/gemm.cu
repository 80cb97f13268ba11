// gemm.cu — the batched PREFILL GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), sm_100a only.
//
//   C[M,N] = bf16( A[M,K] · B[N,K]ᵀ )      A = activations of M prompt tokens, B = Linear.weight [out,in] (K-contiguous)
//
// Replaces, for m > 1, op::matmul → cublasGemmStridedBatchedEx / cublasGemmEx
//   [ref: third_party/TinyTorch/src/Operation/OpLinalg.cpp:244-277, OpLinalgCuda.cuh:193-216,276-293]
// with the reference's numerics: bf16 × bf16 products, fp32 accumulation, ONE rounding to bf16; what the reference does in a kernel
// of its own behind a Linear keeps its own rounding when it rides on the store.  Decode (m = 1) never comes
// here — it is HBM-bound and runs on the CUDA-core GEMV (gemv.cu).
//
// Two kernels, chosen per shape (pick_gemm): persistent CTA pairs on 256 × 256 tiles when the tiles fill the GPU, clusters that may
// split K when they do not.  The engines' products never split: a row's sum has one order whatever M is.  In both (warp-specialised, 192 threads
// or 320):
//   warp 0   TMA producer: 64-column k-blocks of A and B (128-byte swizzle) into a shared-memory ring, completion on `full[s]`
//   warp 1   MMA issuer: one thread issues 4 × tcgen05.mma.kind::f16 (K16) per k-block, accumulator in TMEM; tcgen05.commit
//            releases the stage to the producer (`empty[s]`) and signals the epilogue (`tmem_full`).  It looks at the next stage's barrier
//            before it issues, and builds half descriptors: with a wait in every k-block and whole descriptors the issuer, not the products, set the
//            pace.  µs, 2 048 rows: 3 072 × 8 192 85 → 75 (with 192-column
//            tiles), 16 384 × 3 072 137 → 133, 12 288 × 2 048 76 → 70.5; 17 × 2 048 × 6 144 on one-CTA tiles 27 → 23
//   the other warps: epilogue, tcgen05.ld 32x32b (each warp owns the TMEM lane quarter warp_id % 4)
// TMA zero-fills out-of-range rows/columns, so M, N, K need not be multiples of the tile.  Every wait is bounded: one that gives up
// leaves a code in the host-visible word of wait_word() and lets the kernel end.
#include "ops.cuh"
#include "tc.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

namespace b200 {

namespace {

constexpr int kBK = 64;                          // bf16 per k-block: 128 bytes = one swizzle row
constexpr int kGemmThreads = 192;
constexpr int kTileBytes = 128 * kBK * 2;        // 16 KB: 128 rows of an operand's k-block
constexpr unsigned kGemmWaitCode = 0x6e000000u;

// what the epilogue does with the fp32 sums
enum GemmEpi : int {
  GEPI_STORE = 0,      // C = T(acc + bias) (fp32 bias, may be null)
  GEPI_RESIDUAL = 1,   // C = bf16(add + bf16(acc)); add [M, N] may be C itself: a linear followed by the residual's add
  GEPI_BIAS = 2,       // C = bf16(bf16(acc) + add), add [N]: a linear followed by its bias as the second rounding
  GEPI_ACCUM = 4,      // C += mult·acc (fp32 C): a layer-stack model's residual stream
  GEPI_LOGITS = 5,     // C = cap·tanh(acc / cap) (mult = cap; 0: acc itself); fp32 C: and c2 = bf16(C)
  GEPI_SILU = 3,       // B holds N gate rows, then N up rows: C = bf16(bf16(silu(bf16 gate)) · bf16 up)
};
template <typename OT>
struct GemmArgs {
  OT* C;
  const float* bias;
  const __nv_bfloat16* add;
  int M, N, K;
  unsigned* err;
  float mult = 0.f;
  __nv_bfloat16* c2 = nullptr;
  // 1: launched beside the end of the kernel in front, whose end it waits for; 2: the same, and B are weights that no kernel writes: the first ring
  // of their tiles is asked for ahead of the wait
  int pdl = 0;
};
__device__ __forceinline__ float cap_logit(float v, float cap) { return cap > 0.f ? cap * tanhf(v / cap) : v; }

// bf16(silu(bf16 g))·bf16 u of two fp32 sums each
__device__ __forceinline__ uint32_t silu_mul2(uint32_t g0, uint32_t g1, uint32_t u0, uint32_t u1) {
  return silu_mul_bf16x2(pack2(__uint_as_float(g0), __uint_as_float(g1)), pack2(__uint_as_float(u0), __uint_as_float(u1)));
}

// ------------------------------------------------------------------------------------------- persistent CTA pairs
// One tcgen05.mma.cta_group::2 covers a 256 × bn tile (M256 K16, bn = 256, 224 or 192): CTA r of the pair holds rows 128·r of A and half of
// B's rows, so per 64-wide k-block an SM loads 32 KB at most where two one-CTA 128 × 256 tiles take 48 KB each.  Persistent pairs (grid =
// min(tiles, #SMs / 2) pairs) walk tiles m-fastest, so pairs that run side by side share weight rows in L2; the fp32
// accumulator is double-buffered in TMEM (256 columns apart): the epilogue of tile i drains one buffer while the MMA warp
// fills the other.  Eight epilogue warps, two to a quarter of the rows, turn rows of TMEM lanes into whole 128-byte row pieces through a swizzled
// 4 KB patch per warp and store 16 bytes per lane along the row (four of them took 13 µs for SiLU products of a 256 × 256 tile, as long as
// K = 2 048).  Bound by the tensor pipe under the power cap (busy 87 % of the active cycles, at 224 and 192 columns).
// The width is what wastes least in the last round of tiles, any
// width sums the same bits: 2 048 × 3 072 × 8 192 is 96 tiles of 256 (two rounds of 74 pairs, 83.6 µs) or 128 of 192 (75.0),
// 2 048 × 12 288 × 2 048 384 (six rounds, 73.1) or 440 of 224 (six, 70.4), 2 048 × 16 400 × 2 048 520 (eight, 95.9) or 592 of 224 (92.7).
constexpr int kPairBN = 256;
constexpr int kPairStages = 6;
constexpr int kPairStageBytes = 2 * kTileBytes;
constexpr int kPairPatch = 4096;   // 32 rows × 128 bytes per epilogue warp
constexpr int kPairEpiWarps = 8, kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr int kPairSmem = kPairStages * kPairStageBytes + kPairEpiWarps * kPairPatch + 1024 /*align*/ + 256 /*barriers*/;

template <typename OT, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmArgs<OT> p, const int bn) {
  constexpr int BN = kPairBN, ST = kPairStages;     // BN: columns from one accumulator to the next
  const int HB = bn / 2;
  const int OUT = EPI == GEPI_SILU ? HB : bn;       // output columns of a tile
  const uint32_t idesc = umma_idesc(256, bn);
  constexpr int kCols = 2 * BN;                     // TMEM: two accumulators
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;                               // [stages][128 × 64 bf16]
  uint8_t* sB = smem + ST * kTileBytes;             // [stages][128 × 64 bf16]
  uint8_t* patch = smem + ST * kPairStageBytes;     // [8 warps][32 rows × 128 bytes]
  uint64_t* full = reinterpret_cast<uint64_t*>(patch + kPairEpiWarps * kPairPatch);   // CTA 0's count the pair's bytes
  uint64_t* empty = full + ST;
  uint64_t* tmem_full = empty + ST;                 // [2]
  uint64_t* tmem_empty = tmem_full + 2;             // [2], CTA 0's: one arrival per epilogue warp of the pair
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank(), pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
  const int mt = (p.M + 255) / 256, nt = (p.N + OUT - 1) / OUT;
  const int tiles = mt * nt;
  const int kblocks = (p.K + kBK - 1) / kBK;
  bool ok = true;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 2 * kPairEpiWarps);
    }
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc<2>(tmem_slot, kCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the pair's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto first_row = [&](int t) { return (t / mt) * OUT + rank * (EPI == GEPI_SILU ? p.N : HB); };   // of this CTA's half of B
  auto load_b = [&](int s, uint32_t bar, int n0, int kb) {
    if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * (kTileBytes + HB * kBK * 2));
    tma_load_2d_pair(sB + s * kTileBytes, &tmap_b, kb * kBK, n0, bar);
  };
  const int early = p.pdl == 2 && pair < tiles ? min(ST, kblocks) : 0;   // k-blocks of the first tile whose weights go ahead
  if (threadIdx.x == 0)
    for (int s = 0; s < early; ++s) load_b(s, mapa_u32(smem_u32(&full[s]), 0), first_row(pair), s);
  if (p.pdl) {
    pdl_wait();
    pdl_trigger();   // behind the wait: what starts beside this product finds all that lies before it done
  }

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 1;
      for (int t = pair; t < tiles && ok; t += pairs) {
        const int m0 = (t % mt) * 256 + rank * 128, n0 = first_row(t), ahead = t == pair ? early : 0;
        for (int kb = 0; kb < kblocks; ++kb) {
          const uint32_t bar = mapa_u32(smem_u32(&full[s]), 0);
          if (kb >= ahead) {
            if (!(ok = mbar_wait_limited(&empty[s], ph, p.err, kGemmWaitCode | 1))) break;
            load_b(s, bar, n0, kb);
          }
          tma_load_2d_pair(sA + s * kTileBytes, &tmap_a, kb * kBK, m0, bar);
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (!ok) drain_async();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------ MMA issuer (CTA 0)
    if (rank == 0 && elect_one()) {
      const uint32_t a0 = desc_lo(smem_u32(sA)), b0 = desc_lo(smem_u32(sB));
      int s = 0;
      uint32_t ph = 0;
      int i = 0;
      bool ready = false;   // of the next stage, looked at before the products of this one go out
      for (int t = pair; t < tiles && ok; t += pairs, ++i) {
        const int acc = i & 1;
        if (!(ok = mbar_wait_limited(&tmem_empty[acc], (uint32_t)(((i >> 1) & 1) ^ 1), p.err, kGemmWaitCode | 2))) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!ready && !(ok = mbar_wait_limited(&full[s], ph, p.err, kGemmWaitCode | 3))) break;
          tc_fence_after();
          const uint32_t a = a0 + s * (kTileBytes >> 4), b = b0 + s * (kTileBytes >> 4);
          uint64_t* const done = &empty[s];
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
          ready = mbar_test(&full[s], ph);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) umma_lo<2>(tmem_d, a + 2 * k, b + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(done);
        }
        if (ok) umma_commit_pair(&tmem_full[acc]);
      }
      if (!ok) drain_async();
    }
  } else {
    // ---------------------------------------------------------------------------------------------- epilogue
    constexpr int CW = 128 / (int)sizeof(OT);       // columns of a patch row
    constexpr int VW = 16 / (int)sizeof(OT);        // columns per lane when the patch is read back
    const int q = warp & 3, grp = (warp - 2) >> 2;  // two warps share a quarter of the lanes and take its column chunks in turn
    uint8_t* const pw = patch + (warp - 2) * kPairPatch;
    const int rr = lane >> 3, cc = lane & 7;        // read-back: lane takes 16-byte piece cc of rows rr, rr + 4, …
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    int i = 0;
    for (int t = pair; t < tiles; t += pairs, ++i) {
      const int acc = i & 1;
      const int row0 = (t % mt) * 256 + rank * 128 + q * 32, n0 = (t / mt) * OUT;
      ok = __all_sync(0xffffffffu, mbar_wait_limited(&tmem_full[acc], (uint32_t)((i >> 1) & 1), p.err, kGemmWaitCode | 4));
      if (!ok) break;
      tc_fence_after();
      const int n_end = min(p.N, n0 + OUT);
#pragma unroll 1
      for (int c = grp * CW; c < OUT; c += 2 * CW) {   // at least one chunk a warp (OUT is 96 and more); of a last chunk that reaches past the tile, what lies there is not stored
        if constexpr (EPI == GEPI_SILU) {           // 64 columns: gate at c, up at HB + c
          uint32_t g[32], u[32];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            tmem_ld32(lane_base + (uint32_t)(acc * BN + c + 32 * h), g);
            tmem_ld32(lane_base + (uint32_t)(acc * BN + HB + c + 32 * h), u);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 o;
              o.x = silu_mul2(g[8 * j], g[8 * j + 1], u[8 * j], u[8 * j + 1]);
              o.y = silu_mul2(g[8 * j + 2], g[8 * j + 3], u[8 * j + 2], u[8 * j + 3]);
              o.z = silu_mul2(g[8 * j + 4], g[8 * j + 5], u[8 * j + 4], u[8 * j + 5]);
              o.w = silu_mul2(g[8 * j + 6], g[8 * j + 7], u[8 * j + 6], u[8 * j + 7]);
              *reinterpret_cast<uint4*>(pw + lane * 128 + (((4 * h + j) ^ (lane & 7)) << 4)) = o;
            }
          }
        } else if constexpr (sizeof(OT) == 2) {
          uint32_t a[32], b[32];
          tmem_ld32(lane_base + (uint32_t)(acc * BN + c), a);
          tmem_ld32(lane_base + (uint32_t)(acc * BN + c + 32), b);
          tmem_wait_ld();
          if (EPI == GEPI_STORE && p.bias != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (n0 + c + j < p.N) a[j] = __float_as_uint(__uint_as_float(a[j]) + p.bias[n0 + c + j]);
              if (n0 + c + 32 + j < p.N) b[j] = __float_as_uint(__uint_as_float(b[j]) + p.bias[n0 + c + 32 + j]);
            }
          }
          if (EPI == GEPI_LOGITS && p.mult > 0.f) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              a[j] = __float_as_uint(cap_logit(__uint_as_float(a[j]), p.mult));
              b[j] = __float_as_uint(cap_logit(__uint_as_float(b[j]), p.mult));
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* v = j < 4 ? a + 8 * j : b + 8 * (j - 4);
            uint4 o;
            o.x = pack2(__uint_as_float(v[0]), __uint_as_float(v[1]));
            o.y = pack2(__uint_as_float(v[2]), __uint_as_float(v[3]));
            o.z = pack2(__uint_as_float(v[4]), __uint_as_float(v[5]));
            o.w = pack2(__uint_as_float(v[6]), __uint_as_float(v[7]));
            *reinterpret_cast<uint4*>(pw + lane * 128 + ((j ^ (lane & 7)) << 4)) = o;
          }
        } else {
          uint32_t a[32];
          tmem_ld32(lane_base + (uint32_t)(acc * BN + c), a);
          tmem_wait_ld();
          if (p.bias != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (n0 + c + j < p.N) a[j] = __float_as_uint(__uint_as_float(a[j]) + p.bias[n0 + c + j]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(pw + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]);
        }
        if (c + 2 * CW >= OUT) {   // this warp holds the tile's last columns: the accumulator may be filled again
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
        }
        __syncwarp();
        const int col = n0 + c + cc * VW;
        if (col < n_end) {     // N and the tile are multiples of 8: a 16-byte piece lies inside the row or outside it
          uint4 add[8];
          if constexpr (EPI == GEPI_RESIDUAL) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (row0 + rr + 4 * k < p.M) add[k] = *reinterpret_cast<const uint4*>(p.add + (size_t)(row0 + rr + 4 * k) * p.N + col);
          } else if constexpr (EPI == GEPI_ACCUM) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (row0 + rr + 4 * k < p.M) add[k] = *reinterpret_cast<const uint4*>(p.C + (size_t)(row0 + rr + 4 * k) * p.N + col);
          } else if constexpr (EPI == GEPI_BIAS) {
            add[0] = *reinterpret_cast<const uint4*>(p.add + col);
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r = rr + 4 * k;
            if (row0 + r >= p.M) continue;
            uint4 v = *reinterpret_cast<const uint4*>(pw + r * 128 + ((cc ^ (r & 7)) << 4));
            if constexpr (EPI == GEPI_ACCUM || (EPI == GEPI_LOGITS && sizeof(OT) == 4)) {
              uint32_t* f = reinterpret_cast<uint32_t*>(&v);
              const uint32_t* o = reinterpret_cast<const uint32_t*>(&add[EPI == GEPI_ACCUM ? k : 0]);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                f[j] = __float_as_uint(EPI == GEPI_ACCUM ? fmaf(p.mult, __uint_as_float(f[j]), __uint_as_float(o[j])) : cap_logit(__uint_as_float(f[j]), p.mult));
              if constexpr (EPI == GEPI_LOGITS)
                *reinterpret_cast<uint2*>(p.c2 + (size_t)(row0 + r) * p.N + col) =
                    make_uint2(pack2(__uint_as_float(f[0]), __uint_as_float(f[1])), pack2(__uint_as_float(f[2]), __uint_as_float(f[3])));
            }
            if constexpr (EPI == GEPI_RESIDUAL || EPI == GEPI_BIAS) {
              const uint4 w = add[EPI == GEPI_BIAS ? 0 : k];
              v = make_uint4(add_bf16x2(w.x, v.x), add_bf16x2(w.y, v.y), add_bf16x2(w.z, v.z), add_bf16x2(w.w, v.w));
            }
            *reinterpret_cast<uint4*>(p.C + (size_t)(row0 + r) * p.N + col) = v;
          }
        }
        __syncwarp();          // the patch is free again
      }
    }
  }

  tc_fence_before();
  __syncwarp();
  __syncthreads();
  cluster_sync_all();   // neither CTA still reads the pair's operands, barriers or accumulators
  if (warp == 2) {
    tc_fence_after();
    tmem_free<2>(tmem_base, kCols);
  }
  cluster_sync_all();
}

// -------------------------------------------------------------------------------------- one tile per CTA; split-K clusters
// The kernel for shapes with fewer tiles than the persistent pairs need: short prompts, and the o_proj / down_proj of
// middling ones.  A rows past M are neither loaded nor stored (box of ≤ 128 rows; what the MMA reads there only reaches rows that
// nobody reads).  The forms:
//   kWhole      one CTA, 128 × 128, the whole K; each epilogue thread takes a row from TMEM to global memory, 16 bytes at a time, and
//               a residual's row is on its way while the products run.  As a cluster of one, through shared memory, a tile took 1.5 to 3 µs longer
//               (µs: 37 × 2 048 × 2 048 15.1, now 13.5; 1 024 × 10 944 × 2 048 83, now 71).
//   kWide       the same with 256 columns: half the tiles, for row counts at which pairs of 256 rows leave a second round to a few of them
//   kHalf, kNarrow   the same with 64 and 32 columns: short prompts of a narrow model, whose 128-column tiles would leave all of W to a few SMs
//   kSplit      a cluster per 128 × 128 tile, for operators whose whole-K tiles would leave most SMs idle while the few busy ones stream
//               all of W: `splits` CTAs take neighbouring ranges of K, leave their fp32 partial tiles in their own shared memory
//               (the drained operand ring), and after one cluster barrier each sums its share of the rows over all partials
//               through distributed shared memory, in rank order, and stores it.  No workspace, no second launch, no atomics.
//   kSplitPair  the same with 256 × 256 tiles on CTA pairs; one split is a pair's plain tile.
enum GemmForm : int { kWhole = 0, kSplit = 1, kSplitPair = 2, kWide = 3, kHalf = 4, kNarrow = 5 };
constexpr int form_columns(int form) { return form == kSplitPair || form == kWide ? 256 : form == kHalf ? 64 : form == kNarrow ? 32 : 128; }

// The ring holds as many stages as 192 KB take: six of 128 rows of A, ten of 16 rows and fewer; up to fourteen of the narrow forms.
constexpr int kSplitRing = 192 * 1024;
constexpr int kSplitStagesMax = 14;
constexpr int kSplitSmem = kSplitRing + 1024 /*align*/ + 256 /*barriers*/;
static_assert(128 * (256 + 4) * 4 <= kSplitRing, "a partial tile fits in the drained ring");
__host__ __device__ constexpr int split_stages(int box_rows, int b_bytes) {   // the MMA reads 128 rows (16 KB) from the last stage's A on
  const int fit = (kSplitRing - kTileBytes + box_rows * kBK * 2) / (box_rows * kBK * 2 + b_bytes), most = b_bytes < kTileBytes ? kSplitStagesMax : 10;
  return fit < most ? fit : most;
}
constexpr bool split_ring_holds(int b_bytes) {
  for (int r = 8; r <= 128; r += 8)
    if (split_stages(r, b_bytes) * b_bytes + (split_stages(r, b_bytes) - 1) * r * kBK * 2 + kTileBytes > kSplitRing) return false;
  return true;
}
static_assert(split_ring_holds(kTileBytes / 4) && split_ring_holds(kTileBytes / 2) && split_ring_holds(kTileBytes) && split_ring_holds(2 * kTileBytes), "what the MMA reads stays inside the ring");

template <typename OT, int EPI, int FORM>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmArgs<OT> p,
                  const int splits, const int box_rows) {
  constexpr bool PAIR = FORM == kSplitPair, STRAIGHT = FORM != kSplit && FORM != kSplitPair;
  constexpr int BN = form_columns(FORM), BMT = PAIR ? 256 : 128, LD = BN + 4, GROUP = PAIR ? 2 : 1;
  constexpr int B_BYTES = BN / GROUP * kBK * 2;   // of a k-block, per CTA
  constexpr int OUT = EPI == GEPI_SILU ? BN / 2 : BN;
  constexpr uint32_t kIdesc = umma_idesc(BMT, BN);
  static_assert(BN >= 128 || EPI != GEPI_SILU, "an epilogue thread reads 32 gate and 32 up columns");
  static_assert(STRAIGHT || (sizeof(OT) == 2 && (EPI == GEPI_STORE || EPI == GEPI_BIAS)), "what operators ask for");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int stages = split_stages(box_rows, B_BYTES), a_bytes = box_rows * kBK * 2;
  uint8_t* sB = smem;                                       // [stages][BN / GROUP × 64 bf16], one box or (SiLU) two
  uint8_t* sA = smem + stages * B_BYTES;                    // [stages][box_rows × 64 bf16]
  float* part = reinterpret_cast<float*>(smem);             // [128][LD] once the ring has drained
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kSplitRing);
  uint64_t* empty = full + kSplitStagesMax;
  uint64_t* tmem_full = empty + kSplitStagesMax;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
  int* gave_up = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int crank = (int)cluster_rank(), half = PAIR ? crank & 1 : 0, split = PAIR ? crank >> 1 : crank;
  const int tile = (int)blockIdx.x / (splits * GROUP);
  const int n0 = tile * OUT, m0 = (int)blockIdx.y * BMT + half * 128;
  const int kblocks = (p.K + kBK - 1) / kBK;
  const int kb0 = (int)((int64_t)kblocks * split / splits), kb1 = (int)((int64_t)kblocks * (split + 1) / splits);
  const int valid = max(0, min(128, p.M - m0));             // rows of this CTA that exist
  bool ok = true;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tmem_full, 1);
    *gave_up = 0;
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc<GROUP>(tmem_slot, BN);
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // the pair's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto load_b = [&](int s, int kb) {
    const uint32_t bytes = (uint32_t)(a_bytes + B_BYTES) * (uint32_t)GROUP;
    const int b0 = n0 + half * 128;   // SiLU: gate rows, and the up rows that belong to them
    uint8_t* const b_dst = sB + s * B_BYTES;
    if constexpr (PAIR) {
      if (half == 0) mbar_arrive_expect_tx(&full[s], bytes);
      tma_load_2d_pair(b_dst, &tmap_b, kb * kBK, b0, mapa_u32(smem_u32(&full[s]), (uint32_t)(crank & ~1)));
    } else {
      mbar_arrive_expect_tx(&full[s], bytes);
      tma_load_2d(b_dst, &tmap_b, kb * kBK, b0, &full[s]);
      if constexpr (EPI == GEPI_SILU) tma_load_2d(b_dst + B_BYTES / 2, &tmap_b, kb * kBK, n0 + p.N, &full[s]);
    }
  };
  const int early = p.pdl == 2 ? min(stages, kb1 - kb0) : 0;   // k-blocks whose weights go ahead
  if (threadIdx.x == 0)
    for (int s = 0; s < early; ++s) load_b(s, kb0 + s);
  if (p.pdl) {
    pdl_wait();
    pdl_trigger();   // behind the wait: what starts beside this product finds all that lies before it done
  }

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 1;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (kb - kb0 >= early) {
          if (!(ok = mbar_wait_limited(&empty[s], ph, p.err, kGemmWaitCode | 5))) break;
          load_b(s, kb);
        }
        uint8_t* const a_dst = sA + s * a_bytes;
        if constexpr (PAIR) tma_load_2d_pair(a_dst, &tmap_a, kb * kBK, m0, mapa_u32(smem_u32(&full[s]), (uint32_t)(crank & ~1)));
        else tma_load_2d(a_dst, &tmap_a, kb * kBK, m0, &full[s]);
        if (++s == stages) {
          s = 0;
          ph ^= 1;
        }
      }
      if (!ok) drain_async();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------------- MMA issuer
    if (half == 0 && elect_one()) {
      const uint32_t a0 = desc_lo(smem_u32(sA)), b0 = desc_lo(smem_u32(sB));
      int s = 0;
      uint32_t ph = 0;
      bool ready = false;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!ready && !(ok = mbar_wait_limited(&full[s], ph, p.err, kGemmWaitCode | 6))) break;
        tc_fence_after();
        const uint32_t a = a0 + s * (uint32_t)(a_bytes >> 4), b = b0 + s * (B_BYTES >> 4);
        uint64_t* const done = &empty[s];
        if (++s == stages) {
          s = 0;
          ph ^= 1;
        }
        ready = mbar_test(&full[s], ph);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k)   // 16 bf16 = 32 bytes further along K inside the 128-byte swizzle row
          umma_lo<GROUP>(tmem_base, a + 2 * k, b + 2 * k, kIdesc, (kb > kb0 || k > 0) ? 1u : 0u);
        if constexpr (PAIR) umma_commit_pair(done, (uint16_t)(3u << crank));
        else umma_commit(done);
      }
      if (ok) {
        if constexpr (PAIR) umma_commit_pair(tmem_full, (uint16_t)(3u << crank));
        else umma_commit(tmem_full);
      } else {
        drain_async();
      }
    }
  } else if constexpr (STRAIGHT) {
    // ---------------------------------------------------------------------------------------------- epilogue, a row per thread
    const int q = warp & 3, row = q * 32 + lane;
    const bool mine = row < valid;
    const size_t o0 = (size_t)(m0 + (mine ? row : 0)) * p.N + n0;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    uint4 res[EPI == GEPI_RESIDUAL ? OUT / 8 : 1];
    if constexpr (EPI == GEPI_RESIDUAL) {
#pragma unroll
      for (int j = 0; j < OUT / 8; ++j)
        if (mine && n0 + 8 * j < p.N) res[j] = *reinterpret_cast<const uint4*>(p.add + o0 + 8 * j);
    }
    ok = __all_sync(0xffffffffu, mbar_wait_limited(tmem_full, 0, p.err, kGemmWaitCode | 7));
    if (ok && q * 32 < valid) {
      tc_fence_after();
#pragma unroll(EPI == GEPI_RESIDUAL ? OUT / 32 : 1)
      for (int c = 0; c < OUT; c += 32) {
        uint32_t r[32], u[32];
        float4 old[8];
        tmem_ld32(lane_base + (uint32_t)c, r);
        if constexpr (EPI == GEPI_SILU) tmem_ld32(lane_base + (uint32_t)(OUT + c), u);   // the up columns of these gate columns
        if constexpr (EPI == GEPI_ACCUM) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (mine && n0 + c + 4 * j < p.N) old[j] = *reinterpret_cast<const float4*>(p.C + o0 + c + 4 * j);
        }
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 4; ++j) {      // N is a multiple of 8: eight columns lie inside the row or outside it
          const int col = n0 + c + 8 * j;
          if (!mine || col >= p.N) continue;
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * j + e]);
          if (EPI == GEPI_STORE && p.bias != nullptr) {
            float b[8];
            if ((reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
              reinterpret_cast<float4*>(b)[0] = reinterpret_cast<const float4*>(p.bias + col)[0];
              reinterpret_cast<float4*>(b)[1] = reinterpret_cast<const float4*>(p.bias + col)[1];
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) b[e] = p.bias[col + e];
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] += b[e];
          }
          if constexpr (EPI == GEPI_ACCUM) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = fmaf(p.mult, v[e], reinterpret_cast<const float*>(old)[8 * j + e]);
          }
          OT* const dst = p.C + o0 + c + 8 * j;
          if constexpr (EPI == GEPI_LOGITS) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = cap_logit(v[e], p.mult);
            if constexpr (sizeof(OT) == 4) *reinterpret_cast<uint4*>(p.c2 + o0 + c + 8 * j) = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
          }
          if constexpr (sizeof(OT) == 4) {
            reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
            reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
          } else {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if constexpr (EPI == GEPI_SILU) w[e] = silu_mul2(r[8 * j + 2 * e], r[8 * j + 2 * e + 1], u[8 * j + 2 * e], u[8 * j + 2 * e + 1]);
              else w[e] = pack2(v[2 * e], v[2 * e + 1]);
            }
            if constexpr (EPI == GEPI_RESIDUAL || EPI == GEPI_BIAS) {
              uint4 a;
              if constexpr (EPI == GEPI_RESIDUAL) a = res[c / 8 + j];
              else a = *reinterpret_cast<const uint4*>(p.add + col);
              w[0] = add_bf16x2(a.x, w[0]); w[1] = add_bf16x2(a.y, w[1]); w[2] = add_bf16x2(a.z, w[2]); w[3] = add_bf16x2(a.w, w[3]);
            }
            *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------------- the partial tile, into shared memory
    const int q = warp & 3, row = q * 32 + lane;
    ok = __all_sync(0xffffffffu, mbar_wait_limited(tmem_full, 0, p.err, kGemmWaitCode | 7));
    if (ok && q * 32 < valid) {
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c, r);
        tmem_wait_ld();
        if (row < valid) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(part + row * LD + c + 4 * j) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        }
      }
    }
  }
  if (!STRAIGHT && !ok) *gave_up = 1;
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if constexpr (!STRAIGHT) {
    cluster_sync_all();   // every partial of the tile is in place

    // -------------------------------------------------------------------------------- sum, epilogue, store: 8 columns at a time
    const int share = (valid + splits - 1) / splits, r_lo = split * share, r_hi = min(valid, r_lo + share);
    const uint32_t part_u = smem_u32(part);
    constexpr int G = OUT / 8;
    int lost = 0;   // a split that gave up has no part: nothing is stored then
#pragma unroll 4
    for (int sp = 0; sp < splits; ++sp) lost |= ld_cluster_i32(mapa_u32(smem_u32(gave_up), (uint32_t)(PAIR ? 2 * sp + half : sp)));
    for (int it = threadIdx.x; it < (r_hi - r_lo) * G; it += kGemmThreads) {
      const int r = r_lo + it / G, c = (it % G) * 8, col = n0 + c;
      if (col >= p.N) continue;              // N is a multiple of 8: a piece lies inside the row or outside it
      uint4 add = make_uint4(0, 0, 0, 0);
      if constexpr (EPI == GEPI_BIAS) add = *reinterpret_cast<const uint4*>(p.add + col);
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll 4
      for (int sp = 0; sp < splits; ++sp) {
        const uint32_t base = mapa_u32(part_u + (uint32_t)(r * LD + c) * 4u, (uint32_t)(PAIR ? 2 * sp + half : sp));
        const float4 x = ld_cluster_f4(base), y = ld_cluster_f4(base + 16);
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
      }
      if (lost) break;
      uint4 w = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
      if constexpr (EPI == GEPI_BIAS) w = make_uint4(add_bf16x2(add.x, w.x), add_bf16x2(add.y, w.y), add_bf16x2(add.z, w.z), add_bf16x2(add.w, w.w));
      *reinterpret_cast<uint4*>(p.C + (size_t)(m0 + r) * p.N + col) = w;
    }
    __syncthreads();
    cluster_sync_all();   // no CTA leaves while another still reads its partial
  }
  if (warp == 2) {
    tc_fence_after();
    tmem_free<GROUP>(tmem_base, BN);
  }
  if constexpr (PAIR) cluster_sync_all();
}

int make_tmap(CUtensorMap* out, const void* base, int64_t rows, int64_t cols, int box_rows) {
  return make_tmap_sw128(out, 2, base, 1, rows, cols, rows * cols, cols, box_rows);
}

// SM pairs of the current device (0 on error)
int sm_pairs() {
  static std::atomic<int> known{0};
  int n = known.load(std::memory_order_relaxed);
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    n /= 2;
    known.store(n, std::memory_order_relaxed);
  }
  return n;
}

template <typename OT, int EPI>
int launch_pair(const GemmArgs<OT>& args, const void* A, const void* B, int64_t rows_b, int bn, cudaStream_t st) {
  static PerDevice attrs;
  B200_CUDA(attrs([] { return cudaFuncSetAttribute(gemm_pair_kernel<OT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem); }));
  GemmArgs<OT> p = args;
  int rc;
  if ((rc = wait_word(&p.err)) != B200_OK) return rc;
  CUtensorMap ta, tb;
  if ((rc = make_tmap(&ta, A, p.M, p.K, 128)) != B200_OK) return rc;
  if ((rc = make_tmap(&tb, B, rows_b, p.K, bn / 2)) != B200_OK) return rc;
  const int OUT = EPI == GEPI_SILU ? bn / 2 : bn;
  const int64_t tiles = (int64_t)((p.M + 255) / 256) * ((p.N + OUT - 1) / OUT);
  const int pairs = sm_pairs();
  B200_CHECK_ARG(pairs > 0 && tiles < (1ll << 30), "gemm: no device, or shape out of range");
  B200_CUDA(launch_pdl(gemm_pair_kernel<OT, EPI>, dim3((unsigned)(2 * std::min<int64_t>(tiles, pairs))), dim3(kPairThreads), kPairSmem, st, p.pdl != 0, ta, tb, p, bn));
  return B200_OK;
}

template <typename OT, int EPI, int FORM>
int split_setup() {
  static PerDevice attrs;
  B200_CUDA(attrs([] { return cudaFuncSetAttribute(gemm_split_kernel<OT, EPI, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem); }));
  return B200_OK;
}

struct ClusterLaunch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  ClusterLaunch(dim3 grid, unsigned cluster, cudaStream_t st, bool pdl = false) {
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kSplitSmem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = cluster > 1 ? attr : attr + 1;
    cfg.numAttrs = (cluster > 1 ? 1 : 0) + (pdl ? 1 : 0);
  }
};

// CTAs of clusters of `n` ≤ 8 CTAs that the GPU holds at a time
template <int FORM>
int split_capacity(int n) {
  static std::atomic<int> known[9];
  const int c = known[n].load(std::memory_order_relaxed);
  if (c != 0) return c;
  ClusterLaunch l(dim3((unsigned)n, 64), (unsigned)n, nullptr);
  int clusters = 0;
  if (split_setup<__nv_bfloat16, GEPI_STORE, FORM>() != B200_OK ||
      cudaOccupancyMaxActiveClusters(&clusters, gemm_split_kernel<__nv_bfloat16, GEPI_STORE, FORM>, &l.cfg) != cudaSuccess || clusters < 1) {
    (void)cudaGetLastError();
    clusters = std::max(1, 2 * sm_pairs() / n);
  }
  known[n].store(clusters * n, std::memory_order_relaxed);
  return clusters * n;
}

template <typename OT, int EPI, int FORM>
int launch_split(const GemmArgs<OT>& args, const void* A, const void* B, int64_t rows_b, int splits, cudaStream_t st) {
  GemmArgs<OT> p = args;
  int rc;
  if ((rc = split_setup<OT, EPI, FORM>()) != B200_OK || (rc = wait_word(&p.err)) != B200_OK) return rc;
  constexpr int W = FORM == kSplitPair ? 2 : 1, BN = form_columns(FORM), OUT = BN / (EPI == GEPI_SILU ? 2 : 1);
  const int box_rows = (int)std::min<int64_t>(128, ((int64_t)p.M + 7) / 8 * 8);
  CUtensorMap ta, tb;
  if ((rc = make_tmap(&ta, A, p.M, p.K, box_rows)) != B200_OK) return rc;
  if ((rc = make_tmap(&tb, B, rows_b, p.K, EPI == GEPI_SILU ? BN / 2 : BN / W)) != B200_OK) return rc;
  ClusterLaunch l(dim3((unsigned)((p.N + OUT - 1) / OUT * splits * W), (unsigned)((p.M + 128 * W - 1) / (128 * W))), (unsigned)(splits * W), st, p.pdl != 0);
  g_launches.fetch_add(1);
  B200_CUDA(cudaLaunchKernelEx(&l.cfg, gemm_split_kernel<OT, EPI, FORM>, ta, tb, (const GemmArgs<OT>)p, splits, box_rows));
  return B200_OK;
}

constexpr int kSplitMinKb = 8;   // k-blocks that a split takes at least: shorter ones save less than their sum costs

// Which kernel, by what each would take (µs): rounds of resident tiles × (k-blocks × the time of one + what a tile costs
// besides).  The constants are fits to graph-timed launches over M = 17 … 2 048 and the (N, K) of the four model
// configurations: a k-block is 0.205 µs on a 128 × 128 tile, 0.33 µs on a 128 × 256 one, 0.25 µs on a pair's, which grows to 0.39 µs when
// every SM runs several tiles (power, L2); the rest is launch, pipeline fill and epilogue.  Measured, µs, M × N × K, one-CTA tiles / wide ones /
// pairs / splits: 40 × 2 048 × 6 144 23.2 / 34.0 / 26.9 / 11.0; 128 × 16 384 × 3 072 22.3 / 27.3 / 24.7; 300 × 12 288 × 2 048, where 96 tiles are
// two rounds of pairs and 288 two of single CTAs, but 144 wide ones a single round, 26.2 / 22.1 / 23.6; 2 048 × 2 048 × 2 048 21.6 / 16.2 / 17.0;
// 2 048 × 12 288 × 2 048 123 / 108 / 71.  Narrower tiles are as many k-blocks long, and a k-block of theirs takes hardly less (0.2 µs, what the issuing
// thread needs), but their results leave sooner and weights come through more SMs: 128 / 64 / 32 columns, 60 × 896 × 896 6.7 / 6.2 / 6.1, 128 × 896 × 896
// 8.0 / 6.8 / 6.3, 300 × 1 152 × 896 7.9 / 6.8 / 6.2, 300 × 896 × 4 864 20.3 / 19.0 / 18.3, 128 × 4 096 × 4 096 18.4 / 17.4 / 17.2, 512 × 2 048 × 2 048 10.9 /
// 10.3 / 18.2 (two rounds).  B200_GEMM = "persistent" (with a width: "persistent192") | "tile" | "wide" | "half" | "narrow" forces the
// persistent pairs or one whole-K tile of 128, 256, 64 or 32 columns per CTA (SiLU pairs have none of the last two).  The products of a prompt pass (no split) find their weights in HBM and their epilogue
// is not hidden when a pair has one tile: 5 µs on top of the fit, so pairs start later there (ms a prompt, tiles / pairs / the choice: 24 layers,
// 896 wide, 60 rows 1.76 / 2.31 / 1.75, 300 rows 2.15 / 2.67 / 2.05; 28 layers, 2 048 wide, 500 rows 3.68 / 4.03 / 3.59, 1 000 rows 5.62 / 4.84 / 4.56).
struct GemmPick {
  int kind;     // 0: a CTA per tile (and split); 1: a pair per tile (and split); 2: persistent pairs; 3, 4, 5: a CTA per tile of 256, 64, 32 columns
  int splits;
  int bn;       // kind 2: columns of a tile
};
// Without SPLIT the order in which a row's products are summed is the same whatever M is, so a prompt's rows have the same bits in one
// pass, in portions and in a batch.
template <typename OT, int EPI, bool SPLIT>
void pick_gemm(int64_t M, int64_t N, int64_t K, GemmPick* out) {
  constexpr int D = EPI == GEPI_SILU ? 2 : 1;
  const int64_t kb = (K + kBK - 1) / kBK;
  const int pairs = std::max(1, sm_pairs());
  auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
  double best = 1e30;
  auto consider = [&](int kind, int splits, double cost, int bn = 0) {
    if (cost < best) {
      best = cost;
      *out = GemmPick{kind, splits, bn};
    }
  };
  // rows of tiles run over grid.y: up to 65 535 of them, 8.4 M rows; the persistent pairs take any number
  const bool fits = up(M, 128) <= 65535;
  const double f32_us = sizeof(OT) == 4 ? 2.5 : 0.0;   // 128 columns of fp32 results, a row per thread (2 049 × 2 048 × 2 048 logits: wide 24.9, pairs 22.1)
  const char* env = std::getenv("B200_GEMM");   // looked up once: routed experts' products wait for the host
  const char forced = env != nullptr ? env[0] : 0;
  const bool slim = fits && EPI != GEPI_SILU && (forced == 'h' || forced == 'n');
  const bool tile = fits && forced == 't', wide = fits && forced == 'w', any_split = fits && !wide && forced != 'p';
  if (wide) consider(3, 1, 0.0);
  if (slim) consider(forced == 'h' ? 4 : 5, 1, -1.0);
  if (!tile) {
    int only = forced == 'p' ? std::atoi(env + std::strcspn(env, "0123456789")) : 0;   // "persistent224": that width
    if (only != kPairBN && only != 224 && only != 192) only = 0;                       // one that is not built: any
    for (int bn = kPairBN; bn >= 192; bn -= 32) {
      if (only != 0 && bn != only) continue;
      const int64_t t = up(M, 256) * up(N, bn / D), rounds = up(t, pairs);
      const double block = 0.25 + 0.10 * std::min(1.0, (double)t / 64.0) + 0.02 * (double)std::min<int64_t>(rounds - 1, 2);
      const double tile_us = (double)kb * block * std::max(0.79, (double)bn / kPairBN);
      const double epilogue = EPI == GEPI_SILU ? 6.5 * bn / kPairBN : 0.0;   // longer than a short k range
      consider(2, 1, (SPLIT ? 5.2 : 10.5) + (double)rounds * std::max(tile_us, epilogue) + epilogue, bn);
    }
  }
  if (any_split && !tile) {
    const int64_t t = up(M, 128) * up(N, 256 / D);
    const double rows = (double)std::min<int64_t>(M, 128) / 128.0;
    consider(3, 1, (double)up(t, 2 * pairs) * (4.0 + 2.2 * rows + (t >= 100 ? 0.42 : 0.33) * (double)kb + (EPI == GEPI_SILU ? 2.0 : f32_us * 2)));
  }
  if (any_split && !tile && EPI != GEPI_SILU) {
    const double rows = (double)std::min<int64_t>(M, 128) / 128.0;
    consider(4, 1, (double)up(up(M, 128) * up(N, 64), 2 * pairs) * (3.3 + 0.7 * rows + 0.2 * (double)kb + f32_us / 2));
    consider(5, 1, (double)up(up(M, 128) * up(N, 32), 2 * pairs) * (3.25 + 0.25 * rows + 0.2 * (double)kb + f32_us / 4));
  }
  if (any_split) {
    const double rows = (double)std::min<int64_t>(M, 128) / 128.0;
    for (int s = 1; s <= (SPLIT && !tile ? 8 : 1) && (s == 1 || s * kSplitMinKb <= kb); ++s) {
      const int64_t t = up(M, 128) * up(N, 128 / D) * s;
      if (s == 1) consider(0, s, (double)up(t, 2 * pairs) * (3.6 + rows * 1.4 + 0.205 * (double)kb + (EPI == GEPI_SILU ? 1.5 : f32_us)));
      else if constexpr (SPLIT)
        consider(0, s, (double)up(t, split_capacity<kSplit>(s)) * (5.0 + 0.15 * s + rows * (2.0 + 0.25 * s) + 0.23 * (double)up(kb, s)));
    }
    if constexpr (SPLIT) {
      for (int s = 1; s <= 4 && (s == 1 || s * kSplitMinKb <= kb) && M > 128 && !tile; ++s) {
        const int64_t t = up(M, 256) * up(N, 256) * 2 * s;
        consider(1, s, (double)up(t, split_capacity<kSplitPair>(2 * s)) * (9.5 + 1.0 * s + 0.30 * (double)up(kb, s)));
      }
    }
  }
}

template <typename OT, int EPI, bool SPLIT = false>
int launch_gemm(const GemmArgs<OT>& args, const void* A, const void* B, int64_t rows_b, cudaStream_t st) {
  GemmArgs<OT> p = args;
  // A prompt pass: B are the model's weights, and the pass's first launch waits for all that was written before it.  Prompts of 9 / 60 / 300 rows
  // with the first weights behind → ahead of the wait: 0.5B 1.250 → 1.168 / 1.301 → 1.229 / 1.631 → 1.606 ms, 1.7B
  // 1.953 → 1.865 / 1.992 → 1.945 / 2.530 → 2.477 ms; 2 048 rows the same.
  if (pdl_scope()) p.pdl = 2;
  GemmPick g{};
  pick_gemm<OT, EPI, SPLIT>(p.M, p.N, p.K, &g);
  if (g.kind == 3) return launch_split<OT, EPI, kWide>(p, A, B, rows_b, 1, st);
  if constexpr (EPI != GEPI_SILU) {
    if (g.kind == 4) return launch_split<OT, EPI, kHalf>(p, A, B, rows_b, 1, st);
    if (g.kind == 5) return launch_split<OT, EPI, kNarrow>(p, A, B, rows_b, 1, st);
  }
  if (g.kind == 0 && g.splits == 1) return launch_split<OT, EPI, kWhole>(p, A, B, rows_b, 1, st);
  if constexpr (SPLIT) {
    if (g.kind == 0) return launch_split<OT, EPI, kSplit>(p, A, B, rows_b, g.splits, st);
    if (g.kind == 1) return launch_split<OT, EPI, kSplitPair>(p, A, B, rows_b, g.splits, st);
  }
  return launch_pair<OT, EPI>(p, A, B, rows_b, g.bn, st);
}

int check_gemm(const void* C, const void* A, const void* B, int64_t M, int64_t N, int64_t K) {
  B200_CHECK_ARG(C && A && B && M > 0 && N > 0 && K > 0, "gemm: bad arguments");
  B200_CHECK_ARG(K % 8 == 0 && N % 8 == 0, "gemm: K=%lld and N=%lld must be multiples of 8 (16-byte rows)", (long long)K,
                 (long long)N);
  B200_CHECK_ARG(aligned16(A, B, C), "gemm: operands must be 16-byte aligned");
  B200_CHECK_ARG(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "gemm: shape out of range");
  return B200_OK;
}

template <typename OT>
int launch_gemm_store(OT* C, const void* A, const void* B, const float* bias, int64_t M, int64_t N, int64_t K, cudaStream_t st) {
  int rc = check_gemm(C, A, B, M, N, K);
  if (rc != B200_OK) return rc;
  return launch_gemm<OT, GEPI_STORE>(GemmArgs<OT>{C, bias, nullptr, (int)M, (int)N, (int)K, nullptr}, A, B, N, st);
}

}  // namespace

int launch_gemm_bf16(void* C, const void* A, const void* B, int64_t M, int64_t N, int64_t K, cudaStream_t st) {
  return launch_gemm_store<__nv_bfloat16>((__nv_bfloat16*)C, A, B, nullptr, M, N, K, st);
}
int launch_gemm_bf16_bias(void* C, const void* A, const void* B, const float* bias, int64_t M, int64_t N, int64_t K, cudaStream_t st) {
  return launch_gemm_store<__nv_bfloat16>((__nv_bfloat16*)C, A, B, bias, M, N, K, st);
}
int launch_linear_bf16(void* C, const void* A, const void* B, int64_t M, int64_t N, int64_t K, LinearTail tail, const void* add, cudaStream_t st) {
  int rc = check_gemm(C, A, B, M, N, K);
  if (rc != B200_OK) return rc;
  B200_CHECK_ARG((tail == LinearTail::bias || tail == LinearTail::residual) == (add != nullptr) && aligned16(add), "linear: bad operand of the tail");
  const GemmArgs<__nv_bfloat16> p{(__nv_bfloat16*)C, nullptr, (const __nv_bfloat16*)add, (int)M, (int)N, (int)K, nullptr};
  switch (tail) {
    case LinearTail::bias: return launch_gemm<__nv_bfloat16, GEPI_BIAS>(p, A, B, N, st);
    case LinearTail::residual: return launch_gemm<__nv_bfloat16, GEPI_RESIDUAL>(p, A, B, N, st);
    case LinearTail::silu_mul: return launch_gemm<__nv_bfloat16, GEPI_SILU>(p, A, B, 2 * N, st);
    case LinearTail::none: break;
  }
  return launch_gemm<__nv_bfloat16, GEPI_STORE>(p, A, B, N, st);
}
int launch_linear_split_bf16(void* C, const void* A, const void* B, int64_t M, int64_t N, int64_t K, const void* bias, cudaStream_t st) {
  int rc = check_gemm(C, A, B, M, N, K);
  if (rc != B200_OK) return rc;
  B200_CHECK_ARG(aligned16(bias), "linear: bias must be 16-byte aligned");
  GemmArgs<__nv_bfloat16> p{(__nv_bfloat16*)C, nullptr, (const __nv_bfloat16*)bias, (int)M, (int)N, (int)K, nullptr};
  p.pdl = op_pdl(st);
  return bias != nullptr ? launch_gemm<__nv_bfloat16, GEPI_BIAS, true>(p, A, B, N, st) : launch_gemm<__nv_bfloat16, GEPI_STORE, true>(p, A, B, N, st);
}
int launch_gemm_bf16_f32(float* C, const void* A, const void* B, const float* bias, int64_t M, int64_t N, int64_t K, cudaStream_t st) {
  return launch_gemm_store<float>(C, A, B, bias, M, N, K, st);
}

int launch_gemm_bf16_accum(float* C, const void* A, const void* B, float mult, int64_t M, int64_t N, int64_t K, cudaStream_t st) {
  int rc = check_gemm(C, A, B, M, N, K);
  if (rc != B200_OK) return rc;
  return launch_gemm<float, GEPI_ACCUM>(GemmArgs<float>{C, nullptr, nullptr, (int)M, (int)N, (int)K, nullptr, mult}, A, B, N, st);
}
int launch_gemm_bf16_logits(float* C, void* C_bf16, const void* A, const void* B, float softcap, int64_t M, int64_t N, int64_t K,
                            cudaStream_t st) {
  int rc = check_gemm(C_bf16, A, B, M, N, K);
  if (rc != B200_OK) return rc;
  if (C == nullptr)
    return launch_gemm<__nv_bfloat16, GEPI_LOGITS>(GemmArgs<__nv_bfloat16>{(__nv_bfloat16*)C_bf16, nullptr, nullptr, (int)M, (int)N, (int)K, nullptr, softcap},
                                                   A, B, N, st);
  B200_CHECK_ARG(aligned16(C), "gemm: bad fp32 logits");
  return launch_gemm<float, GEPI_LOGITS>(GemmArgs<float>{C, nullptr, nullptr, (int)M, (int)N, (int)K, nullptr, softcap, (__nv_bfloat16*)C_bf16}, A,
                                         B, N, st);
}

}  // namespace b200

extern "C" int b200_gemm_bf16(void* C, const void* A, const void* B, int64_t M, int64_t N, int64_t K, void* stream) {
  int rc = b200::op_check();
  if (rc != B200_OK) return rc;
  return b200::launch_linear_split_bf16(C, A, B, M, N, K, nullptr, (cudaStream_t)stream);
}
