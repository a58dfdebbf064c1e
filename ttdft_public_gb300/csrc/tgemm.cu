// Dense contractions on the fifth-generation tensor cores (tcgen05.mma with
// the accumulator in tensor memory), FP32-accurate and free of accumulation
// rounding.
//
// C(m, n) = sum_k A(m, k) B(n, k) for FP32 operands stored K-contiguous
// (row-major, one row per m or n), optionally batched over z, with the K
// range cut into G groups (the Hartree expansion's terms, or the density's
// states) whose results the epilogue combines in double-FP32.
//
// Arithmetic (an Ozaki-type error-free split).  The tensor cores' FP32
// accumulation does not round to nearest: measured on the Hartree
// contraction with FP32 operands split into three BF16 terms, the products
// accumulated in one FP32 accumulator kept only ~7e-7 relative accuracy over
// a few dozen additions, as if each addition were truncated toward zero.
// Instead, every operand value v of a group (or batch) with max |v| < 2^e is
// cut into three integer slices on a common grid,
//   v 2^(8-e) = a0 + a1 2^-8 + a2 2^-16 + O(2^-17),  a_p integers, |a_p| <= 256,
// which BF16 holds exactly.  Products of slices are exact integers; the sums
// of one level L = p + q (a0b0; a0b1 + a1b0; a0b2 + a1b1 + a2b0; a1b2 + a2b1)
// stay below 2^24 for a group of up to 192 K values, so each level
// accumulates in its own tensor-memory accumulator without rounding
// (integer-valued operands come out exact); only a2b2, 2^-32 of the leading
// product, is left out.  The epilogue adds S0 + S1 2^-8 + S2 2^-16 + S3 2^-24
// without error (the levels can cancel), scales by 2^(eA + eB - 16) and sums
// the groups in double-FP32: the result carries the operands' FP32
// quantisation (2^-25 of each group's largest value) and nothing else.  The
// group maxima come from the kernels that write the operands (atomicMax on |v|).
//
// Two kernels, as in ozgemm.cu: k_tg_slice cuts each operand once into slice
// planes (4 bytes read, 6 written a value) in the order of the MMA's operands,
// per 128 rows and 16 values of K one 12 KB block; k_tg_mma multiplies planes.
// Slicing inside the GEMM repeated the work for every column tile of A and
// bound it (tensor pipe 12 %).  A's rows are taken in slabs that keep the planes
// within kPlaneBudget.
//
// k_tg_mma: persistent CTAs over output tiles of 128 x 64, 20 warps.
//  - A slice p of A meets the slices of B in one MMA (the planes of B's tile lie
//    one after the other, and so do the level accumulators): N = 192, 192 and
//    128 columns for p = 0, 1, 2, three MMAs a chunk instead of eight.
//  - Two accumulator buffers (2 x 256 tensor-memory columns), each with an
//    issuing thread (warps 1 and 3) that takes every other group: one issues
//    while the other is held up in its commits.  They are elected (elect_one).
//  - warp 0, one thread: the copies (TMA); warp 2, one thread: waits for a
//    chunk's copies in order and publishes the count;
//  - warps 4-19 (four per 32 TMEM lanes, 16 columns each): combine the levels
//    and store (one group: FP32, with the output's per-batch max |v| for the
//    next contraction) or add into double-FP32 sums in registers, stored as
//    FP64 after the last group.
// Bound: the instruction issue of the fold (about 21 FP32 instructions a value
// and group).  Measured, 64-atom sizes: last Hartree product 7.36 -> 3.4 ms with
// its slicing, last density product 14.0 -> 5.4 ms.
// Every wait is bounded; a wait that runs out sets the error word and an
// abort flag that stops every role from issuing further work.

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "ttg_internal.cuh"
#include "tgemm.cuh"
#include "tc_common.cuh"

namespace ttg {
namespace {

using namespace tc;

constexpr int TG_M = 128;                         // rows of an A tile (MMA M)
constexpr int TG_N = 64;                          // rows of a B tile
constexpr int TG_K = 16;                          // K per chunk (one MMA)
constexpr int kSlices = 3;
constexpr int kLevels = 4;
constexpr int kPlaneA = TG_M * TG_K * 2;          // 4 KB: one BF16 slice plane of 128 rows
constexpr int kPlaneB = TG_N * TG_K * 2;          // 2 KB: of a B tile
constexpr int kBlock = kSlices * kPlaneA;         // 12 KB: 128 rows, one chunk
constexpr int kStage = kBlock + kSlices * kPlaneB;   // 18 KB
constexpr int kStages = 10;
constexpr int kSmem = kStages * kStage + 1024;
constexpr int kEpiWarp0 = 4, kEpiWarps = 16;      // four warps per 32 TMEM lanes
constexpr int TG_E = TG_N / 4;                    // columns of an epilogue warp
constexpr int kThreads = (kEpiWarp0 + kEpiWarps) * 32;   // 640
constexpr int kBufCols = kLevels * TG_N;          // 256
constexpr uint32_t kTmemCols = 512;               // two buffers
constexpr int64_t kPlaneBudget = (int64_t)1 << 30;

// kind::f16: BF16 x BF16 -> FP32, A and B K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc_mma(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(TG_M >> 4) << 24);
}

struct TileSched {
  int tiles_m, tiles_n;
  __device__ void at(int64_t t, int& tm, int& tn, int& z) const {
    const int64_t per = (int64_t)tiles_m * tiles_n;
    z = (int)(t / per);
    const int64_t r = t - (int64_t)z * per;
    tm = (int)(r / tiles_n);     // n fastest: CTAs that share an A tile run together
    tn = (int)(r - (int64_t)tm * tiles_n);
  }
};

// exponent e with max |v| < 2^e (0 for an all-zero group)
__device__ __forceinline__ int grid_exp(float amax) {
  int e = 0;
  if (amax > 0.f) frexpf(amax, &e);
  return e;
}

// three integer slices of 8 values on the grid 2^(e-8): v 2^(8-e) = a0 + a1/256 + a2/65536
__device__ __forceinline__ void slice8(const float* v, float sc, uint4& p0, uint4& p1,
                                       uint4& p2) {
  uint32_t w0[4], w1[4], w2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a[2], b[2], c[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float x = v[2 * j + h] * sc;          // |x| < 256, exact (power-of-two scale)
      a[h] = rintf(x);
      const float r = (x - a[h]) * 256.f;         // exact, |r| <= 128
      b[h] = rintf(r);
      c[h] = rintf((r - b[h]) * 256.f);
    }
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(a[0], a[1]);   // integers <= 256: exact
    const __nv_bfloat162 h1 = __floats2bfloat162_rn(b[0], b[1]);
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(c[0], c[1]);
    w0[j] = *reinterpret_cast<const uint32_t*>(&h0);
    w1[j] = *reinterpret_cast<const uint32_t*>(&h1);
    w2[j] = *reinterpret_cast<const uint32_t*>(&h2);
  }
  p0 = make_uint4(w0[0], w0[1], w0[2], w0[3]);
  p1 = make_uint4(w1[0], w1[1], w1[2], w1[3]);
  p2 = make_uint4(w2[0], w2[1], w2[2], w2[3]);
}




// One operand to slice: planes of 128-row blocks from r0 on, all batches; block
// (chunk, rows, batch z) -> 12 KB at planes + ((z blocks + y) chunks + chunk).
// The slicing grid is amax[chunk / kg] (kg > 0) or amax[z].
struct TSlice {
  const float* p;
  int64_t rows, kext, ld, bstride, r0;
  const float* amax;
  int kg, blocks;
  int64_t items;              // blocks x batches x chunks
  unsigned char* planes;
};

// Both operands of a product in one launch (items of the first, then of the second).
__global__ void __launch_bounds__(256) k_tg_slice(const TSlice sa, const TSlice sb, int chunks) {
  const bool second = blockIdx.x >= sa.items;
  const TSlice& o = second ? sb : sa;
  const int64_t item = second ? blockIdx.x - sa.items : blockIdx.x;
  const int64_t yz = item / chunks;
  const int chunk = (int)(item - yz * chunks), z = (int)(yz / o.blocks);
  const int half = threadIdx.x & 1, rt = threadIdx.x >> 1;
  const int64_t r = o.r0 + (yz - (int64_t)z * o.blocks) * 128 + rt;
  const int64_t k = (int64_t)chunk * TG_K + half * 8;
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  if (r < o.rows) {
    const float* s = o.p + z * o.bstride + r * o.ld + k;    // 16-byte aligned, ld a multiple of 4
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      if (k + i + 3 < o.kext) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(s + i));
        v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
      } else {
#pragma unroll
        for (int j = i; j < i + 4; ++j)
          if (k + j < o.kext) v[j] = __ldg(s + j);
      }
    }
  }
  const float sc = ldexpf(1.f, 8 - grid_exp(__ldg(o.amax + (o.kg > 0 ? chunk / o.kg : z))));
  uint4 p0, p1, p2;
  slice8(v, sc, p0, p1, p2);
  unsigned char* out = o.planes + item * kBlock + (rt >> 3) * 256 + half * 128 + (rt & 7) * 16;
  *reinterpret_cast<uint4*>(out) = p0;
  *reinterpret_cast<uint4*>(out + kPlaneA) = p1;
  *reinterpret_cast<uint4*>(out + 2 * kPlaneA) = p2;
}

struct TMma {
  const unsigned char* pa;     // A's planes; B's by the tensor map
  int64_t row0;                // first row of A's slab
  int M, N, G, kg;             // rows of the slab, columns, groups, chunks of a group
  int a_blocks, b_blocks;      // 128-row blocks of a batch in the planes
  int a_batch, b_batch;        // batched?
  int a_chunks, b_chunks;      // chunks of a row
  const float *amaxA, *amaxB;
};

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1) k_tg_mma(const __grid_constant__ CUtensorMap tmB,
                                                        const TMma g, const TileSched sch,
                                                        const int64_t ntiles, const TOut out,
                                                        int* err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t fin[2];                     // all MMAs issued have completed
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t landed;                                  // chunks whose copies landed
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = g.G, kg = g.kg;
  // slice-grid index of the group's A and B values
  auto sidx_a = [&](int gr, int z) { return MODE == TG_STORE_F32 ? (g.a_batch ? z : 0) : gr; };
  auto sidx_b = [&](int gr, int z) { return MODE == TG_SUM_F64 ? gr : (g.b_batch ? z : 0); };

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(su32(&tmem_slot)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      bar_init(&acc_full[b], 1);
      bar_init(&acc_empty[b], kEpiWarps);
      bar_init(&fin[b], 1);
    }
    landed = 0;
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  volatile int* abrt = &abort_flag;
  bool ok = true;

  if (warp == 0) {
    // ---- copies of chunk q into stage q % kStages once chunk q - kStages has
    // been multiplied: A's planes are one piece, the 2 KB pieces of B one tensor copy
    if (lane == 0) {
      uint32_t q = 0;
      for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        int tm, tn, z;
        sch.at(t, tm, tn, z);
        for (int c = 0; c < G * kg; ++c, ++q) {
          const int s = q % kStages;
          // TG_SQSUM_F64: group c / kg reads batch c / kg of A at chunk c % kg
          const int ca = MODE == TG_SQSUM_F64 ? c % kg : c;
          const int za = MODE == TG_SQSUM_F64 ? c / kg : (g.a_batch ? z : 0);
          const int cb = MODE == TG_SQSUM_F64 ? c % kg : c, zb = g.b_batch ? z : 0;
          if (q >= kStages) {
            const uint32_t par = (q / kStages - 1) & 1;
            if (!bar_wait(&empty[s], par, abrt, 0)) {
              ok = false;
              break;
            }
            // the stage's previous copies must have landed before it is armed
            // again (holds by construction; a broken invariant ends the kernel
            // with an error, not with a bad barrier)
            if (!bar_test(&full[s], par)) {
              atomicExch(err, 3);
              ok = false;
              *abrt = 1;
              break;
            }
          }
          const uint32_t fb = su32(&full[s]), dst = su32(smem) + s * kStage;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                       "r"(kStage) : "memory");
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
              ::"r"(dst), "l"(g.pa + (((int64_t)za * g.a_blocks + tm) * g.a_chunks + ca) * kBlock),
                "r"(kBlock), "r"(fb) : "memory");
          tma_load(dst + kBlock, &tmB, (tn & 1) * (kPlaneB / 8), 0,
                   (zb * g.b_blocks + (tn >> 1)) * g.b_chunks + cb, true, fb);
        }
      }
      // on abort, let the copies already issued land before the CTA exits
      if (!ok)
        for (uint32_t r = (q > kStages ? q - kStages : 0); r < q; ++r)
          bar_drain(&full[r % kStages], (r / kStages) & 1);
    }
  } else if (warp == 2) {
    // ---- chunks landed, in order
    if (lane == 0) {
      uint32_t q = 0;
      for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
        for (int c = 0; c < G * kg; ++c, ++q) {
          if (!bar_wait(&full[q % kStages], (q / kStages) & 1, abrt, 0)) {
            ok = false;
            break;
          }
          asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(su32(&landed)),
                       "r"(q + 1) : "memory");
        }
    }
  } else if (warp == 1 || warp == 3) {
    // ---- MMAs of every other group into accumulator buffer b
    const int b = warp >> 1;
    if (elect_one()) {
      const uint32_t base0 = su32(smem), dcol = tmem + (uint32_t)(b * kBufCols);
      uint32_t avail = 0, gg = 0;                    // groups over all tiles
      for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        for (int gr = 0; gr < G && ok; ++gr, ++gg) {
          if ((gg & 1) != (uint32_t)b) continue;
          // the buffer emptied (this thread's MMAs are long done by then)
          if (gg >= 2 && !bar_wait(&acc_empty[b], ((gg >> 1) - 1) & 1, abrt, 0)) {
            ok = false;
            break;
          }
          for (int c = 0; c < kg; ++c) {
            const uint32_t q = gg * kg + c;
            for (int i = 0; i < kTcMaxWait && avail <= q; ++i) {
              asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(avail)
                           : "r"(su32(&landed)) : "memory");
              if (avail > q || *abrt) break;
            }
            if (avail <= q) { ok = false; *abrt = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = base0 + (q % kStages) * kStage;
            // (slice of A, first slice of B, slices, first level, accumulate):
            // a0 (b0 b1 b2) -> levels 0-2, a1 (b0 b1 b2) -> 1-3, a2 (b0 b1) -> 2-3;
            // a group's first product into level 3 starts it
            auto mma = [&](int pa, int pb, int cnt, int level, bool acc) {
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                  ::"r"(dcol + (uint32_t)(level * TG_N)), "l"(kmajor_desc(base + pa * kPlaneA)),
                    "l"(kmajor_desc(base + kBlock + pb * kPlaneB)), "r"(idesc_mma(cnt * TG_N)),
                    "r"(acc ? 1u : 0u));
            };
            mma(0, 0, 3, 0, c > 0);
            if (c > 0) {
              mma(1, 0, 3, 1, true);
            } else {
              mma(1, 0, 2, 1, true);
              mma(1, 2, 1, 3, false);
            }
            mma(2, 0, 2, 2, true);
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(su32(&empty[q % kStages])) : "memory");
          }
          if (!ok) break;
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
              ::"r"(su32(&acc_full[b])) : "memory");
        }
      }
      // every MMA issued has completed before tensor memory is released
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
          ::"r"(su32(&fin[b])) : "memory");
      bar_drain(&fin[b], 0);
    }
  } else if (warp >= kEpiWarp0) {
    // ---- epilogue: TMEM lanes 32 (warp & 3) .., 16 columns a warp
    const int qd = warp & 3, cw = ((warp - kEpiWarp0) >> 2) * TG_E;
    const int row = qd * 32 + lane;
    const uint32_t lanes = (uint32_t)(qd * 32) << 16;
    uint32_t gg = 0;
    for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
      int tm, tn, z;
      sch.at(t, tm, tn, z);
      const int ml = tm * TG_M + row;
      const bool mok = ml < g.M;
      const int64_t m = g.row0 + ml;
      const int64_t base = mok ? (m % out.r1) * out.s1 + (m / out.r1) * out.s2 + z * out.bs : 0;
      const int n0 = tn * TG_N + cw;
      float hi[TG_E], lo[TG_E];               // double-FP32 sums of the groups
      float vmax = 0.f;
      bool oob = false;
#pragma unroll
      for (int c = 0; c < TG_E; ++c) { hi[c] = 0.f; lo[c] = 0.f; }
      for (int gr = 0; gr < G; ++gr, ++gg) {
        bool w = true;
        if (lane == 0) w = bar_wait(&acc_full[gg & 1], (gg >> 1) & 1, abrt, 32);
        ok = __shfl_sync(0xffffffffu, w, 0);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // level sums are exact integers on the grid 2^(eA + eB - 16)
        const float scale = ldexpf(1.f, grid_exp(__ldg(g.amaxA + sidx_a(gr, z))) +
                                            grid_exp(__ldg(g.amaxB + sidx_b(gr, z))) - 16);
        const float wg = MODE == TG_SQSUM_F64 ? __ldg(out.w + gr) : 0.f;
        const uint32_t acol = tmem + lanes + (uint32_t)((gg & 1) * kBufCols + cw);
#pragma unroll
        for (int c0 = 0; c0 < TG_E; c0 += 8) {
          float s0[8], s1[8], s2[8], s3[8];
          tmem_ld8x4(acol + c0, acol + TG_N + c0, acol + 2 * TG_N + c0, acol + 3 * TG_N + c0, s0,
                     s1, s2, s3);
          if (c0 + 8 == TG_E) {              // the last loads are in registers: release the buffer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&acc_empty[gg & 1]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            // S0 + S1 2^-8 + S2 2^-16 + S3 2^-24 as an unevaluated pair (h, l),
            // without error: x = fl(a + s) and the rest (a - x) + s, where a - x
            // is exact: |S| < 2^24, so it is a multiple of the grid of s (2^-8,
            // 2^-16, 2^-24) of at most 2^24 units
            const float x1 = fmaf(s1[i], 1.f / 256.f, s0[i]);
            float l = fmaf(s1[i], 1.f / 256.f, s0[i] - x1);
            const float x2 = fmaf(s2[i], 1.f / 65536.f, x1);
            l += fmaf(s2[i], 1.f / 65536.f, x1 - x2);
            const float x3 = fmaf(s3[i], 1.f / 16777216.f, x2);
            l += fmaf(s3[i], 1.f / 16777216.f, x2 - x3);
            float vh = x3 * scale, vl = l * scale;
            if constexpr (MODE == TG_STORE_F32) {
              const float v = vh + vl;
              const int64_t n = n0 + c0 + i;
              if (mok && n < g.N) {
                const int64_t off = base + n * out.cs;
                if ((uint64_t)off < (uint64_t)out.limit) {
                  reinterpret_cast<float*>(out.p)[off] = v;
                  vmax = fmaxf(vmax, fabsf(v));
                } else {
                  oob = true;
                }
              }
            } else {
              if constexpr (MODE == TG_SQSUM_F64) {      // w (vh + vl)^2 to double-FP32
                const float sq = vh * vh;
                const float sqe = fmaf(vh, vh, -sq) + 2.f * vh * vl;
                vh = wg * sq;
                vl = fmaf(wg, sq, -vh) + wg * sqe;
              }
              const int c = c0 + i;                      // two-sum of hi and the group's value
              const float sum = hi[c] + vh;
              const float bv = sum - hi[c];
              lo[c] += (hi[c] - (sum - bv)) + (vh - bv) + vl;
              hi[c] = sum;
            }
          }
        }
      }
      if (!ok) break;
      if constexpr (MODE != TG_STORE_F32) {
        double* C = reinterpret_cast<double*>(out.p);
#pragma unroll
        for (int c = 0; c < TG_E; ++c) {
          const int64_t n = n0 + c;
          if (mok && n < g.N) {
            const int64_t off = base + n * out.cs;
            if ((uint64_t)off < (uint64_t)out.limit) {
              const double v = (double)hi[c] + (double)lo[c];
              double* o = C + off;
              *o = out.accumulate ? *o + v : v;
            } else {
              oob = true;
            }
          }
        }
      }
      if (oob) atomicExch(err, 2);
      if constexpr (MODE == TG_STORE_F32) {
        if (out.omax) {
          const unsigned int mb = __reduce_max_sync(0xffffffffu, __float_as_uint(vmax));
          if (lane == 0 && mb) atomicMax(reinterpret_cast<unsigned int*>(out.omax) + z, mb);
        }
      }
    }
  }
  if (!ok) {
    *abrt = 1;
    atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  });
  return fn;
}

// B's planes as (8-byte words of a 4 KB plane, slice, 128-row block and chunk);
// a box is 64 rows (2 KB) of the three slices
ttg_status plane_map(CUtensorMap* map, const unsigned char* planes, int64_t blocks) {
  auto fn = encode_fn();
  if (!fn) return TTG_CUDA_ERR;
  cuuint64_t dims[3] = {kPlaneA / 8, kSlices, (cuuint64_t)blocks};
  cuuint64_t strides[2] = {kPlaneA, kBlock};
  cuuint32_t box[3] = {kPlaneB / 8, kSlices, 1}, es[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<unsigned char*>(planes),
                        dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TTG_OK : TTG_BAD_ARG;
}

bool operand_ok(const TOperand& o) {
  return o.p && o.amax && o.rows > 0 && o.kext > 0 && o.ld >= o.kext && (o.ld * 4) % 16 == 0 &&
         (reinterpret_cast<uintptr_t>(o.p) & 15) == 0 && o.batch >= 0 &&
         !(o.batch > 0 && ((o.bstride * 4) % 16 != 0 || o.bstride <= 0));
}

TSlice slice_of(const TOperand& o, int64_t batches, int64_t r0, int64_t blocks, int chunks, int kg,
                unsigned char* planes) {
  return TSlice{o.p,  o.rows,      o.kext, o.ld, o.bstride, r0, o.amax, kg, (int)blocks,
                blocks * batches * chunks, planes};
}

// Slabs of A's rows that keep the planes within the budget.
struct TPlan {
  int chunks;                       // of a row
  int64_t za, zb, ab, bb;           // batches and 128-row blocks
  int64_t slab, bytes_b, bytes;     // A's blocks at a time, plane bytes
};

TPlan plan_of(int mode, const TOperand& A, const TOperand& B, int Z, int G, int kg,
              int64_t budget = kPlaneBudget) {
  TPlan P;
  P.chunks = mode == TG_SQSUM_F64 ? kg : G * kg;
  P.za = mode == TG_SQSUM_F64 ? G : A.batch > 0 ? Z : 1;
  P.zb = B.batch > 0 ? Z : 1;
  P.ab = (A.rows + 127) / 128;
  P.bb = (B.rows + 127) / 128;
  const int64_t per_block = P.za * P.chunks * kBlock;
  P.bytes_b = P.zb * P.bb * P.chunks * kBlock;
  P.slab = std::max<int64_t>(
      1, std::min(P.ab, (budget - std::min(P.bytes_b, budget / 2)) / per_block));
  P.bytes = P.slab * per_block + P.bytes_b;
  return P;
}

template <int MODE>
ttg_status launch_mode(int grid, cudaStream_t st, const CUtensorMap& mb, const TMma& g,
                       TileSched sch, int64_t ntiles, const TOut& out, int* err) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_tg_mma<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  });
  if (attr != cudaSuccess) return TTG_CUDA_ERR;
  k_tg_mma<MODE><<<grid, kThreads, kSmem, st>>>(mb, g, sch, ntiles, out, err);
  TTG_COUNT();
  cudaError_t e = cudaGetLastError();
  // TTG_SYNC_LAUNCHES=1: wait for each contraction and report its own error
  // (debugging: a fault is then charged to the launch that caused it)
  if (e == cudaSuccess && sync_launches()) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    fprintf(stderr, "ttg: k_tg_mma<%d> (grid %d, M %d, N %d, G %d, kg %d) failed: %s\n", MODE, grid,
            g.M, g.N, g.G, g.kg, cudaGetErrorString(e));
    return TTG_CUDA_ERR;
  }
  return TTG_OK;
}

// amax[g] = max |x[r][k]| over rows r < rows and k in [g gk, (g+1) gk) within kext
__global__ void k_group_max(const float* __restrict__ x, int64_t rows, int64_t kext, int64_t ld,
                            int64_t gk, float* __restrict__ amax) {
  const int g = blockIdx.y;
  const int64_t k0 = (int64_t)g * gk, k1 = min(kext, k0 + gk);
  float vmax = 0.f;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < rows * (k1 - k0);
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / (k1 - k0), k = k0 + e % (k1 - k0);
    vmax = fmaxf(vmax, fabsf(x[r * ld + k]));
  }
  const unsigned int mb = __reduce_max_sync(0xffffffffu, __float_as_uint(vmax));
  if ((threadIdx.x & 31) == 0 && mb) atomicMax(reinterpret_cast<unsigned int*>(amax) + g, mb);
}

}  // namespace

int64_t tgemm_plane_bytes(int mode, const TOperand& A, const TOperand& B, int Z, int G, int kg) {
  return plan_of(mode, A, B, Z, G, kg).bytes;
}

ttg_status tgemm(cudaStream_t st, int mode, const TOperand& A, const TOperand& B, int Z, int G,
                 int kg, const TOut& out, int* err, DevBuf& planes) {
  if (Z <= 0 || G <= 0 || kg <= 0 || kg * TG_K > 192 || !out.p || !err || out.r1 <= 0 ||
      out.limit <= 0)
    return TTG_BAD_ARG;
  if (mode < TG_STORE_F32 || mode > TG_SQSUM_F64) return TTG_BAD_ARG;
  if (mode == TG_STORE_F32 && G != 1) return TTG_BAD_ARG;
  if (mode == TG_SQSUM_F64 && (Z != 1 || A.batch < G || !out.w)) return TTG_BAD_ARG;
  if ((A.batch > 0 && A.batch < Z) || (B.batch > 0 && B.batch < Z)) return TTG_BAD_ARG;
  if (A.rows > INT32_MAX || B.rows > INT32_MAX) return TTG_BAD_ARG;
  if (!operand_ok(A) || !operand_ok(B)) return TTG_BAD_ARG;
  TPlan P = plan_of(mode, A, B, Z, G, kg);
  const int chunks = P.chunks;
  if ((P.slab * P.za + P.bb * P.zb) * chunks > INT32_MAX) return TTG_BAD_ARG;
  // smaller slabs where there is no room for these
  for (int64_t budget = kPlaneBudget; planes.bytes < (size_t)P.bytes;) {
    const ttg_status s = planes.alloc(P.bytes);
    if (s == TTG_OK) break;
    if (s != TTG_OOM || P.slab == 1) return s;
    while (budget > 1 && plan_of(mode, A, B, Z, G, kg, budget).slab >= P.slab) budget /= 2;
    P = plan_of(mode, A, B, Z, G, kg, budget);
  }
  unsigned char* pb = planes.as<unsigned char>();
  unsigned char* pa = pb + P.bytes_b;
  const int by_chunk = mode == TG_SUM_F64 ? kg : 0;
  CUtensorMap mb;
  TTG_TRY(plane_map(&mb, pb, P.zb * P.bb * chunks));
  int dev = 0, sms = 0;
  TTG_CUDA_TRY(cudaGetDevice(&dev));
  TTG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  for (int64_t b0 = 0; b0 < P.ab; b0 += P.slab) {
    const int64_t nb = std::min(P.slab, P.ab - b0), rows = std::min(nb * 128, A.rows - b0 * 128);
    const TSlice sa = slice_of(A, P.za, b0 * 128, nb, chunks, by_chunk, pa);
    TSlice sb = slice_of(B, P.zb, 0, P.bb, chunks, by_chunk, pb);
    if (b0 > 0) sb.items = 0;                       // B's planes are there
    k_tg_slice<<<(unsigned)(sa.items + sb.items), 256, 0, st>>>(sa, sb, chunks); TTG_COUNT();
    TTG_CUDA_TRY(cudaGetLastError());
    const TileSched sch{(int)nb, (int)((B.rows + TG_N - 1) / TG_N)};
    const int64_t ntiles = (int64_t)sch.tiles_m * sch.tiles_n * Z;
    const int grid = (int)std::min<int64_t>(ntiles, sms);
    const TMma g{pa, b0 * 128, (int)rows, (int)B.rows, G, kg, (int)nb, (int)P.bb,
                 A.batch > 0 ? 1 : 0, B.batch > 0 ? 1 : 0, chunks, chunks, A.amax, B.amax};
    switch (mode) {
      case TG_STORE_F32:
        TTG_TRY(launch_mode<TG_STORE_F32>(grid, st, mb, g, sch, ntiles, out, err));
        break;
      case TG_SUM_F64:
        TTG_TRY(launch_mode<TG_SUM_F64>(grid, st, mb, g, sch, ntiles, out, err));
        break;
      default:
        TTG_TRY(launch_mode<TG_SQSUM_F64>(grid, st, mb, g, sch, ntiles, out, err));
    }
  }
  return TTG_OK;
}

}  // namespace ttg

extern "C" ttg_status ttg_tc_gemm(int64_t m, int64_t n, int64_t k, const float* a_dev,
                                  int64_t lda, const float* b_dev, int64_t ldb, int32_t groups,
                                  double* c_dev, int64_t ldc, void* stream) {
  using namespace ttg;
  if (m <= 0 || n <= 0 || k <= 0 || !a_dev || !b_dev || !c_dev || lda < k || ldb < k ||
      ldc < n || groups <= 0)
    return TTG_BAD_ARG;
  const int64_t gk = (k + groups - 1) / groups;              // K values per group
  const int kg = (int)((gk + TG_K - 1) / TG_K);              // chunks per group
  const int64_t gw = (int64_t)kg * TG_K;                     // groups are whole chunks
  if (groups > 1 && gw * (groups - 1) >= k) return TTG_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  DevBuf am, err, planes;
  TTG_TRY(am.alloc((size_t)2 * groups * 4));
  TTG_TRY(err.alloc(sizeof(int)));
  TTG_CUDA_TRY(cudaMemsetAsync(am.p, 0, (size_t)2 * groups * 4, st));
  TTG_CUDA_TRY(cudaMemsetAsync(err.p, 0, sizeof(int), st));
  k_group_max<<<dim3(64, groups), 256, 0, st>>>(a_dev, m, k, lda, gw, am.as<float>()); TTG_COUNT();
  k_group_max<<<dim3(64, groups), 256, 0, st>>>(b_dev, n, k, ldb, gw, am.as<float>() + groups); TTG_COUNT();
  TTG_CUDA_TRY(cudaGetLastError());
  TOperand A{a_dev, m, k, lda, 0, 0, am.as<float>()};
  TOperand B{b_dev, n, k, ldb, 0, 0, am.as<float>() + groups};
  TOut o{c_dev, m + 1, ldc, 0, 1, 0};
  o.limit = (m - 1) * ldc + n;
  TTG_TRY(tgemm(st, TG_SUM_F64, A, B, 1, groups, kg, o, err.as<int>(), planes));
  int e = 0;
  TTG_CUDA_TRY(cudaMemcpyAsync(&e, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  TTG_CUDA_TRY(cudaStreamSynchronize(st));
  return e == 0 ? TTG_OK : e == 2 ? TTG_BAD_ARG : e == 3 ? TTG_CUDA_ERR : TTG_TIMEOUT;
}
