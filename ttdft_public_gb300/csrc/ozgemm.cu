// FP64-accurate GEMMs on the tcgen05 tensor cores: the Gram matrices X^T X and
// X^T (H X), the update X L^-T and the rotation X Q (eigensolver/MultTm.cu:
// 86-224, main.cc:1066-1207 compute them in FP64), the mode Grams and products
// of the STHOSVD and the contraction of the Hamiltonian update.
//
// C[m][n] = sum_k A(m, k) B(n, k) with FP64 operands A (M x K) and B (N x K)
// of any strides (OzOperand); C is FP64.
//
// Arithmetic (an Ozaki-type error-free split).  Every row r of an operand has
// a power-of-two scale with max_k |A(r, k)| < 2^e_r (k_rowexp_*, one pass
// over the operand).  The value v 2^(8 - e_r), below 256 in magnitude, is
// rounded to 40 fractional bits and written as six balanced base-256 digits
//   v 2^(8 - e_r) = d0 + d1 2^-8 + d2 2^-16 + ... + d5 2^-40,
//   |d0| <= 256, |d1..d5| <= 128,
// all exact in BF16.  The digits come from the double's bit pattern by
// integer operations: no FP64 arithmetic, which runs at a small fraction of
// the FP32 rate on this part.  The product of two values is sum_{i,j} d_i d'_j 2^-8(i+j);
// the 21 digit products with i + j <= 5 are summed per level L = i + j in six
// FP32 accumulators in tensor memory.  Over a group of 128 values of K a level
// sum is an integer of magnitude at most 128 * 2^17 = 2^24, so the accumulators
// hold it exactly.  The epilogue folds the six levels of a group with
// error-free two-sums and adds the groups in double-FP32 (about 2^-48
// relative).  Left out: the digit products with i + j >= 6 and the rounding
// of each value to 2^-40 of its row's scale, each below 2^-47 of the product
// of the two rows' scales.
//
// Two kernels.  Cutting a value into digits costs about forty integer
// instructions; inside the GEMM every CTA repeats it for its tile of both
// operands, and that issue rate bounded the product (tensor pipe 6 %).  So
//  - k_oz_slice cuts each operand once into digit planes in a workspace
//    (8 bytes read, 12 written a value: bound by HBM), already in the order
//    the tensor cores read: per 128 rows and 16 values of K one 24 KB block;
//  - k_oz_mma multiplies planes only: three copies (TMA) a chunk into a ring,
//    MMAs, and the fold.
// Operands larger than the workspace (kPlaneBudget) are taken in slabs of K
// (Gram matrices: the sums are added in C's partial) or of A's rows.
//
// k_oz_mma: persistent CTAs over items of a 128 x 64 output tile and a range of
// K (split K), 20 warps.
//  - The six digit planes of 32 rows of B lie one after the other, and so do
//    the six level accumulators, so digit i of A times digits 0 .. 5-i of B is
//    ONE MMA of N = 32 (6 - i) columns, starting at level i: six MMAs a chunk
//    instead of 21, each reading A's plane once (a 128 x 32 MMA alone is bound
//    by the shared-memory read of A).
//  - The tile's two halves of 32 columns (2 x 192 tensor-memory columns) each
//    have an issuing thread (warps 1 and 3): while one half waits for its eight
//    epilogue warps to empty its accumulators, the other's MMAs have the tensor
//    pipe, and the half that is ahead by then stays so.  One thread for both
//    spent a third of its time in the commits (330 cycles each then).  They are
//    elected (elect_one): the MMAs of a 512,000 x 1,200 orthonormalisation
//    took 35.6 ms under `lane == 0`, 33.1 now.  A chunk costs 36 KB of copies
//    for 2 x 336 MMA cycles.
//  - warp 0, one thread: the copies (few and large: 18 copies of 1 to 4 KB a
//    chunk took four times as long, at 85 ns each); warp 2, one thread: waits
//    for a chunk's copies in order and publishes the count (a thread that
//    issues MMAs must not wait on an mbarrier with MMAs in flight: the wait
//    queues behind them); warps 4-11 and 12-19: the folds of the two halves,
//    running double-FP32 sums in registers, at the end scaled by
//    2^(e_m + e_n - 16) and stored.
// Bound: the shared-memory reads of the MMAs (376 cycles a half chunk against
// 336 of arithmetic) and the folds' tensor-memory reads between them.
// Measured (GB300): X^T X of 512,000 x 1,200 in FP64: 150 -> 19 ms with the
// slicing; X L^-T 132 -> 20 ms; X^T Y of 9,261 x 57: 0.17 -> 0.035 ms.
// Every wait is bounded; a wait that runs out sets the error word and the
// abort flag, after which no role issues new copies or MMAs and the CTA
// drains what it issued before releasing tensor memory.

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <vector>
#include <mutex>

#include "ttg_internal.cuh"
#include "tc_common.cuh"

namespace ttg {
namespace {

using namespace tc;

constexpr int OZ_M = 128;                               // rows of an A tile (MMA M)
constexpr int OZ_H = 32;                                // columns of half a tile
constexpr int OZ_N = 2 * OZ_H;                          // rows of a B tile
constexpr int OZ_K = 16;                                // K per chunk
constexpr int kDigits = 6;
constexpr int kLevels = 6;
constexpr int kGroupChunks = 8;                         // 128 values of K per exact level sum
constexpr int kPlA = OZ_M * OZ_K * 2;                   // 4 KB: one BF16 digit plane of A
constexpr int kPlH = OZ_H * OZ_K * 2;                   // 1 KB: of half a B tile
constexpr int kStageA = kDigits * kPlA;                 // 24 KB
constexpr int kStageH = kDigits * kPlH;                 // 6 KB
constexpr int kStage = kStageA + 2 * kStageH;           // 36 KB
constexpr int kStages = 6;
constexpr int kSmem = kStages * kStage + 1024;
constexpr int kEpiWarp0 = 4, kEpiWarps = 8;             // per half: two per 32 TMEM lanes
constexpr int OZ_E = OZ_H / 2;                          // columns of an epilogue warp
constexpr int kThreads = (kEpiWarp0 + 2 * kEpiWarps) * 32;   // 640
constexpr int kHalfCols = kLevels * OZ_H;               // 192
constexpr uint32_t kTmemCols = 512;                     // two halves (384)
constexpr int64_t kPlaneBudget = (int64_t)1 << 30;      // workspace of the digit planes
constexpr int kSMs = 152;                               // one persistent CTA each
constexpr int64_t kRowPad = OZ_M;                       // planes hold whole A tiles of rows

// kind::f16: BF16 x BF16 -> FP32, A and B K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc_oz(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(OZ_M >> 4) << 24);
}

// Six balanced base-256 digits of v 2^(8 - e) (see the file comment) from the
// bits of v; zero for zeros and subnormals (below 2^-1022, far under the
// 2^-40 resolution of any row whose scale is a normal number); NaN in, NaN out.
// One 64-bit shift places the 48-bit fixed-point value; the digits come from
// its two 24-bit halves with 32-bit integer operations.
__device__ __forceinline__ void digits6(double v, int e, int adj, float* d) {
  const int hi = __double2hiint(v);
  const uint32_t lo = (uint32_t)__double2loint(v);
  int E = (hi >> 20) & 0x7FF;
  if (E == 0x7FF) {
#pragma unroll
    for (int i = 0; i < kDigits; ++i) d[i] = __int_as_float(0x7fc00000);
    return;
  }
  uint32_t xl = 0, xh = 0;
  if (E != 0) E = min(E + adj, 2046);                    // v 2^adj (a K scale)
  if (E > 0) {
    const unsigned long long M =
        ((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | lo;
    // v 2^(8-e) 2^40 = M 2^(E - 1075 + 48 - e); |v| < 2^e makes the shift >= 5
    const int rs = 1075 - 48 + e - E;
    if (rs < 63) {
      const unsigned long long X = (M + (1ull << (rs - 1))) >> rs;   // rounded, < 2^48 + 1
      xl = (uint32_t)X & 0xFFFFFFu;
      xh = (uint32_t)(X >> 24);
    }
  }
  // balanced digits, lowest first: d = ((t + 128) mod 256) - 128, t <- (t + 128) / 256
  int t = (int)xl, g[kDigits];
  g[5] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[4] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[3] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  int u = (int)xh + t;
  g[2] = ((u + 128) & 255) - 128; u = (u + 128) >> 8;
  g[1] = ((u + 128) & 255) - 128; u = (u + 128) >> 8;
  g[0] = u;                                             // 0 .. 256
  const int sm = hi >> 31;                              // 0 or -1
#pragma unroll
  for (int i = 0; i < kDigits; ++i) d[i] = (float)((g[i] ^ sm) - sm);
}

// three 8-column tensor-memory loads and one wait, in one statement (the
// registers are defined only after the wait)
__device__ __forceinline__ void tmem_ld8x3(uint32_t a0, uint32_t a1, uint32_t a2, float* v0,
                                           float* v1, float* v2) {
  uint32_t r[24];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
      : "r"(a0), "r"(a1), "r"(a2)
      : "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v0[j] = __uint_as_float(r[j]);
    v1[j] = __uint_as_float(r[8 + j]);
    v2[j] = __uint_as_float(r[16 + j]);
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);   // integers <= 256: exact
  return *reinterpret_cast<const uint32_t*>(&h);
}

// row scale 2^e from the largest biased exponent of the row (0 for an all-zero
// row; a NaN or Inf row, 2047, keeps a large scale: its digits are NaN anyway)
__device__ __forceinline__ int exp_of_bits(int b) { return b == 0 ? 0 : min(b, 2046) - 1022; }

__device__ __forceinline__ int64_t row_at(const OzOperand& o, int64_t r) {
  if (o.idx) r = __ldg(o.idx + r);
  return o.rin >= o.rows ? r * o.rs : (r % o.rin) * o.rs + (r / o.rin) * o.rs2;
}

// One or two operands of the same rows and K (blockIdx.z).
struct OzSlices {
  OzOperand o[2];
  int* ebits[2];              // largest biased exponent of each row
  unsigned char* planes[2];
};

// Digit planes of `chunks` x 16 values of K from k0 on and of 128 gridDim.y rows
// from r0 on: per 128 rows and chunk one 24 KB block, per digit 4 KB of 8-row x
// 16-byte core matrices.  A block cuts kSliceChunks chunks of 128 rows, a thread
// eight values of one row at a time; rows beyond the operand and values beyond
// kext are zero.  K scales (kexp, ksign): v 2^(ksign kexp[k]).
// diag: collects sum_k d3^2 of each row, see k_oz_reduce.
constexpr int kSliceChunks = 4;

template <bool ROWS_FAST>
__global__ void __launch_bounds__(256) k_oz_slice(const OzSlices S, int64_t r0, int64_t k0,
                                                  int chunks, const int* __restrict__ kexp,
                                                  int ksign, unsigned long long* diag) {
  const OzOperand& o = S.o[blockIdx.z];
  const int rt = ROWS_FAST ? threadIdx.x & 127 : threadIdx.x >> 1;
  const int half = ROWS_FAST ? threadIdx.x >> 7 : threadIdx.x & 1;
  const int64_t r = r0 + (int64_t)blockIdx.y * 128 + rt;
  const bool row_ok = r < o.rows;
  const int e = row_ok ? exp_of_bits(__ldg(S.ebits[blockIdx.z] + r)) : 0;
  const double* p = o.p + (row_ok ? row_at(o, r) : 0);
  const int cb = blockIdx.x * kSliceChunks, ce = min(chunks, cb + kSliceChunks);
  unsigned int d3sum = 0;                               // at most 4 x 8 x 2^14
  for (int ch = cb; ch < ce; ++ch) {
    const int64_t k = k0 + (int64_t)ch * OZ_K + half * 8;
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.0;
    if (row_ok) {
      int64_t ki = k, kb = 0;
      if (o.kin < o.kext) {
        kb = k / o.kin;
        ki = k - kb * o.kin;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (k + j < o.kext) v[j] = __ldg(p + ki * o.ks + kb * o.ks2);
        if (++ki == o.kin) {
          ki = 0;
          ++kb;
        }
      }
    }
    uint32_t w[kDigits][4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const int a0 = kexp ? ksign * __ldg(kexp + k + j) : 0;
      const int a1 = kexp ? ksign * __ldg(kexp + k + j + 1) : 0;
      float d0[kDigits], d1[kDigits];
      digits6(v[j], e, a0, d0);
      digits6(v[j + 1], e, a1, d1);
      if (diag) d3sum += (unsigned int)(d0[3] * d0[3] + d1[3] * d1[3]);
#pragma unroll
      for (int d = 0; d < kDigits; ++d) w[d][j / 2] = pack_bf16(d0[d], d1[d]);
    }
    unsigned char* out = S.planes[blockIdx.z] + ((int64_t)blockIdx.y * chunks + ch) * kStageA +
                         (rt >> 3) * 256 + half * 128 + (rt & 7) * 16;
#pragma unroll
    for (int d = 0; d < kDigits; ++d)
      *reinterpret_cast<uint4*>(out + d * kPlA) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
  }
  if (diag) {
    if (!ROWS_FAST) d3sum += __shfl_down_sync(0xffffffffu, d3sum, 1);
    if (row_ok && (ROWS_FAST || half == 0) && d3sum) atomicAdd(diag + r, (unsigned long long)d3sum);
  }
}

// With K scales (kexp, ksign): the biased exponent of v 2^(ksign kexp[k]).
__device__ __forceinline__ int scaled_ebits(double v, const int* kexp, int ksign, int64_t k) {
  int E = (__double2hiint(v) >> 20) & 0x7FF;
  if (E != 0 && E != 0x7FF && kexp) E = max(0, min(2046, E + ksign * __ldg(kexp + k)));
  return E;
}

// Row scales: the largest biased exponent of each row (any v with biased
// exponent E is below 2^(E - 1022)) into ebits, zeroed before.
// Rows contiguous: 32 rows x 8 lanes over K, `kb` values of K a block.
__global__ void __launch_bounds__(256) k_rowexp_rows(const OzSlices S, int64_t kb,
                                                     const int* __restrict__ kexp, int ksign) {
  __shared__ int red[8][33];
  const OzOperand& o = S.o[blockIdx.z];
  const int64_t r = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const int64_t k0 = (int64_t)blockIdx.y * kb, k1 = min(o.kext, k0 + kb);
  int m = 0;
  if (r < o.rows) {
    const double* p = o.p + row_at(o, r);
#pragma unroll 8
    for (int64_t k = k0 + threadIdx.y; k < k1; k += 8) {
      const int64_t q = o.kin < o.kext ? (k % o.kin) * o.ks + (k / o.kin) * o.ks2 : k * o.ks;
      m = max(m, scaled_ebits(p[q], kexp, ksign, k));
    }
  }
  red[threadIdx.y][threadIdx.x] = m;
  __syncthreads();
  if (threadIdx.y == 0 && r < o.rows) {
    for (int y = 1; y < 8; ++y) m = max(m, red[y][threadIdx.x]);
    if (m) atomicMax(S.ebits[blockIdx.z] + r, m);
  }
}

// K contiguous: one warp per row and `kb` values of K
__global__ void __launch_bounds__(256) k_rowexp_k(const OzSlices S, int64_t kb,
                                                  const int* __restrict__ kexp, int ksign) {
  const OzOperand& o = S.o[blockIdx.z];
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= o.rows) return;
  const int64_t k0 = (int64_t)blockIdx.y * kb, k1 = min(o.kext, k0 + kb);
  const double* p = o.p + row_at(o, r);
  int m = 0;
#pragma unroll 4
  for (int64_t k = k0 + lane; k < k1; k += 32) {
    const int64_t q = o.kin < o.kext ? (k % o.kin) * o.ks + (k / o.kin) * o.ks2 : k * o.ks;
    m = max(m, scaled_ebits(p[q], kexp, ksign, k));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0 && m) atomicMax(S.ebits[blockIdx.z] + r, m);
}

__global__ void k_exp_from_bits(int* __restrict__ e, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) e[i] = exp_of_bits(e[i]);
}

// 2^e times a float, as a double: the exponent is rebased in the bits (the
// FP64 pipe, two lanes per SM, would take five operations a value)
__device__ __forceinline__ double scaled_float(float x, int e) {
  const uint32_t b = __float_as_uint(x), m = b & 0x7fffffffu;
  if (m == 0) return 0.0;
  return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + ((896u + (uint32_t)e) << 20))),
                          (int)(b << 29));
}

// (hi + lo) 2^e
__device__ __forceinline__ double scaled_sum(float hi, float lo, int e) {
  // normal floats (sums of multiples of 2^-40) whose doubles stay normal
  if (isfinite(hi) && isfinite(lo) && e > -800 && e < 800)
    return scaled_float(hi, e) + scaled_float(lo, e);
  return ((double)hi + (double)lo) * ldexp(1.0, e);
}

struct OzTiles {
  int tiles_m, tiles_n;
  int sym;          // only tiles with n0 <= m0 + 127 (on and below the diagonal)
  const int* first; // ragged: prefix sums of the column tiles (null: all tiles_n)
  __device__ void at(int t, int& mt, int& nt) const {
    if (first) {
      int lo = 0, hi = tiles_m;              // first[lo] <= t < first[hi]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(first + mid) <= t) lo = mid;
        else hi = mid;
      }
      mt = lo;
      nt = t - __ldg(first + lo);
      return;
    }
    if (!sym) {
      // rotated: a persistent CTA's items (a fixed step apart) then run through
      // all columns, whose K ranges differ for a triangular B
      mt = t / tiles_n;
      nt = (t + mt) % tiles_n;
      return;
    }
    int m = 0;
    for (;; ++m) {
      const int row = min(2 * m + 2, tiles_n);
      if (t < row) break;
      t -= row;
    }
    mt = m;
    nt = t;
  }
};

struct OzOut {
  double* p;
  int64_t rin, rs, rs2, cs, zs;  // (m % rin) rs + (m / rin) rs2 + n cs + split zs
  int accumulate;                // add to p
  const int64_t* base;           // ragged: base[mt] + row ld[mt] + n
  const int* ld;
};

struct OzMma {
  const unsigned char* pa;       // A's digit planes (B's: the tensor map)
  const int *ea, *eb;            // biased exponents of A's and B's rows
  int M, N, chunks, split_chunks;
  int64_t row0;                  // first row of A's slab, for C
  int b_lower_k0;                // >= 0: B(n, k) = 0 for k > n, planes start at this k
};

// What one CTA does of a work item: a tile and a range of K.
struct OzItem {
  int mt, m0, n0, c0, nq, nh, split;     // nq chunks from c0 on, nh halves with columns
  int N;                                 // columns of C here
  __device__ OzItem(const OzMma& g, const OzTiles& tiles, const OzOut& out, int w, int ntiles) {
    split = w / ntiles;
    int nt;
    tiles.at(w - split * ntiles, mt, nt);
    m0 = mt * OZ_M;
    n0 = nt * OZ_N;
    c0 = split * g.split_chunks;
    int c1 = min(g.chunks, c0 + g.split_chunks);
    if (g.b_lower_k0 >= 0) c1 = min(c1, max(0, n0 + OZ_N - g.b_lower_k0 + OZ_K - 1) / OZ_K);
    nq = max(0, c1 - c0);
    N = out.ld ? __ldg(out.ld + mt) : g.N;
    nh = n0 + OZ_H < N ? 2 : 1;
  }
};

// Persistent: CTA b takes items b, b + gridDim.x, ...; the copies and MMAs of
// an item run under the fold and the stores of the one before.  Counters
// (chunks, groups) run on over the items, and so do the barriers' phases.
__global__ void __launch_bounds__(kThreads, 1) k_oz_mma(const __grid_constant__ CUtensorMap tmB,
                                                        const OzMma g, const OzTiles tiles,
                                                        const int ntiles, const int items,
                                                        const OzOut out, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t fin[2];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t landed;                                 // chunks whose copies are there
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(su32(&tmem_slot)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 2);
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
    // been multiplied by both halves: A's six planes are one piece, the six
    // 1 KB pieces of a half of B one tensor copy
    if (lane == 0) {
      uint32_t q = 0;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const OzItem it(g, tiles, out, w, ntiles);
        const unsigned char* src = g.pa + ((int64_t)it.mt * g.chunks + it.c0) * kStageA;
        const int bz = (it.n0 >> 7) * g.chunks + it.c0, bx = (it.n0 & 127) * 4;
        for (int c = 0; c < it.nq; ++c, ++q) {
          const int s = q % kStages;
          if (q >= kStages) {
            const uint32_t par = (q / kStages - 1) & 1;
            if (!bar_wait(&empty[s], par, abrt, 0)) {
              ok = false;
              break;
            }
            // the stage's previous copies must have landed before it is armed again
            if (!bar_test(&full[s], par)) {
              atomicExch(err, 3);
              ok = false;
              *abrt = 1;
              break;
            }
          }
          const uint32_t fb = su32(&full[s]), dst = su32(smem) + s * kStage;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                       ::"r"(fb), "r"(kStageA + it.nh * kStageH) : "memory");
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
              ::"r"(dst), "l"(src + (int64_t)c * kStageA), "r"(kStageA), "r"(fb) : "memory");
          for (int h = 0; h < it.nh; ++h)
            tma_load(dst + kStageA + h * kStageH, &tmB, bx + h * OZ_H * 4, 0, bz + c, true, fb);
        }
      }
      if (!ok)
        for (uint32_t r = (q > kStages ? q - kStages : 0); r < q; ++r)
          bar_drain(&full[r % kStages], (r / kStages) & 1);
    }
  } else if (warp == 2) {
    // ---- chunks landed, in order
    if (lane == 0) {
      uint32_t q = 0;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const OzItem it(g, tiles, out, w, ntiles);
        for (int c = 0; c < it.nq; ++c, ++q) {
          if (!bar_wait(&full[q % kStages], (q / kStages) & 1, abrt, 0)) {
            ok = false;
            break;
          }
          asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(su32(&landed)),
                       "r"(q + 1) : "memory");
        }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ---- MMAs of one half: digit i of A times digits 0 .. 5 - i of B in one
    const int h = warp >> 1;
    if (elect_one()) {
      const uint32_t base0 = su32(smem), dcol = tmem + (uint32_t)(h * kHalfCols);
      uint32_t avail = 0, q = 0, gr = 0;                  // chunks, groups of this half
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const OzItem it(g, tiles, out, w, ntiles);
        const bool on = h < it.nh;
        for (int j = 0; j < it.nq; ++j, ++q) {
          const int c = j % kGroupChunks, s = q % kStages;
          // the group's accumulators emptied (its own MMAs are long done by then)
          if (on && c == 0 && gr > 0 && !bar_wait(&acc_empty[h], (gr - 1) & 1, abrt, 0)) {
            ok = false;
            break;
          }
          for (int i = 0; i < kTcMaxWait && avail <= q; ++i) {
            asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(avail)
                         : "r"(su32(&landed)) : "memory");
            if (avail > q || *abrt) break;
          }
          if (avail <= q) { ok = false; *abrt = 1; break; }
          if (!on) {                        // no columns in this half: it only frees the stage
            bar_arrive(&empty[s]);
            continue;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t base = base0 + (uint32_t)(s * kStage);
          const uint64_t db = kmajor_desc(base + kStageA + h * kStageH);
#pragma unroll
          for (int i = 0; i < kDigits; ++i) {
            const uint64_t da = kmajor_desc(base + i * kPlA);
            const uint32_t acc = (c > 0 || i > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                ::"r"(dcol + (uint32_t)(i * OZ_H)), "l"(da), "l"(db),
                  "r"(idesc_oz(OZ_H * (kDigits - i))), "r"(acc));
          }
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
              ::"r"(su32(&empty[s])) : "memory");
          if (c == kGroupChunks - 1 || j == it.nq - 1) {
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(su32(&acc_full[h])) : "memory");
            ++gr;
          }
        }
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
          ::"r"(su32(&fin[h])) : "memory");
      bar_drain(&fin[h], 0);
    }
  } else if (warp >= kEpiWarp0) {
    // ---- fold of half a tile: TMEM lanes 32 (warp & 3) .., 16 columns a warp
    // (two warps per lane quarter: each waits on its tensor-memory loads)
    const int h = (warp - kEpiWarp0) / kEpiWarps, qd = warp & 3;
    const int cb = (((warp - kEpiWarp0) >> 2) & 1) * OZ_E;
    const int row = qd * 32 + lane;
    const uint32_t acol = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(h * kHalfCols + cb);
    uint32_t gr = 0;
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const OzItem it(g, tiles, out, w, ntiles);
      if (h >= it.nh) continue;
      const int ng = (it.nq + kGroupChunks - 1) / kGroupChunks;
      float hi[OZ_E], lo[OZ_E];
#pragma unroll
      for (int c = 0; c < OZ_E; ++c) { hi[c] = 0.f; lo[c] = 0.f; }
      for (int t = 0; t < ng; ++t, ++gr) {
        // one lane polls: 512 threads on two barriers would slow every wait
        bool wt = true;
        if (lane == 0) wt = bar_wait(&acc_full[h], gr & 1, abrt, 32);
        ok = __shfl_sync(0xffffffffu, wt, 0);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int cc = 0; cc < OZ_E; cc += 8) {
          float S[kLevels][8];
          tmem_ld8x3(acol + cc, acol + OZ_H + cc, acol + 2 * OZ_H + cc, S[0], S[1], S[2]);
          tmem_ld8x3(acol + 3 * OZ_H + cc, acol + 4 * OZ_H + cc, acol + 5 * OZ_H + cc, S[3], S[4],
                     S[5]);
          if (cc + 8 == OZ_E) {              // the last loads are in registers: release the buffer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&acc_empty[h]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            // S0 + S1 2^-8 + ... + S5 2^-40 as (f, l), then into (hi, lo)
            float f = S[0][i], l = 0.f;
            float sc = 1.f / 256.f;
#pragma unroll
            for (int L = 1; L < kLevels; ++L, sc *= (1.f / 256.f)) {
              const float u = S[L][i] * sc;
              const float h2 = f + u;
              const float bv = h2 - f;
              l += (f - (h2 - bv)) + (u - bv);
              f = h2;
            }
            const float sum = hi[cc + i] + f;
            const float bv = sum - hi[cc + i];
            lo[cc + i] += (hi[cc + i] - (sum - bv)) + (f - bv) + l;
            hi[cc + i] = sum;
          }
        }
      }
      if (!ok || it.m0 + row >= g.M) continue;
      const int em = exp_of_bits(__ldg(g.ea + it.m0 + row)) - 16;
      const int64_t m = g.row0 + it.m0 + row;
      const int nb = it.n0 + h * OZ_H + cb;
      double* o = out.p;
      if (out.ld)
        o += __ldg(out.base + it.mt) + (int64_t)row * it.N + nb;
      else
        o += it.split * out.zs + nb * out.cs +
             (m < out.rin ? m * out.rs : (m % out.rin) * out.rs + (m / out.rin) * out.rs2);
      const bool pairs = out.cs == 1 && !out.accumulate && (reinterpret_cast<uintptr_t>(o) & 15) == 0;
#pragma unroll
      for (int c = 0; c < OZ_E; c += 2) {
        double v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int n = min(nb + c + u, g.N - 1);
          v[u] = scaled_sum(hi[c + u], lo[c + u], em + exp_of_bits(__ldg(g.eb + n)));
        }
        if (pairs && nb + c + 1 < it.N) {
          *reinterpret_cast<double2*>(o + c) = make_double2(v[0], v[1]);
        } else {
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (nb + c + u < it.N) {
              double* t = o + (c + u) * out.cs;
              *t = out.accumulate ? *t + v[u] : v[u];
            }
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

// S = sum of the split partials (column-major M x N); sym: tiles above the
// diagonal were not computed, S[m, n] is read from [n, m] there.  Eight
// threads share an element's splits (fixed order), 32 elements a block.
// diag (X^T X): the products left out, of digits i + j >= 6, sum to about zero
// except the squares on the diagonal; sum_k d3^2 of each row, exact, is added
// there (weight 2^-48 of the row's scale squared).  Without it the diagonal of
// a peaked field's Gram matrix is low by 1e-13, which turns the trailing
// eigenvectors of an STHOSVD more than double-FP32 sums did.
__global__ void __launch_bounds__(256) k_oz_reduce(const double* __restrict__ part, int nsplit,
                                                   int M, int N, int sym,
                                                   const unsigned long long* __restrict__ diag,
                                                   const int* __restrict__ ebits,
                                                   double* __restrict__ C, int64_t c_rs,
                                                   int64_t c_cs) {
  __shared__ double red[8][33];
  const int64_t mn = (int64_t)M * N;
  for (int64_t b = blockIdx.x; b * 32 < mn; b += gridDim.x) {
    const int64_t i = b * 32 + threadIdx.x;
    double s = 0.0;
    const int m = (int)(i % M), n = (int)(i / M);
    if (i < mn) {
      int64_t src = i;
      if (sym && (n / OZ_N) * OZ_N > (m / OZ_M) * OZ_M + OZ_M - 1) src = n + (int64_t)m * M;
      for (int z = threadIdx.y; z < nsplit; z += 8) s += part[(int64_t)z * mn + src];
    }
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && i < mn) {
      for (int y = 1; y < 8; ++y) s += red[y][threadIdx.x];
      if (diag && m == n) s += ldexp((double)diag[m], 2 * exp_of_bits(ebits[m]) - 16 - 48);
      C[m * c_rs + n * c_cs] = s;
    }
    __syncthreads();
  }
}

int64_t rup(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

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

// B's planes as (8-byte words of a 4 KB plane, digit, 128-row block and chunk);
// a box is 32 rows (1 KB) of all six digits
ttg_status plane_map(CUtensorMap* map, const unsigned char* planes, int64_t blocks) {
  auto fn = encode_fn();
  if (!fn) return TTG_CUDA_ERR;
  cuuint64_t dims[3] = {kPlA / 8, kDigits, (cuuint64_t)blocks};
  cuuint64_t strides[2] = {kPlA, kStageA};
  cuuint32_t box[3] = {kPlH / 8, kDigits, 1}, es[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<unsigned char*>(planes),
                        dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TTG_OK : TTG_BAD_ARG;
}

bool rows_fast(const OzOperand& o) { return o.rs == 1 && o.ks != 1; }

bool same_operand(const OzOperand& a, const OzOperand& b) {
  return a.p == b.p && a.rows == b.rows && a.kext == b.kext && a.rin == b.rin && a.rs == b.rs &&
         a.rs2 == b.rs2 && a.kin == b.kin && a.ks == b.ks && a.ks2 == b.ks2 && a.idx == b.idx;
}

ttg_status row_exps(cudaStream_t st, const OzSlices& S, int nz, const int* kexp, int ksign) {
  const OzOperand& o = S.o[0];
  for (int z = 0; z < nz; ++z)
    TTG_CUDA_TRY(cudaMemsetAsync(S.ebits[z], 0, (size_t)o.rows * sizeof(int), st));
  if (rows_fast(o)) {
    int64_t kb = 128;            // values of K a block: many blocks for a narrow operand
    while ((o.kext + kb - 1) / kb > 8192) kb *= 2;
    k_rowexp_rows<<<dim3((unsigned)((o.rows + 31) / 32), (unsigned)((o.kext + kb - 1) / kb), nz),
                    dim3(32, 8), 0, st>>>(S, kb, kexp, ksign); TTG_COUNT();
  } else {
    int64_t kb = 4096;
    while ((o.kext + kb - 1) / kb > 8192) kb *= 2;
    k_rowexp_k<<<dim3((unsigned)((o.rows + 7) / 8), (unsigned)((o.kext + kb - 1) / kb), nz), 256,
                 0, st>>>(S, kb, kexp, ksign); TTG_COUNT();
  }
  TTG_CUDA_TRY(cudaGetLastError());
  return TTG_OK;
}

ttg_status error_word(cudaStream_t st, OzWork& ws, int** err) {
  if (!ws.word && !ws.err.p) {
    TTG_TRY(ws.err.alloc(sizeof(int)));
    TTG_CUDA_TRY(cudaMemsetAsync(ws.err.p, 0, sizeof(int), st));
  }
  *err = ws.word ? ws.word : ws.err.as<int>();
  return TTG_OK;
}

// TTG_FAKE_TIMEOUT=1 (tests of the callers): the error word as a kernel whose
// wait ran out leaves it.
__global__ void k_oz_fake_timeout(int* err) { atomicExch(err, 1); }

ttg_status fake_timeout(cudaStream_t st, int* err) {
  if (!getenv("TTG_FAKE_TIMEOUT")) return TTG_OK;
  k_oz_fake_timeout<<<1, 1, 0, st>>>(err);
  TTG_CUDA_TRY(cudaGetLastError());
  return TTG_OK;
}

ttg_status slice(cudaStream_t st, const OzSlices& S, int nz, int64_t r0, int64_t rpad, int64_t k0,
                 int64_t chunks, const int* kexp, int ksign, unsigned long long* diag = nullptr) {
  if (chunks <= 0) return TTG_OK;
  const dim3 grid((unsigned)((chunks + kSliceChunks - 1) / kSliceChunks), (unsigned)(rpad / 128), nz);
  if (rows_fast(S.o[0]))
    k_oz_slice<true><<<grid, 256, 0, st>>>(S, r0, k0, (int)chunks, kexp, ksign, diag);
  else
    k_oz_slice<false><<<grid, 256, 0, st>>>(S, r0, k0, (int)chunks, kexp, ksign, diag);
  TTG_COUNT();
  TTG_CUDA_TRY(cudaGetLastError());
  return TTG_OK;
}

}  // namespace

int64_t ozgemm_ragged_rows(int64_t K, int64_t N) {
  const int64_t row = (K + OZ_K - 1) / OZ_K * kDigits * 32;        // bytes of a row's planes
  return std::max<int64_t>(0, (kPlaneBudget - rup(N, kRowPad) * row) / row / kRowPad * kRowPad);
}

ttg_status ozgemm_reserve(ttg_op* op, int64_t M, int64_t N, int64_t K) {
  OzWork& w = op->oz;
  const int64_t row = (K + OZ_K - 1) / OZ_K * kDigits * 32;
  const size_t planes = (size_t)((rup(M, kRowPad) + rup(N, kRowPad)) * row);
  const size_t exps = (size_t)(M + N) * sizeof(int);
  if (w.planes.bytes < planes) TTG_TRY(w.planes.alloc(planes));
  if (w.exp.bytes < exps) TTG_TRY(w.exp.alloc(exps));
  return TTG_OK;
}

bool ozgemm_supported(const OzOperand& A, const OzOperand& B) {
  if (getenv("TTG_DISABLE_OZGEMM")) return false;
  return A.p && B.p && A.rows > 0 && B.rows > 0 && A.kext > 0 && A.kext == B.kext &&
         A.rows <= INT32_MAX - 256 && B.rows <= INT32_MAX - 256 && A.kext <= INT32_MAX - 256;
}

ttg_status ozgemm(cudaStream_t st, OzWork& ws, DevBuf& partial_buf, const OzOperand& A,
                  const OzOperand& B, double* C, OzLayout c, bool sym, bool b_lower,
                  const OzOperand* kscale_of, const OzRagged* ragged) {
  if (!ozgemm_supported(A, B) || !C) return TTG_BAD_ARG;
  if (sym && (A.rows != B.rows || c.rin < A.rows)) return TTG_BAD_ARG;
  if (ragged && (sym || b_lower || kscale_of || A.rows > ozgemm_ragged_rows(A.kext, B.rows)))
    return TTG_BAD_ARG;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_oz_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  });
  if (attr != cudaSuccess) return TTG_CUDA_ERR;
  const int64_t M = A.rows, N = B.rows, K = A.kext;
  const int64_t mpad = rup(M, kRowPad), npad = rup(N, kRowPad), chunks = (K + OZ_K - 1) / OZ_K;
  const bool same = !kscale_of && same_operand(A, B);
  // Slabs that keep the digit planes within the workspace: of A's rows when
  // B's planes take a quarter of it at most (N x k products), else of K
  // (Gram matrices), whole groups at a time.
  const int64_t per_chunk = kDigits * 32;                       // bytes of a row's chunk
  const int64_t bytes_a = mpad * chunks * per_chunk, bytes_b = same ? 0 : npad * chunks * per_chunk;
  int64_t mslab = mpad, kslab = chunks;                          // rows, chunks
  if (bytes_a + bytes_b > kPlaneBudget) {
    if (!sym && !same && bytes_b <= kPlaneBudget / 4) {
      mslab = std::max<int64_t>(1, (kPlaneBudget - bytes_b) / (chunks * per_chunk) / kRowPad) * kRowPad;
    } else {
      const int64_t rows = same ? mpad : mpad + npad;
      kslab = std::max<int64_t>(1, kPlaneBudget / (rows * per_chunk) / kGroupChunks) * kGroupChunks;
    }
    mslab = std::min(mslab, mpad);
    kslab = std::min(kslab, chunks);
  }
  const int64_t need_a = mslab * kslab * per_chunk, need_b = same ? 0 : npad * kslab * per_chunk;
  if (ws.planes.bytes < (size_t)(need_a + need_b)) TTG_TRY(ws.planes.alloc(need_a + need_b));
  unsigned char* pa = ws.planes.as<unsigned char>();
  unsigned char* pb = same ? pa : pa + need_a;
  if (ws.exp.bytes < (size_t)(M + N) * sizeof(int))
    TTG_TRY(ws.exp.alloc((size_t)(M + N) * sizeof(int)));
  unsigned long long* diag = nullptr;            // X^T X: the diagonal's share of d3 d3
  if (same && sym) {
    if (ws.diag.bytes < (size_t)M * 8) TTG_TRY(ws.diag.alloc((size_t)M * 8));
    diag = ws.diag.as<unsigned long long>();
    TTG_CUDA_TRY(cudaMemsetAsync(diag, 0, (size_t)M * 8, st));
  }
  int* err = nullptr;
  TTG_TRY(error_word(st, ws, &err));
  int* ea = ws.exp.as<int>();
  int* eb = same ? ea : ea + M;
  // K scales: the row scales of kscale_of (a view whose rows are the K
  // index), A scaled by 2^-f_k and B by 2^f_k; the buffer is padded with zeros
  // to whole chunks
  const int* kexp = nullptr;
  if (kscale_of) {
    if (kscale_of->rows != K) return TTG_BAD_ARG;
    const size_t kb = (size_t)(chunks * OZ_K) * sizeof(int);
    if (ws.kexp.bytes < kb) TTG_TRY(ws.kexp.alloc(kb));
    TTG_CUDA_TRY(cudaMemsetAsync(ws.kexp.p, 0, kb, st));
    OzSlices S{};
    S.o[0] = *kscale_of;
    S.ebits[0] = ws.kexp.as<int>();
    TTG_TRY(row_exps(st, S, 1, nullptr, 0));
    k_exp_from_bits<<<(unsigned)((K + 255) / 256), 256, 0, st>>>(ws.kexp.as<int>(), K); TTG_COUNT();
    TTG_CUDA_TRY(cudaGetLastError());
    kexp = ws.kexp.as<int>();
  }
  // both operands in one launch where they have one shape and orientation
  const bool pair = !same && !kexp && M == N && rows_fast(A) == rows_fast(B);
  OzSlices SA{}, SB{};
  SA.o[0] = A;
  SA.ebits[0] = ea;
  SA.planes[0] = pa;
  SB.o[0] = B;
  SB.ebits[0] = eb;
  SB.planes[0] = pb;
  if (pair) {
    SA.o[1] = B;
    SA.ebits[1] = eb;
    SA.planes[1] = pb;
  }
  TTG_TRY(row_exps(st, SA, pair ? 2 : 1, kexp, -1));
  if (!same && !pair) TTG_TRY(row_exps(st, SB, 1, kexp, 1));
  const int tiles_n = (int)((N + OZ_N - 1) / OZ_N);
  OzTiles tiles{(int)((std::min(mslab, M) + OZ_M - 1) / OZ_M), tiles_n, sym ? 1 : 0,
                ragged ? ragged->first : nullptr};
  int64_t ntiles = ragged ? ragged->items : (int64_t)tiles.tiles_m * tiles_n;
  if (sym) {
    ntiles = 0;
    for (int m = 0; m < tiles.tiles_m; ++m) ntiles += std::min(2 * m + 2, tiles_n);
  }
  // Split K for the least time: items per CTA (one per SM) times their groups
  // (about 1.2 us each, two more to fill the ring and to store), plus the
  // partials written and summed.
  const int64_t kgroups = (kslab + kGroupChunks - 1) / kGroupChunks;
  int64_t nsplit = 1;
  if (!b_lower && !ragged && c.rin >= M) {
    double best = 1e300;
    for (int64_t t = 1; t <= std::min<int64_t>(kgroups, 8 * kSMs / ntiles + 1); ++t) {
      const double cost = (double)((ntiles * t + kSMs - 1) / kSMs) * ((kgroups + t - 1) / t + 2) +
                          (t > 1 || sym ? t * (double)M * N * 16 / 7e6 : 0.0);
      if (cost < best) {
        best = cost;
        nsplit = t;
      }
    }
  }
  const int64_t sgroups = (kgroups + nsplit - 1) / nsplit;
  nsplit = (kgroups + sgroups - 1) / sgroups;
  if (ntiles > INT32_MAX || nsplit > 65535 || mslab / 128 > 65535 || npad / 128 > 65535)
    return TTG_BAD_ARG;
  OzOut out{C, c.rin, c.rs, c.rs2, c.cs, 0, 0, nullptr, nullptr};
  if (ragged) {
    out.cs = 1;
    out.base = ragged->base;
    out.ld = ragged->ld;
  }
  const bool partial = nsplit > 1 || sym;
  if (partial) {
    const size_t need = (size_t)nsplit * M * N * sizeof(double);
    if (partial_buf.bytes < need) TTG_TRY(partial_buf.alloc(need));
    out = OzOut{partial_buf.as<double>(), M, 1, 0, M, M * N, 0, nullptr, nullptr};
  }
  for (int64_t q0 = 0; q0 < chunks; q0 += kslab) {
    const int64_t nq = std::min(kslab, chunks - q0);
    if (!same && !pair) TTG_TRY(slice(st, SB, 1, 0, npad, q0 * OZ_K, nq, kexp, 1));
    for (int64_t r0 = 0; r0 < M; r0 += mslab) {
      const int64_t rows = std::min(mslab, M - r0), rpad = rup(rows, kRowPad);
      TTG_TRY(slice(st, SA, pair ? 2 : 1, r0, rpad, q0 * OZ_K, nq, kexp, -1, diag));
      OzTiles tl = tiles;
      tl.tiles_m = (int)((rows + OZ_M - 1) / OZ_M);
      const int64_t nt = sym || ragged ? ntiles : (int64_t)tl.tiles_m * tiles_n;
      CUtensorMap mb;
      TTG_TRY(plane_map(&mb, pb, npad / 128 * nq));
      OzMma g{pa, ea + r0, eb, (int)rows, (int)N, (int)nq,
              (int)(sgroups * kGroupChunks), r0, b_lower ? (int)(q0 * OZ_K) : -1};
      OzOut o = out;
      o.accumulate = q0 > 0 ? 1 : 0;
      const int64_t items = nt * nsplit;
      if (items > INT32_MAX) return TTG_BAD_ARG;
      k_oz_mma<<<(unsigned)std::min<int64_t>(items, kSMs), kThreads, kSmem, st>>>(
          mb, g, tl, (int)nt, (int)items, o, err); TTG_COUNT();
      cudaError_t e = cudaGetLastError();
      if (e == cudaSuccess && sync_launches()) e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) {
        fprintf(stderr, "ttg: k_oz_mma (M %lld, N %lld, K %lld) failed: %s\n", (long long)M,
                (long long)N, (long long)K, cudaGetErrorString(e));
        return TTG_CUDA_ERR;
      }
    }
  }
  if (partial) {
    const int64_t mn = M * N;
    k_oz_reduce<<<(unsigned)std::min<int64_t>((mn + 31) / 32, 152 * 16), dim3(32, 8), 0, st>>>(
        out.p, (int)nsplit, (int)M, (int)N, sym ? 1 : 0, diag, ea, C, c.rs, c.cs); TTG_COUNT();
    TTG_CUDA_TRY(cudaGetLastError());
  }
  return fake_timeout(st, err);
}

ttg_status ozgemm_error(cudaStream_t st, OzWork& ws) {
  int e = 0;
  if (ws.err.p)
    TTG_CUDA_TRY(cudaMemcpyAsync(&e, ws.err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  TTG_CUDA_TRY(cudaStreamSynchronize(st));
  if (ws.word) e = *static_cast<volatile int*>(ws.word);
  if (e) {
    if (ws.word) *static_cast<volatile int*>(ws.word) = 0;
    else TTG_CUDA_TRY(cudaMemsetAsync(ws.err.p, 0, sizeof(int), st));
    fprintf(stderr, "ttg: FP64 tensor-core GEMM: %s\n",
            e == 3 ? "a copy barrier out of phase" : "a bounded wait ran out");
    return e == 3 ? TTG_CUDA_ERR : TTG_TIMEOUT;
  }
  return TTG_OK;
}

ttg_status ozgemm(ttg_op* op, const OzOperand& A, const OzOperand& B, double* C, OzLayout c,
                  bool sym, bool b_lower, const OzOperand* kscale_of, const OzRagged* ragged) {
  return ozgemm(op->stream, op->oz, op->partial, A, B, C, c, sym, b_lower, kscale_of, ragged);
}

ttg_status ozgemm_error(ttg_op* op) { return ozgemm_error(op->stream, op->oz); }

}  // namespace ttg

// ------------------------------------------------------------- H X in FP64 ----
//
// The Rayleigh-Ritz product H X (eigensolver/MultTm.cu computes it in FP64) on
// the tiles of the filter degrees (spmm_umma.cu: 128 rows, their sorted column
// union in chunks of 16 slots), with the digits, levels and folds of k_oz_mma,
// but seven of them: a row of H holds values far below its diagonal, and with
// six its eigenvectors were off by twice what double-FP32 sums had (4.2e-10
// against 2.3e-10).  A is a tile's rows of H, cut once per operator and set of
// values into a 28 KB block a chunk; B are the gathered rows of X, cut before
// each product and laid out row by row, for 32 states seven digits of 64 bytes
// each (512 bytes with the place of an eighth).  Two such groups of a row are
// an item's columns, and digit i of H times digits 0 .. 6-i of a group is one
// MMA, as in k_oz_mma.  (Level 6 may pass 2^24 and lose its last place, 2^-64
// of the product of the two scales.)
// Bound: the MMAs' shared-memory reads and the copies (42 KB a chunk and 64
// states through L2).  k_apply_df64 (spmm.cu) -> this, 64,000 functions: 160
// states 14.8 -> 4.6 ms, 40 states 6.3 -> 1.7 ms; 1,728 functions, 16 states 0.47
// -> 0.07 ms; H is cut in about 3 ms at 64,000 functions.  It is faster at every
// width; the other kernel is left where there are no tiles or no room.

namespace ttg {
namespace {

constexpr int kApThreads = 768;                       // 24 warps, the last four gather
constexpr int kApGather = 4;
constexpr int kApDigits = 7, kApLevels = 7;
constexpr int kApH = kApDigits * kPlA;                // 28 KB: H's digits of a chunk
constexpr int kApAtom = 16 * 128;                     // 16 slots x 128 bytes (two digits of 32 states)
constexpr int kApAtoms = (kApDigits + 1) / 2;         // of a group
constexpr int kApRows = 2 * kApAtoms * kApAtom;       // 16 KB: the gathered digits of a chunk
constexpr int kApStages = 5;
constexpr int kApSmem = kApStages * (kApH + kApRows) + 1024;
constexpr int kXGroup = kApAtoms * 128;               // 512 bytes: a row's digits of 32 states
constexpr int kApCols = kApLevels * OZ_H;             // 224

// Seven balanced base-256 digits of v 2^(8 - e), rounded to 48 fractional bits;
// as digits6, which has 40.
__device__ __forceinline__ void digits7(double v, int e, float* d) {
  const int hi = __double2hiint(v);
  const uint32_t lo = (uint32_t)__double2loint(v);
  const int E = (hi >> 20) & 0x7FF;
  if (E == 0x7FF) {
#pragma unroll
    for (int i = 0; i < kApDigits; ++i) d[i] = __int_as_float(0x7fc00000);
    return;
  }
  unsigned long long X = 0;
  if (E > 0) {
    const unsigned long long M =
        ((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | lo;
    // v 2^(8-e) 2^48 = M 2^(E - 1075 + 56 - e); |v| < 2^e makes the shift >= -3
    const int rs = 1075 - 56 + e - E;
    if (rs <= 0) X = M << -rs;
    else if (rs < 63) X = (M + (1ull << (rs - 1))) >> rs;
  }
  // balanced digits, lowest first (see digits6), from the two 32-bit halves
  int t = (int)(uint32_t)(X & 0xFFFFFFu), g[kApDigits];
  g[6] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[5] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[4] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  t += (int)((X >> 24) & 0xFFFFFFu);
  g[3] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[2] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[1] = ((t + 128) & 255) - 128; t = (t + 128) >> 8;
  g[0] = t + (int)(X >> 48);                            // 0 .. 256
  const int sm = hi >> 31;                              // 0 or -1
#pragma unroll
  for (int i = 0; i < kApDigits; ++i) d[i] = (float)((g[i] ^ sm) - sm);
}

// B operand (slots x states, states contiguous) in the 128-byte swizzle layout,
// pieces of 128 bytes x 16 slots 2 KB apart (spmm_umma.cu)
__device__ __forceinline__ uint64_t gathered_desc(uint32_t addr) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)(kApAtom >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// tile * 128 + lane of each row
__global__ void k_oz_tile_rows(const int* __restrict__ rowmap, int64_t n, int* __restrict__ urow) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && rowmap[i] >= 0) urow[rowmap[i]] = (int)i;
}

struct OzCut {
  const int64_t* gptr;        // row groups: slots, columns, values
  const int* gcol;
  const double* v64;
  const int64_t* tptr;        // tiles
  const int* tcol;
  const int* urow;
  int* he;                    // largest biased exponent of each tile row
  unsigned char* hd;          // digit blocks of tiles [t0, t1), zero
  int64_t n;
  int t0, t1;
};

// A block takes a row group, a thread every 32nd slot of one of its rows: the
// row's scale, then its values' digits, each at the place that its column has
// in the list of the row's tile (both lists are sorted: a search from the place
// of the value before).
__global__ void __launch_bounds__(256) k_oz_cut_rows(const OzCut a) {
  __shared__ int top[8];
  const int64_t first = (int64_t)blockIdx.x * 8;
  bool any = false;                              // the same for all threads
  for (int64_t i = first; i < min(first + 8, a.n); ++i) {
    const int t = __ldg(a.urow + i) >> 7;
    any |= t >= a.t0 && t < a.t1;
  }
  if (!any) return;
  const int64_t s0 = a.gptr[blockIdx.x];
  const int ns = (int)(a.gptr[blockIdx.x + 1] - s0), r = threadIdx.x & 7;
  const int64_t row = first + r;
  if (threadIdx.x < 8) top[r] = 0;
  __syncthreads();
  int m = 0;
  for (int s = threadIdx.x >> 3; s < ns; s += 32)
    m = max(m, (__double2hiint(__ldg(a.v64 + (s0 + s) * 8 + r)) >> 20) & 0x7FF);
  atomicMax(&top[r], m);
  __syncthreads();
  if (row >= a.n) return;
  const int ur = a.urow[row], lane = ur & 127, e = exp_of_bits(top[r]);
  if ((ur >> 7) < a.t0 || (ur >> 7) >= a.t1) return;
  if (threadIdx.x < 8) a.he[ur] = top[r];
  const int64_t t0 = a.tptr[ur >> 7];
  const int nt = (int)(a.tptr[(ur >> 7) + 1] - t0);
  unsigned char* out = a.hd + (t0 - a.tptr[a.t0]) / OZ_K * kApH + (lane >> 3) * 256 + (lane & 7) * 16;
  int from = 0;
  for (int s = threadIdx.x >> 3; s < ns; s += 32) {
    const double v = __ldg(a.v64 + (s0 + s) * 8 + r);
    if (((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) == 0) continue;
    const int col = __ldg(a.gcol + s0 + s);
    int lo = from, hi = nt;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(a.tcol + t0 + mid) < col) lo = mid + 1;
      else hi = mid;
    }
    from = lo;
    float d[kApDigits];
    digits7(v, e, d);
    unsigned char* o = out + (int64_t)(lo >> 4) * kApH + ((lo >> 3) & 1) * 128 + (lo & 7) * 2;
#pragma unroll
    for (int i = 0; i < kApDigits; ++i)
      *reinterpret_cast<__nv_bfloat16*>(o + i * kPlA) = __float2bfloat16_rn(d[i]);
  }
}

// Digits of the block's rows: eight states of a row a thread.
__global__ void __launch_bounds__(256) k_oz_cut_states(const double* __restrict__ x, int64_t rows,
                                                       int k, int64_t ld, int groups,
                                                       const int* __restrict__ xe,
                                                       unsigned char* __restrict__ xd) {
  const int64_t total = rows * groups * 4;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * 256) {
    const int64_t r = i / (groups * 4);
    const int c = (int)(i - r * (groups * 4)) * 8;
    const double* p = x + r * ld + c;
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      double2 q = make_double2(0.0, 0.0);
      if (c + j + 1 < k) q = __ldg(reinterpret_cast<const double2*>(p + j));   // ld is a multiple of 8
      else if (c + j < k) q.x = __ldg(p + j);
      v[j] = q.x;
      v[j + 1] = q.y;
    }
    uint32_t w[kApDigits][4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float d0[kApDigits], d1[kApDigits];
      digits7(v[j], c + j < k ? exp_of_bits(__ldg(xe + c + j)) : 0, d0);
      digits7(v[j + 1], c + j + 1 < k ? exp_of_bits(__ldg(xe + c + j + 1)) : 0, d1);
#pragma unroll
      for (int d = 0; d < kApDigits; ++d) w[d][j / 2] = pack_bf16(d0[d], d1[d]);
    }
    unsigned char* o = xd + (r * groups + (c >> 5)) * kXGroup + (c & 31) * 2;
#pragma unroll
    for (int d = 0; d < kApDigits; ++d)
      *reinterpret_cast<uint4*>(o + d * (OZ_H * 2)) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
  }
}

struct OzApply {
  const int64_t* tptr;
  const int* tcol;
  const int* rowmap;
  const int* lptr;            // tiles of each of `ctas` CTAs (spmm_umma.cu)
  const int* litem;
  int ctas, par, nblk;        // column blocks of 64 states
  int t0, t1;                 // tiles whose digits hd holds
  const unsigned char* hd;
  const int* he;
  const unsigned char* xd;
  const int* xe;
  int groups;                 // of 32 states in a row of xd
  double* dst;
  int64_t ld;
  int k;
  int* err;
};

// the CTA's items, as in k_cheb_umma; f returns false to stop
template <typename F>
__device__ __forceinline__ void apply_items(const OzApply& a, F f) {
  const int q = blockIdx.x / a.ctas, g = blockIdx.x - q * a.ctas;
  bool flip = false;
  for (int b = q; b < a.nblk; b += a.par, flip = !flip) {
    const int j = flip ? a.ctas - 1 - g : g, e = __ldg(a.lptr + j + 1);
    for (int i = __ldg(a.lptr + j); i < e; ++i) {
      const int tile = __ldg(a.litem + i);
      if (tile >= a.t0 && tile < a.t1 && !f(tile, b)) return;
    }
  }
}

// seven 4-column tensor-memory loads `step` columns apart and one wait
__device__ __forceinline__ void tmem_ld4x7(uint32_t a, uint32_t step, float (*v)[4]) {
  uint32_t r[28];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%28];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%29];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%30];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12,%13,%14,%15}, [%31];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16,%17,%18,%19}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20,%21,%22,%23}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%24,%25,%26,%27}, [%34];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27])
      : "r"(a), "r"(a + step), "r"(a + 2 * step), "r"(a + 3 * step), "r"(a + 4 * step),
        "r"(a + 5 * step), "r"(a + 6 * step)
      : "memory");
#pragma unroll
  for (int L = 0; L < kApLevels; ++L)
#pragma unroll
    for (int j = 0; j < 4; ++j) v[L][j] = __uint_as_float(r[L * 4 + j]);
}

__global__ void __launch_bounds__(kApThreads, 1) k_oz_apply(const OzApply a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
  unsigned char* hring = smem + kApStages * kApRows;
  __shared__ __align__(8) uint64_t full[kApStages], empty[kApStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t fin[2];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t landed;                                 // chunks whose copies are there
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(su32(&tmem_slot)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int s = 0; s < kApStages; ++s) {
      bar_init(&full[s], 2);                                  // H's copy, the gathering warp
      bar_init(&empty[s], 2);
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
    // ---- H: the digit block of chunk q into stage q % kApStages
    if (lane == 0) {
      uint64_t pol_stream;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_stream));
      uint32_t q = 0;
      const int64_t h0 = __ldg(a.tptr + a.t0) / OZ_K;
      apply_items(a, [&](int tile, int) {
        const int64_t c0 = __ldg(a.tptr + tile) / OZ_K - h0, c1 = __ldg(a.tptr + tile + 1) / OZ_K - h0;
        for (int64_t c = c0; c < c1; ++c, ++q) {
          const int s = q % kApStages;
          if (q >= kApStages && !bar_wait(&empty[s], (q / kApStages - 1) & 1, abrt, 0)) {
            ok = false;
            return false;
          }
          const uint32_t fb = su32(&full[s]);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                       "r"(kApH) : "memory");
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
              " [%0], [%1], %2, [%3], %4;"
              ::"r"(su32(hring + s * kApH)), "l"(a.hd + c * kApH), "r"(kApH), "r"(fb),
                "l"(pol_stream) : "memory");
        }
        return true;
      });
      // on abort, let the copies already issued land: the gathering warps
      // arrive for theirs before they stop
      if (!ok)
        for (uint32_t r = (q > kApStages ? q - kApStages : 0); r < q; ++r)
          bar_drain(&full[r % kApStages], (r / kApStages) & 1);
    }
  } else if (warp == 2) {
    // ---- chunks landed, in order
    if (lane == 0) {
      uint32_t q = 0;
      apply_items(a, [&](int tile, int) {
        const int nq = (int)((__ldg(a.tptr + tile + 1) - __ldg(a.tptr + tile)) / OZ_K);
        for (int c = 0; c < nq; ++c, ++q) {
          if (!bar_wait(&full[q % kApStages], (q / kApStages) & 1, abrt, 0)) {
            ok = false;
            return false;
          }
          asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(su32(&landed)),
                       "r"(q + 1) : "memory");
        }
        return true;
      });
    }
  } else if (warp == 1 || warp == 3) {
    // ---- MMAs of one group of 32 states
    const int h = warp >> 1;
    if (elect_one()) {
      const uint32_t hbase = su32(hring), xbase = su32(smem) + (uint32_t)(h * kApAtoms * kApAtom);
      const uint32_t dcol = tmem + (uint32_t)(h * kApCols);
      uint32_t avail = 0, q = 0, gr = 0;                  // chunks, exact sums of this half
      apply_items(a, [&](int tile, int b) {
        const int nq = (int)((__ldg(a.tptr + tile + 1) - __ldg(a.tptr + tile)) / OZ_K);
        const bool on = (2 * b + h) * OZ_H < a.k;
        for (int j = 0; j < nq; ++j, ++q) {
          const int c = j % kGroupChunks, s = q % kApStages;
          if (on && c == 0 && gr > 0 && !bar_wait(&acc_empty[h], (gr - 1) & 1, abrt, 0)) {
            ok = false;
            return false;
          }
          for (int i = 0; i < kTcMaxWait && avail <= q; ++i) {
            asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(avail)
                         : "r"(su32(&landed)) : "memory");
            if (avail > q || *abrt) break;
          }
          if (avail <= q) {
            ok = false;
            *abrt = 1;
            return false;
          }
          if (!on) {
            // this thread's MMAs of the block before may still run: the commit
            // frees the stage after them, so that `empty` completes in the order
            // of the chunks, which the gathering warps' parity waits need
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(su32(&empty[s])) : "memory");
            continue;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t db = gathered_desc(xbase + (uint32_t)(s * kApRows));
#pragma unroll
          for (int i = 0; i < kApDigits; ++i) {
            const uint64_t da = kmajor_desc(hbase + (uint32_t)(s * kApH + i * kPlA));
            const uint32_t acc = (c > 0 || i > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                ::"r"(dcol + (uint32_t)(i * OZ_H)), "l"(da), "l"(db),
                  "r"(idesc_oz(OZ_H * (kApDigits - i)) | (1u << 16)), "r"(acc));
          }
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
              ::"r"(su32(&empty[s])) : "memory");
          if (c == kGroupChunks - 1 || j == nq - 1) {
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(su32(&acc_full[h])) : "memory");
            ++gr;
          }
        }
        return true;
      });
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
          ::"r"(su32(&fin[h])) : "memory");
      bar_drain(&fin[h], 0);
    }
  } else if (warp >= kEpiWarp0 + 2 * kEpiWarps) {
    // ---- gathered rows, chunk q to warp q % kApGather (see k_cheb_umma)
    const int pw = warp - kEpiWarp0 - 2 * kEpiWarps, lr = lane >> 3, lj = lane & 7;
    uint64_t pol_keep;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_keep));
    const uint32_t sw0 = (uint32_t)(lr * 128 + ((lj ^ lr) << 4));
    const uint32_t sw1 = (uint32_t)((4 + lr) * 128 + ((lj ^ (4 + lr)) << 4));
    const int64_t xrow = (int64_t)a.groups * kXGroup;
    int pending = -1;                                         // stage of the chunk in flight
    auto land = [&]() {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&full[pending]);
      pending = -1;
    };
    uint32_t q0 = 0, q = pw;
    apply_items(a, [&](int tile, int b) {
      const int64_t t0 = __ldg(a.tptr + tile);
      const int nq = (int)((__ldg(a.tptr + tile + 1) - t0) / OZ_K);
      const int atoms = (2 * b + 1) * OZ_H < a.k ? 2 * kApAtoms : kApAtoms;
      const int* colp = a.tcol + t0 + (lane & 15);
      const unsigned char* xb = a.xd + (int64_t)b * 2 * kXGroup + 16 * lj;
      const uint32_t end = q0 + (uint32_t)nq;
      int next = q < end ? __ldg(colp + (int64_t)(q - q0) * OZ_K) : 0;
      for (; q < end; q += kApGather) {
        const int mine = next;
        next = q + kApGather < end ? __ldg(colp + (int64_t)(q + kApGather - q0) * OZ_K) : 0;
        const unsigned char* xs[4];
#pragma unroll
        for (int rq = 0; rq < 4; ++rq)
          xs[rq] = xb + (int64_t)__shfl_sync(0xffffffffu, mine, 4 * rq + lr) * xrow;
        const int s = q % kApStages;
        if (q >= kApStages) {
          const uint32_t par = (q / kApStages - 1) & 1;
          int is = 0;
          if (lane == 0) is = bar_test(&empty[s], par);
          is = __shfl_sync(0xffffffffu, is, 0);
          if (!is) {
            if (pending >= 0) {
              asm volatile("cp.async.wait_group 0;" ::: "memory");
              land();
            }
            bool w = true;
            if (lane == 0) w = bar_wait(&empty[s], par, abrt, 0);
            ok = __shfl_sync(0xffffffffu, w, 0);
            if (!ok) return false;
          }
        }
        const uint32_t sb = su32(smem) + (uint32_t)(s * kApRows);
#pragma unroll
        for (int rq = 0; rq < 4; ++rq) {
          const uint32_t drow = sb + (rq & 1 ? sw1 : sw0) + (rq >> 1) * 1024;
#pragma unroll
          for (int t = 0; t < 2 * kApAtoms; ++t)
            if (t < atoms && (t % kApAtoms < kApAtoms - 1 || lj < 4))       // no eighth digit
              asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;"
                           ::"r"(drow + (uint32_t)(t * kApAtom)), "l"(xs[rq] + t * 128), "l"(pol_keep)
                           : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (pending >= 0) {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          land();
        }
        pending = s;
      }
      q0 = end;
      return true;
    });
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (pending >= 0) land();
  } else {
    // ---- folds of a group of states, as in k_oz_mma, four columns at a time
    const int h = (warp - kEpiWarp0) / kEpiWarps, qd = warp & 3;
    const int cb = (((warp - kEpiWarp0) >> 2) & 1) * OZ_E;
    const uint32_t acol = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(h * kApCols + cb);
    uint32_t gr = 0;
    apply_items(a, [&](int tile, int b) {
      const int col0 = (2 * b + h) * OZ_H + cb;
      if ((2 * b + h) * OZ_H >= a.k) return true;
      const int nq = (int)((__ldg(a.tptr + tile + 1) - __ldg(a.tptr + tile)) / OZ_K);
      const int ng = (nq + kGroupChunks - 1) / kGroupChunks;
      float hi[OZ_E], lo[OZ_E];
#pragma unroll
      for (int c = 0; c < OZ_E; ++c) { hi[c] = 0.f; lo[c] = 0.f; }
      for (int t = 0; t < ng; ++t, ++gr) {
        bool wt = true;
        if (lane == 0) wt = bar_wait(&acc_full[h], gr & 1, abrt, 32);
        ok = __shfl_sync(0xffffffffu, wt, 0);
        if (!ok) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int cc = 0; cc < OZ_E; cc += 4) {
          float S[kApLevels][4];
          tmem_ld4x7(acol + cc, OZ_H, S);
          if (cc + 4 == OZ_E) {              // the last loads are in registers: release the buffer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&acc_empty[h]);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float f = S[0][i], l = 0.f;
            float sc = 1.f / 256.f;
#pragma unroll
            for (int L = 1; L < kApLevels; ++L, sc *= (1.f / 256.f)) {
              const float u = S[L][i] * sc;
              const float h2 = f + u;
              const float bv = h2 - f;
              l += (f - (h2 - bv)) + (u - bv);
              f = h2;
            }
            const float sum = hi[cc + i] + f;
            const float bv = sum - hi[cc + i];
            lo[cc + i] += (hi[cc + i] - (sum - bv)) + (f - bv) + l;
            hi[cc + i] = sum;
          }
        }
      }
      const int64_t ur = (int64_t)tile * OZ_M + qd * 32 + lane;
      const int row = __ldg(a.rowmap + ur);
      if (row < 0) return true;
      const int em = exp_of_bits(__ldg(a.he + ur)) - 16;
      double* o = a.dst + row * a.ld + col0;
#pragma unroll
      for (int c = 0; c < OZ_E; c += 2) {
        double v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          v[u] = scaled_sum(hi[c + u], lo[c + u],
                            em + exp_of_bits(__ldg(a.xe + min(col0 + c + u, a.k - 1))));
        if (col0 + c + 1 < a.k)
          *reinterpret_cast<double2*>(o + c) = make_double2(v[0], v[1]);
        else if (col0 + c < a.k)
          o[c] = v[0];
      }
      return true;
    });
  }
  __syncwarp();
  if (!ok) {
    *abrt = 1;
    atomicExch(a.err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

}  // namespace

bool oz_apply_supported(const ttg_op* op, int k) {
  const UmmaOp& U = op->umma;
  if (getenv("TTG_DISABLE_OZGEMM")) return false;
  if (U.n_tiles == 0 || op->tc_disabled || op->rg.n_groups == 0) return false;
  return k > 0;
}

// dst = H src; src's rows n .. hold W.  H's digits are cut for slabs of tiles
// that fit into a 32nd of the memory: the whole operator up to about 64,000
// functions, whose digits are then kept for the next product with the same
// values; a larger one is cut again for every product (a tenth of its time).
// TTG_OOM (before any work): no room.
ttg_status launch_oz_apply(ttg_op* op, const double* src, double* dst, int k) {
  UmmaOp& U = op->umma;
  OzRows& Z = op->ozrows;
  cudaStream_t st = op->stream;
  const int64_t trows = U.n_tiles * OZ_M;
  const int64_t rows = op->n + (op->C.nnz > 0 ? op->nproj : 0);
  const int groups = (k + OZ_H - 1) / OZ_H;
  auto grow = [&](DevBuf& b, size_t need) -> ttg_status {
    return b.bytes >= need ? TTG_OK : b.alloc(need);
  };
  if (Z.slabs.empty()) {
    size_t free = 0, total = 0;
    TTG_CUDA_TRY(cudaMemGetInfo(&free, &total));
    const int64_t most = std::max<int64_t>((int64_t)(total / 32 / kApH), 1);
    std::vector<int64_t> tp(U.n_tiles + 1);
    TTG_CUDA_TRY(cudaMemcpyAsync(tp.data(), U.tptr.p, tp.size() * 8, cudaMemcpyDeviceToHost, st));
    TTG_CUDA_TRY(cudaStreamSynchronize(st));
    std::vector<int> slabs(1, 0);
    for (int64_t t = 0; t < U.n_tiles; ++t) {
      if ((tp[t + 1] - tp[t]) / OZ_K > most) return TTG_OOM;
      if ((tp[t + 1] - tp[slabs.back()]) / OZ_K > most) slabs.push_back((int)t);
    }
    slabs.push_back((int)U.n_tiles);
    Z.most = 0;
    for (size_t i = 1; i < slabs.size(); ++i)
      Z.most = std::max<int64_t>(Z.most, (tp[slabs[i]] - tp[slabs[i - 1]]) / OZ_K);
    Z.slabs = slabs;
  }
  TTG_TRY(grow(Z.hd, std::max<size_t>((size_t)Z.most * kApH, 16)));
  if (grow(Z.xd, (size_t)rows * groups * kXGroup) != TTG_OK) {
    Z.hd.release();
    Z.cut = false;
    return TTG_OOM;
  }
  TTG_TRY(grow(Z.xe, (size_t)op->ld * sizeof(int)));
  int* err = nullptr;
  TTG_TRY(error_word(st, op->oz, &err));
  if (!Z.urow.p) {
    TTG_TRY(grow(Z.urow, (size_t)op->n * sizeof(int)));
    k_oz_tile_rows<<<(unsigned)((trows + 255) / 256), 256, 0, st>>>(U.rowmap.as<int>(), trows,
                                                                  Z.urow.as<int>()); TTG_COUNT();
    TTG_LAUNCHED(op);
  }
  if (!Z.he.p) TTG_TRY(grow(Z.he, (size_t)trows * sizeof(int)));
  TTG_CUDA_TRY(cudaMemsetAsync(Z.xe.p, 0, (size_t)k * sizeof(int), st));
  OzSlices S{};
  S.o[0] = OzOperand{src, k, rows, 1, op->ld};
  S.ebits[0] = Z.xe.as<int>();
  const int64_t kb = std::max<int64_t>(64, (rows + 255) / 256);
  k_rowexp_rows<<<dim3((unsigned)((k + 31) / 32), (unsigned)((rows + kb - 1) / kb), 1), dim3(32, 8), 0,
                  st>>>(S, kb, nullptr, 0); TTG_COUNT();
  TTG_LAUNCHED(op);
  k_oz_cut_states<<<(unsigned)std::min<int64_t>((rows * groups * 4 + 255) / 256, 152 * 16), 256, 0, st>>>(
      src, rows, k, op->ld, groups, Z.xe.as<int>(), Z.xd.as<unsigned char>()); TTG_COUNT();
  TTG_LAUNCHED(op);
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_oz_apply, cudaFuncAttributeMaxDynamicSharedMemorySize, kApSmem);
  });
  if (attr != cudaSuccess) return TTG_CUDA_ERR;
  OzApply a{};
  a.tptr = U.tptr.as<int64_t>();
  a.tcol = U.tcol.as<int>();
  a.rowmap = U.rowmap.as<int>();
  a.lptr = U.lptr.as<int>();
  a.litem = U.litem.as<int>();
  a.nblk = (k + OZ_N - 1) / OZ_N;
  a.ctas = U.ctas;
  a.par = std::max(1, std::min(a.nblk, kSMs / U.ctas));
  a.hd = Z.hd.as<unsigned char>();
  a.he = Z.he.as<int>();
  a.xd = Z.xd.as<unsigned char>();
  a.xe = Z.xe.as<int>();
  a.groups = groups;
  a.dst = dst;
  a.ld = op->ld;
  a.k = k;
  a.err = err;
  for (size_t i = 1; i < Z.slabs.size(); ++i) {
    a.t0 = Z.slabs[i - 1];
    a.t1 = Z.slabs[i];
    if (!Z.cut) {
      TTG_CUDA_TRY(cudaMemsetAsync(Z.hd.p, 0, Z.hd.bytes, st));
      TTG_CUDA_TRY(cudaMemsetAsync(Z.he.as<int>() + (int64_t)a.t0 * OZ_M, 0,
                                   (size_t)(a.t1 - a.t0) * OZ_M * sizeof(int), st));
      const OzCut c{op->rg.gptr.as<int64_t>(), op->rg.gcol.as<int>(), op->rg.v64.as<double>(),
                    U.tptr.as<int64_t>(), U.tcol.as<int>(), Z.urow.as<int>(), Z.he.as<int>(),
                    Z.hd.as<unsigned char>(), op->n, a.t0, a.t1};
      k_oz_cut_rows<<<(unsigned)op->rg.n_groups, 256, 0, st>>>(c); TTG_COUNT();
      TTG_LAUNCHED(op);
      Z.cut = Z.slabs.size() == 2;
    }
    k_oz_apply<<<(unsigned)(a.ctas * a.par), kApThreads, kApSmem, st>>>(a); TTG_COUNT();
    TTG_LAUNCHED(op);
  }
  return fake_timeout(st, err);
}

}  // namespace ttg
