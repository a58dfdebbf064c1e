// Chebyshev filter degrees on the fifth-generation tensor cores
// (tcgen05.mma, accumulator in tensor memory): Ynew = alpha (H Y) + beta Y +
// delta X (ChebyShevFilter.cc:97-170).  FP32 degrees run FP32-accurate on
// FP16 MMAs (two scaled terms, below); BF16 degrees run one BF16 product.
//
// Tiles.  128 rows per tile (a 4 x 4 x 8 block of the Tucker index, or 128
// consecutive rows without Tucker ranks); the tile's sorted column union is
// padded to chunks of 16 slots.  A chunk is one MMA step: M = 128 rows,
// N = k states, K = 16 slots.
//
// Precision (FP32 degrees).  Every row of H and every column of the block is
// scaled by a power of two (undone, exactly, in the epilogue) and each scaled
// FP32 value is split into two FP16 terms v = v0 + v1, |v1| <= 2^-11 |v|, what
// is left below 2^-22 |v|, or below the half of FP16's smallest step where v1
// runs out of exponents: 2^-39 of the column's largest value, 2^-35 of the
// row's (2^-29 for new values).  The product is
// accumulated in FP32 from v0w0, v0w1 and v1w0; v1w1 is below 2^-22 |v w|.
// An accumulation step of the tensor core truncates, the larger part of a
// degree's error: three steps per 16 slots instead of the six of a three-term
// BF16 split.  Relative error of 8 degrees against FP64, before and
// now: 1.3e-5 and 3.7e-6 (1,728 functions, 24 states), 1.8e-5 and 9.7e-6 (8,000,
// 160), 2.2e-5 and 1.9e-5 (64,000, 400).
//  - Block columns: the largest |Y| of each column comes from the epilogue of
//    the degree before (k_colmax for the first one), and puts it in
//    [2^14, 2^15).  A projector's W_a is at most L1(Cd_a) times that; its
//    power of two is taken out of W_a and put into the entries of C^T.
//  - H rows: the largest entry of a row, C^T's with 2^L included, is put in
//    [2^10, 2^11) when the operator is built.  New values keep the row's scale
//    while they stay in [2^4, 2^15), sixteen times up and 64 down; the first
//    potential of an SCF moves a row's largest entry by a factor of 6 at most.
//    k_umma_rescale gives the other rows a new scale.  (C^T's entries leave H's
//    a coarser step only where L1(Cd_a) is large, and by less than the FP32
//    rounding of the W_a that they multiply.)
//
// Data movement per chunk.
//  - H: the chunk's planes (128 x 16 values each, already in the canonical
//    K-major no-swizzle layout of the MMA operand): two FP16 planes, 8 KB, or
//    one BF16 plane, 4 KB.  The chunks of a tile are contiguous, so a stage of
//    SC chunks is one 16 KB bulk asynchronous copy (TMA, L2 evict-first).
//  - Y: the 16 source rows are gathered from two FP16 planes of the block
//    (written by k_umma_prepare before the launch), or from the BF16 block as
//    it is, with 16-byte cp.async copies (L2 evict-last: rows are re-read by
//    many tiles), in the MN-major operand layout with the 128-byte swizzle:
//    8 lanes read one whole 128-byte piece of a row, so one instruction moves
//    four rows.
// A stage is SC = 2 chunks (FP32) or 4 (BF16): its commit and the round trip
// through its barriers are paid once for all of it.
// Persistent CTAs, one per SM, each with a list of tiles (each_item).  Roles:
//  - warp 4, one thread: the H copies, up to a whole ring ahead;
//  - warps 7-16: the row gathers, whole chunks in turn; a warp waits for its
//    own copies and fences them for the async proxy before it arrives;
//  - warp 6, one thread: waits for each stage's "full" mbarrier in order and
//    publishes the count of ready stages in shared memory;
//  - warp 5, one elected thread: three MMAs (one for BF16) a chunk and one
//    commit (to the stage's "done" mbarrier) per stage.  Between the stages of
//    an item it waits on no mbarrier: such a wait queues behind its
//    outstanding MMAs (about 0.1 us);
//  - warps 0-3 (one per 32 TMEM lanes): read an item's accumulator from tensor
//    memory and apply the recurrence in FP32, while the next item's MMAs fill
//    the other accumulator.
// Blocks wider than one MMA (N <= 256) are column blocks of one launch, a CTA's
// tiles of one block after those of the one before, with its list exchanged for
// one from the other end of the order of loads in every second one.
// Few tiles (FP32): where the tiles would leave half of the SMs without work,
// a cluster of 2, 4 or 8 CTAs (as many as are resident at once) shares a tile,
// each a part of its chunks; the accumulators meet in shared memory and every CTA finishes its share of the
// rows.  BF16 degrees keep one CTA a tile: their sums are rounded to 8 bits at
// every degree, so the order of a sum is part of the result.
// What bounds it (clock counts of its threads): at 160 states a stage takes 670
// clocks, in which H streams at 6.9 TB/s over the SMs: HBM, plus the CTAs'
// uneven ends; at 240 states a column block 820, of which the MMAs need 720.
// Stages of half the size: 520 instead of 400 us and 1,130 instead of 1,018.
// One degree, three-term split with a CTA a tile -> now:
//   64,000 functions, 160 states, FP32: 728 -> 400 us (H's 2.0 GB: 294 us)
//   the same, BF16: 396 -> 183 us (147 us)
//   32,768 functions, 1,200 states, FP32: 2,425 -> 1,018 us
//   1,728 functions, 24 states, FP32 (clusters of 4): 63 (mma.sync) -> 11 us
// Of these, a stage of several chunks and two terms gave 728 -> 514; the
// epilogue beside the next item's MMAs (22 % of the kernel until then), the
// elected MMA thread and addresses made before the wait the rest.
// Every wait (mbarrier or the ready count) is bounded; a wait that runs out
// sets an error word.

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>
#ifdef _OPENMP
#include <omp.h>
#endif

#include "ttg_internal.cuh"

namespace ttg {
namespace {

constexpr int UR = 128;                       // rows per tile (MMA M)
constexpr int UK = 16;                        // slots per chunk (MMA K)
constexpr int PLANE_ELEMS = UR * UK;          // 2048 16-bit values = 4096 bytes
constexpr int kMaxStages = 12;
constexpr int kSmemBudget = 227 * 1024 - 2048;   // dynamic; the kernel has 2 KB of its own
constexpr int kEpiWarps = 4;                  // warps 0-3: read the accumulators
constexpr int kHWarp = 4;                     // one thread copies the H blocks
constexpr int kMmaWarp = 5;                   // one thread issues the MMAs
constexpr int kWaitWarp = 6;                  // waits for full stages on the MMA warp's behalf
constexpr int kFirstBWarp = 7;                // the rest gather the block's rows
constexpr int kBWarps = 10;
constexpr int kThreads = 32 * (kFirstBWarp + kBWarps);
constexpr int kMaxCtas = 152;
constexpr int kMaxWait = 1 << 20;
constexpr int kRowExp = 10;                   // a scaled row's largest entry: [2^10, 2^11)
constexpr float kRowLow = 16.f;               // smallest one that keeps its row's scale
constexpr int kAtom = 64;                     // states per 128-byte swizzle row
constexpr int kAtomBytes = 16 * 128;          // one atom of a chunk: 16 slot rows x 128 bytes

// Canonical no-swizzle layouts (8 x 16-byte core matrices, 128 bytes each):
// core matrices 128 bytes apart along K and 256 bytes apart along M / N.
__host__ __device__ inline int a_elem(int m, int s) {
  return (m >> 3) * 128 + (s >> 3) * 64 + (m & 7) * 8 + (s & 7);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)(128 >> 4) << 16;        // leading byte offset: next core matrix along K
  d |= (uint64_t)(256 >> 4) << 32;        // stride byte offset: next core matrix along M/N
  d |= (uint64_t)1 << 46;                 // descriptor version
  return d;                               // base offset 0, no swizzle
}

// B operand (slots x states, states contiguous) in the 128-byte swizzle
// layout: per 64-state atom 16 slot rows of 128 bytes, the 16-byte piece j of
// row s stored at piece j ^ (s % 8); rows 8-15 1024 bytes after rows 0-7
// (stride byte offset), atoms 2048 bytes apart (leading byte offset).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)(kAtomBytes >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;                 // 128-byte swizzle
  return d;
}

// kind::f16 instruction descriptor: BF16 x BF16 or FP16 x FP16 -> FP32, A
// K-major, B MN-major
__device__ __forceinline__ uint32_t instr_desc(bool bf16, int m, int n) {
  return (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
}

__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity) {
  for (int i = 0; i < kMaxWait; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ int mbar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return (int)ok;
}

// For waits off the critical path: a thread that polls an mbarrier without
// pause slows the mbarrier operations of the threads that are on it.
__device__ __forceinline__ bool mbar_wait_idle(uint64_t* b, uint32_t parity, int ns) {
  for (int i = 0; i < kMaxWait; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
    __nanosleep(ns);
  }
  return false;
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Power of two that puts a largest value of bits `u` (|v| as an integer) into
// [2^14, 2^15), and its inverse; 1 for zero.  Values below 2^-112 stop at 2^126.
__device__ __forceinline__ float scale_up(uint32_t u) {
  if (u == 0) return 1.f;
  return __uint_as_float((uint32_t)min(253, 127 + 14 - ((int)(u >> 23) - 127)) << 23);
}
__device__ __forceinline__ float scale_down(uint32_t u) {
  if (u == 0) return 1.f;
  return __uint_as_float((uint32_t)max(1, 127 - 14 + ((int)(u >> 23) - 127)) << 23);
}

// |v| as an integer (ordered like the values); 0 for infinities and NaN
__device__ __forceinline__ uint32_t finite_bits(float v) {
  const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
  return u < 0x7f800000u ? u : 0u;
}

__device__ __forceinline__ void split_half(float v, __half& a, __half& b) {
  a = __float2half_rn(v);
  b = __float2half_rn(v - __half2float(a));
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ float4 peer_load(uint32_t addr, uint32_t rank) {
  uint32_t r;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r) : "memory");
  return v;
}

struct UmmaArgs {
  const int64_t* tptr;
  const int* tcol;
  const int* rowmap;
  const int* order;
  const uint16_t* hpl;        // FP16: [chunk][2][2048], BF16: [chunk][2048]
  const uint16_t* xpl;        // FP16: [2][rows][ps], BF16: the block
  int64_t pstride;            // of the two planes
  int ps;                     // row stride of xpl
  const float* rscale;        // FP16: inverse scale of each tile row
  const uint32_t* cmax;       // FP16: largest |Y| of each column (bits)
  uint32_t* cmax_next;        // and of each column of the result
  int k, kb;                  // states, and states of a column block (multiple of 16)
  int64_t ld;
  float alpha, beta, delta;
  uint32_t tmem_cols;
  int stages;
  int split;                  // CTAs (of a cluster) per tile
  int n_tiles;
  const int* lptr;            // tiles of each of `ctas` CTAs: litem[lptr[j] .. lptr[j + 1])
  const int* litem;
  int ctas, par, nblk;        // column blocks b, b + par, .. go to the same CTAs
  int* err;
};

// One CTA's items: tiles of a column block.  A split tile is the one item of
// its cluster; else the CTA's list of tiles (lptr, litem), for one column
// block after the other, in every second one the list of the CTA at the other
// end of the order of loads.
template <typename F>
__device__ __forceinline__ void each_item(const UmmaArgs& a, F f) {
  if (a.split > 1) {
    const int w = blockIdx.x / a.split;
    f(__ldg(a.order + w % a.n_tiles), w / a.n_tiles);
    return;
  }
  const int q = blockIdx.x / a.ctas, g = blockIdx.x - q * a.ctas;
  bool flip = false;
  for (int b = q; b < a.nblk; b += a.par, flip = !flip) {
    const int j = flip ? a.ctas - 1 - g : g, e = __ldg(a.lptr + j + 1);
    for (int i = __ldg(a.lptr + j); i < e; ++i) f(__ldg(a.litem + i), b);
  }
}

struct UmmaItem {
  int64_t c_first;            // first chunk
  int nch;                    // chunks
  int cb, kk, kv;             // first state, states of the MMA, states that exist
  __device__ __forceinline__ UmmaItem(const UmmaArgs& a, int tile, int b) {
    const int part = blockIdx.x % a.split;
    const int64_t t0 = __ldg(a.tptr + tile) / UK;
    const int n = (int)(__ldg(a.tptr + tile + 1) / UK - t0), per = (n + a.split - 1) / a.split;
    c_first = t0 + min(part * per, n);
    nch = max(0, min(per, n - part * per));
    cb = b * a.kb;
    kk = min(a.kb, ((a.k + 15) & ~15) - cb);
    kv = min(kk, a.k - cb);
  }
};

// F32: FP32 degree (two FP16 terms of the scaled H and block, three
// products); else BF16 degree (H rounded to BF16, the BF16 block itself, one
// product).  NA: 128-byte pieces of a gathered row.
template <bool F32, int NA>
__global__ void __launch_bounds__(kThreads)
    k_cheb_umma(const UmmaArgs a, const void* __restrict__ srcv, const void* xoldv, void* dstv) {
  using TIO = std::conditional_t<F32, float, __nv_bfloat16>;
  constexpr int P = F32 ? 2 : 1;              // planes
  constexpr int SC = F32 ? 2 : 4;             // chunks of a stage
  constexpr int HC = P * 2 * PLANE_ELEMS;     // H bytes of a chunk
  constexpr int HB = SC * HC;                 // and of a stage
  constexpr int BP = NA * kAtomBytes;         // one gathered plane of a chunk
  constexpr int BC = P * BP;                  // the gathered rows of a chunk
  const TIO* src = static_cast<const TIO*>(srcv);
  const TIO* xold = static_cast<const TIO*>(xoldv);
  TIO* dst = static_cast<TIO*>(dstv);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // the ring starts on a 1024-byte boundary (swizzle atoms; descriptor base
  // offset 0): per stage the gathered rows of SC chunks, and after all of
  // those the H blocks
  unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  // full[s]: the H copy by bytes and an arrival each from the H thread and the
  // warps of the stage's slots; done[s]: its MMAs have read it
  __shared__ __align__(8) uint64_t full[kMaxStages], done[kMaxStages];
  // accumulators: an item's MMAs are done, its sums have been read
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t ready;                 // stages that have filled
  __shared__ uint32_t cnew[256];             // shared tile: largest |result| of each column
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nst = a.stages;
  unsigned char* hring = smem + nst * SC * BC;
  const bool shared_tile = F32 && a.split > 1;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"(a.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < nst; ++s) {
      mbar_init(&full[s], 1 + SC);
      mbar_init(&done[s], 1);                    // one tcgen05.commit
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiWarps);
    }
    ready = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const uint32_t acc_cols = shared_tile ? 0u : a.tmem_cols / 2;
  bool ok = true;

  if (warp == kHWarp) {
    if (elect_one()) {
      uint64_t pol_stream;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_stream));
      int s = 0;
      uint32_t lap = 0;
      each_item(a, [&](int tile, int b) {
        const UmmaItem it(a, tile, b);
        for (int c = 0; c < it.nch; c += SC) {
          if (lap > 0) ok &= mbar_wait(&done[s], (lap - 1) & 1);
          const uint32_t fb = smem_u32(&full[s]);
          const int nc = min(SC, it.nch - c);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                       "r"(nc * HC) : "memory");
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
              " [%0], [%1], %2, [%3], %4;"
              ::"r"(smem_u32(hring + s * HB)), "l"(a.hpl + (it.c_first + c) * (P * PLANE_ELEMS)),
                "r"(nc * HC), "r"(fb), "l"(pol_stream)
              : "memory");
          if (++s == nst) {
            s = 0;
            ++lap;
          }
        }
      });
    }
  } else if (warp >= kFirstBWarp) {
    // gathered rows: slot t (of SC a stage) to warp t % np.  The addresses are
    // made before the wait for the slot; where the slot is free already, a warp
    // issues its copies before it waits for those of its chunk before.
    const int np = min(kBWarps, nst * SC);
    const int pw = warp - kFirstBWarp;
    if (pw < np) {
      // lane = row of a quad (lane / 8) x 16-byte piece of a 128-byte row
      // (lane % 8): one instruction reads four whole 128-byte rows and writes
      // four 128-byte rows of shared memory (128-byte swizzle: piece j of
      // slot row s lands at piece j ^ (s % 8))
      const int lr = lane >> 3, lj = lane & 7;
      uint64_t pol_keep;     // the block's rows are re-read by many tiles
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_keep));
      const uint32_t sw0 = (uint32_t)(lr * 128 + ((lj ^ lr) << 4));             // rows lr, 8 + lr
      const uint32_t sw1 = (uint32_t)((4 + lr) * 128 + ((lj ^ (4 + lr)) << 4)); // 4 + lr, 12 + lr
      const uint32_t ring = smem_u32(smem);
      uint32_t pending = ~0u;                    // full barrier of the chunk in flight
      auto land = [&]() {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(pending) : "memory");
        pending = ~0u;
      };
      int stage0 = 0;                            // stages before this item
      int t = pw;                                // this warp's next slot
      each_item(a, [&](int tile, int b) {
        const UmmaItem it(a, tile, b);
        const int nstage = (it.nch + SC - 1) / SC, base = stage0 * SC, end = (stage0 + nstage) * SC;
        stage0 += nstage;
        const int* colp = a.tcol + it.c_first * UK + (lane & 15);
        const uint16_t* xbase = a.xpl + it.cb + 8 * lj;
        bool on[NA];
#pragma unroll
        for (int q = 0; q < NA; ++q) on[q] = q * 64 + 8 * lj < it.kk;
        int next = t - base < it.nch ? __ldg(colp + (int64_t)(t - base) * UK) : 0;
        for (; t < end; t += np) {
          const int c = t - base;
          const int mine = next;
          next = c + np < it.nch ? __ldg(colp + (int64_t)(c + np) * UK) : 0;
          const uint16_t* xs[4];
#pragma unroll
          for (int rq = 0; rq < 4; ++rq)
            xs[rq] = xbase + (int64_t)__shfl_sync(0xffffffffu, mine, 4 * rq + lr) * a.ps;
          const int g = t / SC, lap = g / nst, s = g - lap * nst;
          const uint32_t sb = ring + (uint32_t)((s * SC + (t - g * SC)) * BC);
          if (lap > 0) {
            const uint32_t ph = (lap - 1) & 1;
            int free = 0;
            if (lane == 0) free = mbar_test(&done[s], ph);
            free = __shfl_sync(0xffffffffu, free, 0);
            if (!free) {
              if (pending != ~0u) {
                cp_async_wait<0>();
                land();
              }
              if (lane == 0) ok &= mbar_wait(&done[s], ph);
              __syncwarp();
            }
          }
          // a slot without a chunk (an item's last stage) is waited for and
          // arrived for as well: a warp's wait, a ring earlier at most, and the
          // MMAs' wait for the warp are what keep the parity unambiguous
          if (c >= it.nch) {
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[s])) : "memory");
            continue;
          }
#pragma unroll
          for (int rq = 0; rq < 4; ++rq) {
            const uint32_t drow = sb + (rq & 1 ? sw1 : sw0) + (rq >> 1) * 1024;
#pragma unroll
            for (int pl = 0; pl < P; ++pl) {
              const uint16_t* x = xs[rq] + pl * a.pstride;
#pragma unroll
              for (int q = 0; q < NA; ++q)
                if (on[q])
                  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;"
                               ::"r"(drow + (uint32_t)(pl * BP + q * kAtomBytes)), "l"(x + q * kAtom),
                                 "l"(pol_keep)
                               : "memory");
            }
          }
          cp_async_commit();
          if (pending != ~0u) {
            cp_async_wait<1>();
            land();
          }
          pending = smem_u32(&full[s]);
        }
      });
      cp_async_wait<0>();
      if (pending != ~0u) land();
    }
  } else if (warp == kWaitWarp) {
    // waits for each stage to fill, in order, and publishes the count of full
    // stages to the MMA thread: an mbarrier wait by the MMA-issuing thread
    // itself queues behind its outstanding MMAs (about 0.1 us)
    if (elect_one()) {
      int s = 0;
      uint32_t lap = 0, g = 0;
      each_item(a, [&](int tile, int b) {
        const UmmaItem it(a, tile, b);
        for (int c = 0; c < it.nch; c += SC) {
          ok &= mbar_wait(&full[s], lap & 1);
          asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(&ready)), "r"(++g)
                       : "memory");
          if (++s == nst) {
            s = 0;
            ++lap;
          }
        }
      });
    }
  } else if (warp == kMmaWarp) {
    // MMA thread: per chunk three MMAs (smallest products first) or one.
    // Elected, not lane 0: with the compiler aware of the single thread an MMA
    // takes about 50 clocks to issue instead of 100.
    if (elect_one()) {
      const uint64_t da_hi = smem_desc(0), db_hi = smem_desc_sw128(0);
      // descriptors hold the address within the CTA: in a cluster the upper bits
      // of a shared address are the CTA's rank
      const uint32_t a_first = (smem_u32(hring) & 0x3FFFF) >> 4, b_first = (smem_u32(smem) & 0x3FFFF) >> 4;
      const uint32_t done0 = smem_u32(&done[0]);
      int s = 0;
      uint32_t avail = 0, g = 0, n = 0;
      each_item(a, [&](int tile, int b) {
        const UmmaItem it(a, tile, b);
        const uint32_t idesc = instr_desc(!F32, UR, it.kk), d = tmem + (n & 1) * acc_cols;
        if (n >= 2) ok &= mbar_wait(&acc_empty[n & 1], ((n >> 1) - 1) & 1);
        uint32_t acc = 0u;
        for (int c = 0; c < it.nch; c += SC, ++g) {
          for (int i = 0; i < kMaxWait && avail <= g; ++i)
            asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(avail) : "r"(smem_u32(&ready))
                         : "memory");
          ok &= avail > g;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_lo = a_first + (uint32_t)(s * (HB >> 4));
          const uint32_t b_lo = b_first + (uint32_t)(s * SC * (BC >> 4));
#pragma unroll
          for (int j = 0; j < SC; ++j) {
            if (c + j >= it.nch) break;
            // (term of A, term of B): (0,1) (1,0) (0,0)
#pragma unroll
            for (int q = F32 ? 0 : 2; q < 3; ++q) {
              const uint64_t da = da_hi | (a_lo + j * (HC >> 4) + (q == 1 ? (2 * PLANE_ELEMS) >> 4 : 0));
              const uint64_t db = db_hi | (b_lo + j * (BC >> 4) + (q == 0 ? BP >> 4 : 0));
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                  ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc));
              acc = 1u;
            }
          }
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
              ::"r"(done0 + 8 * s)
              : "memory");
          if (++s == nst) s = 0;
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
            ::"r"(smem_u32(&acc_full[n & 1]))
            : "memory");
        ++n;
      });
    }
  }

  // result of four states of a row from their scaled sums
  auto finish4 = [&](int64_t row, float rs, int col, float4 v) {
    const int64_t off = row * a.ld + col;
    const uint4 m = __ldg(reinterpret_cast<const uint4*>(a.cmax + col));
    const float4 y = *reinterpret_cast<const float4*>(src + off);
    float4 o;
    o.x = a.alpha * (v.x * rs * scale_down(m.x)) + a.beta * y.x;
    o.y = a.alpha * (v.y * rs * scale_down(m.y)) + a.beta * y.y;
    o.z = a.alpha * (v.z * rs * scale_down(m.z)) + a.beta * y.z;
    o.w = a.alpha * (v.w * rs * scale_down(m.w)) + a.beta * y.w;
    if (a.delta != 0.f) {
      const float4 x = *reinterpret_cast<const float4*>(xold + off);
      o.x = fmaf(a.delta, x.x, o.x);
      o.y = fmaf(a.delta, x.y, o.y);
      o.z = fmaf(a.delta, x.z, o.z);
      o.w = fmaf(a.delta, x.w, o.w);
    }
    *reinterpret_cast<float4*>(dst + off) = o;
    return o;
  };

  // epilogue (one warp per 32 TMEM lanes): row = warp*32 + lane of the tile,
  // 16 states per TMEM load, while the MMAs of the next item run
  float* accs = reinterpret_cast<float*>(smem);  // shared tile: [128][kk + 4] sums
  if (warp < kEpiWarps) {
    uint32_t n = 0;
    each_item(a, [&](int tile, int b) {
      const UmmaItem it(a, tile, b);
      const int kk = it.kk, trow = warp * 32 + lane;
      const int row = __ldg(a.rowmap + (int64_t)tile * UR + trow);
      const float rs = F32 ? __ldg(a.rscale + (int64_t)tile * UR + trow) : 1.f;
      if (lane == 0) ok &= mbar_wait_idle(&acc_full[n & 1], (n >> 1) & 1, 256);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_base = tmem + (n & 1) * acc_cols + ((uint32_t)(warp * 32) << 16);
      for (int c0 = 0; c0 < kk; c0 += 16) {
        uint32_t v[16];
        if (it.nch > 0) {
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
                "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(lane_base + (uint32_t)c0));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0u;
        }
        if constexpr (F32) {
          if (shared_tile) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              *reinterpret_cast<uint4*>(accs + trow * (kk + 4) + c0 + j) =
                  make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              if (c0 + j >= it.kv) break;          // the same for all lanes
              float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
              if (row >= 0)
                o = finish4(row, rs, it.cb + c0 + j,
                            make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                        __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])));
              // largest |value| of each column, for the next degree's scale
              const uint32_t m0 = __reduce_max_sync(0xffffffffu, finite_bits(o.x));
              const uint32_t m1 = __reduce_max_sync(0xffffffffu, finite_bits(o.y));
              const uint32_t m2 = __reduce_max_sync(0xffffffffu, finite_bits(o.z));
              const uint32_t m3 = __reduce_max_sync(0xffffffffu, finite_bits(o.w));
              if (lane < 4)
                atomicMax(a.cmax_next + it.cb + c0 + j + lane,
                          lane == 0 ? m0 : lane == 1 ? m1 : lane == 2 ? m2 : m3);
            }
          }
        } else if (row >= 0) {
          // BF16 block: 8 values (16 bytes) per access, arithmetic in FP32 with
          // its fused steps written out: a contraction the other way round
          // changes the FP32 value's last bit, and now and then the BF16 one
          const int64_t off = (int64_t)row * a.ld + it.cb + c0;
#pragma unroll
          for (int j = 0; j < 16; j += 8) {
            const uint4 yu = *reinterpret_cast<const uint4*>(src + off + j);
            uint4 xu = make_uint4(0u, 0u, 0u, 0u);
            if (a.delta != 0.f) xu = *reinterpret_cast<const uint4*>(xold + off + j);
            const __nv_bfloat162* y2 = reinterpret_cast<const __nv_bfloat162*>(&yu);
            const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xu);
            uint4 ou;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ou);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const float2 yf = __bfloat1622float2(y2[t]);
              const float2 xf = __bfloat1622float2(x2[t]);
              const float a0 =
                  fmaf(a.delta, xf.x, fmaf(a.beta, yf.x, a.alpha * __uint_as_float(v[j + 2 * t])));
              const float a1 =
                  fmaf(a.delta, xf.y, fmaf(a.beta, yf.y, a.alpha * __uint_as_float(v[j + 2 * t + 1])));
              o2[t] = __floats2bfloat162_rn(a0, a1);
            }
            *reinterpret_cast<uint4*>(dst + off + j) = ou;
          }
        }
      }
      // the accumulator may be written again
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[n & 1]))
                     : "memory");
      ++n;
    });
  }
  if constexpr (F32) {
    if (shared_tile) {
      // the cluster's sums of this CTA's share of the rows, in rank order
      for (int c = tid; c < 256; c += kThreads) cnew[c] = 0u;
      __syncthreads();
      cluster_sync_all();
      each_item(a, [&](int tile, int b) {
        const UmmaItem it(a, tile, b);
        const int rows = UR / a.split, quads = it.kv >> 2, part = blockIdx.x % a.split;
        for (int i = tid; i < rows * quads; i += kThreads) {
          const int trow = part * rows + i / quads, c = (i % quads) * 4;
          const int row = __ldg(a.rowmap + (int64_t)tile * UR + trow);
          if (row < 0) continue;
          const uint32_t addr = smem_u32(accs + trow * (it.kk + 4) + c);
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
          for (int q = 0; q < a.split; ++q) {
            const float4 t = peer_load(addr, (uint32_t)q);
            v.x += t.x;
            v.y += t.y;
            v.z += t.z;
            v.w += t.w;
          }
          const float4 o = finish4(row, __ldg(a.rscale + (int64_t)tile * UR + trow), it.cb + c, v);
          atomicMax(&cnew[c], finite_bits(o.x));
          atomicMax(&cnew[c + 1], finite_bits(o.y));
          atomicMax(&cnew[c + 2], finite_bits(o.z));
          atomicMax(&cnew[c + 3], finite_bits(o.w));
        }
        __syncthreads();
        for (int c = tid; c < it.kv; c += kThreads) atomicMax(a.cmax_next + it.cb + c, cnew[c]);
      });
      cluster_sync_all();                        // peers have read this CTA's sums
    }
  }
  if (!ok) atomicExch(a.err, 1);
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols));
}

// Largest |value| of each column of the first FP32 degree's block (bits): a
// thread keeps four columns and has four rows in flight.
__global__ void __launch_bounds__(256) k_colmax(const float* __restrict__ src, int64_t rows, int k,
                                                int64_t ld, uint32_t* __restrict__ cmax) {
  __shared__ uint4 red[256];
  const int q0 = blockIdx.y * 256, nq = min(256, (k >> 2) - q0), lines = 256 / nq;
  const int q = threadIdx.x % nq, line = threadIdx.x / nq;
  uint4 m = make_uint4(0u, 0u, 0u, 0u);
  auto take = [&](float4 v) {
    m.x = max(m.x, finite_bits(v.x));
    m.y = max(m.y, finite_bits(v.y));
    m.z = max(m.z, finite_bits(v.z));
    m.w = max(m.w, finite_bits(v.w));
  };
  if (line < lines) {
    const float* p = src + (q0 + q) * 4;
    const int64_t step = (int64_t)gridDim.x * lines;
    int64_t r = (int64_t)blockIdx.x * lines + line;
    for (; r + 3 * step < rows; r += 4 * step) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(p + (r + u * step) * ld);
#pragma unroll
      for (int u = 0; u < 4; ++u) take(v[u]);
    }
    for (; r < rows; r += step) take(*reinterpret_cast<const float4*>(p + r * ld));
  }
  red[threadIdx.x] = m;
  __syncthreads();
  if (line == 0) {
    for (int j = 1; j < lines; ++j) {
      const uint4 o = red[j * nq + q];
      m = make_uint4(max(m.x, o.x), max(m.y, o.y), max(m.z, o.z), max(m.w, o.w));
    }
    uint32_t* c = cmax + (q0 + q) * 4;
    atomicMax(c, m.x);
    atomicMax(c + 1, m.y);
    atomicMax(c + 2, m.z);
    atomicMax(c + 3, m.w);
  }
}

struct PrepareArgs {
  const float* src;
  int64_t n, ld;
  int nproj, k, kp;
  __half* pl;                 // [2][n + nproj][kp]
  int64_t pstride;
  const uint32_t* cmax;
  uint32_t* cmax_next;
  const int64_t* cptr;
  const int* ccol;
  const double* cval;
  const float* wscale;        // power of two taken out of each W_a
  float* part;                // [nproj][nsplit][kp]
  int* ticket;                // [nproj][column groups], zero between launches
  int chunk, nsplit, groups, proj_blocks;
};

// What an FP32 degree needs of its block, in one launch: the two FP16 planes
// of the scaled columns, and of W_a = sum_J Cd[a,J] Y[J,:] (rows n + a).
// The first blocks sum `chunk` entries of a projector for 64 states (an eighth
// of them a warp, eight loads in flight); the last of a projector's blocks adds
// the parts in order and writes the planes.  The other blocks
// split the rows, 8 states a thread.  Bound: the projectors' gathered rows
// (L2) and the block read and written once.
constexpr int kPrepAhead = 8;
constexpr int kPrepChunk = 128;                  // the smallest chunk
__global__ void __launch_bounds__(256, 5) k_umma_prepare(const PrepareArgs a) {
  const int tid = threadIdx.x;
  if ((int)blockIdx.x < a.proj_blocks) {
    __shared__ float2 red[8][32];
    __shared__ int last;
    const int lane = tid & 31, w = tid >> 5;
    const int g = blockIdx.x % a.groups, sp = blockIdx.x / a.groups % a.nsplit;
    const int p = blockIdx.x / (a.groups * a.nsplit);
    const int c = g * 64 + 2 * lane;                  // k is even
    const int per = a.chunk / 8;
    const int64_t e0 = a.cptr[p] + (int64_t)sp * a.chunk + w * per;
    const int n = (int)max((int64_t)0, min(a.cptr[p + 1] - e0, (int64_t)per));
    const float* src = a.src + min(c, a.k - 2);
    float2 acc = make_float2(0.f, 0.f);
    for (int u0 = 0; u0 < n; u0 += 32) {
      // the columns and values of 32 entries, one a lane
      const int col = u0 + lane < n ? __ldg(a.ccol + e0 + u0 + lane) : 0;
      const float val = u0 + lane < n ? (float)__ldg(a.cval + e0 + u0 + lane) : 0.f;
#pragma unroll
      for (int h = 0; h < 32; h += kPrepAhead) {
        if (u0 + h >= n) break;
        float2 x[kPrepAhead];
#pragma unroll
        for (int u = 0; u < kPrepAhead; ++u) {
          const int64_t row = __shfl_sync(0xffffffffu, col, h + u);
          x[u] = make_float2(0.f, 0.f);
          if (u0 + h + u < n) x[u] = *reinterpret_cast<const float2*>(src + row * a.ld);
        }
#pragma unroll
        for (int u = 0; u < kPrepAhead; ++u) {
          const float v = __shfl_sync(0xffffffffu, val, h + u);
          acc.x = fmaf(v, x[u].x, acc.x);
          acc.y = fmaf(v, x[u].y, acc.y);
        }
      }
    }
    red[w][lane] = acc;
    __syncthreads();
    float* part = a.part + ((int64_t)p * a.nsplit) * a.kp + g * 64;
    const float* r1 = reinterpret_cast<const float*>(red);
    const bool col = tid < 64 && g * 64 + tid < a.k;
    if (col) {
      float s = r1[tid];
#pragma unroll
      for (int j = 1; j < 8; ++j) s += r1[j * 64 + tid];
      part[(int64_t)sp * a.kp + tid] = s;
      __threadfence();
    }
    __syncthreads();
    if (tid == 0) last = atomicAdd(a.ticket + p * a.groups + g, 1) == a.nsplit - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (tid == 0) a.ticket[p * a.groups + g] = 0;
    // four threads a state, each every fourth part
    __shared__ float sum[4][64];
    const int cc = tid & 63, q = tid >> 6;
    if (g * 64 + cc < a.k) {
      float s = 0.f;
#pragma unroll 8
      for (int j = q; j < a.nsplit; j += 4) s += __ldcg(part + (int64_t)j * a.kp + cc);
      sum[q][cc] = s;
    }
    __syncthreads();
    if (col) {
      const float s = ((sum[0][tid] + sum[1][tid]) + (sum[2][tid] + sum[3][tid])) * a.wscale[p];
      __half h, l;
      split_half(s * scale_up(a.cmax[g * 64 + tid]), h, l);
      __half* o = a.pl + (a.n + p) * a.kp + g * 64 + tid;
      o[0] = h;
      o[a.pstride] = l;
    }
    return;
  }
  const int64_t b0 = blockIdx.x - a.proj_blocks, nb = gridDim.x - a.proj_blocks;
  if (b0 == 0)
    for (int c = tid; c < a.k; c += 256) a.cmax_next[c] = 0u;
  const int kg = a.kp >> 3;
  const int64_t total = a.n * kg, step = nb * 256;
  // two items (8 states of a row) at a time
  for (int64_t i = b0 * 256 + tid; i < total; i += 2 * step) {
    float4 v[2][2];
    int c[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t at = i + u * step;
      const int64_t r = total <= INT_MAX ? (int64_t)((uint32_t)at / (uint32_t)kg) : at / kg;
      c[u] = (int)(at - r * kg) * 8;
      v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (at < total) {                               // k is a multiple of 4
        const float* p = a.src + r * a.ld + c[u];
        if (c[u] < a.k) v[u][0] = *reinterpret_cast<const float4*>(p);
        if (c[u] + 4 < a.k) v[u][1] = *reinterpret_cast<const float4*>(p + 4);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t at = i + u * step;
      if (at >= total) break;
      uint4 hi, lo;
      __half* h = reinterpret_cast<__half*>(&hi);
      __half* l = reinterpret_cast<__half*>(&lo);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint4 m = make_uint4(0u, 0u, 0u, 0u);
        if (c[u] + 4 * q < a.k) m = __ldg(reinterpret_cast<const uint4*>(a.cmax + c[u] + 4 * q));
        split_half(v[u][q].x * scale_up(m.x), h[4 * q], l[4 * q]);
        split_half(v[u][q].y * scale_up(m.y), h[4 * q + 1], l[4 * q + 1]);
        split_half(v[u][q].z * scale_up(m.z), h[4 * q + 2], l[4 * q + 2]);
        split_half(v[u][q].w * scale_up(m.w), h[4 * q + 3], l[4 * q + 3]);
      }
      *reinterpret_cast<uint4*>(a.pl + at * 8) = hi;
      *reinterpret_cast<uint4*>(a.pl + a.pstride + at * 8) = lo;
    }
  }
}

// Rows whose new values left the range of their scale (a warp a row): a new
// scale, and the row's entries written again, those of H from the FP64 values
// and those of C^T (slots of columns n + a) from C.
struct RescaleArgs {
  const int64_t* tptr;
  const int* tcol;
  const int* rowmap;
  const float* rmax;          // largest new |H| of each tile row
  const float* cmax;          // and its largest |C^T| 2^L
  float* rscale;
  uint16_t* h16;
  const int64_t* row_ptr;
  const int* umma_pos;
  const int* rg_pos;
  const int64_t* rg_gptr;
  const double* v64;
  const int64_t* cptr;
  const int* ccol;
  const float* cval;          // C 2^L
  int64_t rows, n;
};

__global__ void __launch_bounds__(256) k_umma_rescale(const RescaleArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t ur = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (ur >= a.rows) return;
  const int row = a.rowmap[ur];
  if (row < 0) return;
  const float hmax = a.rmax[ur], largest = fmaxf(hmax, a.cmax[ur]);
  const float scaled = largest / a.rscale[ur];     // a power of two: exact or infinite
  if (largest == 0.f || (scaled >= kRowLow && scaled < 32768.f)) return;
  const int e = min(126, max(-126, kRowExp - ilogbf(largest)));
  const float up = scalbnf(1.f, e);
  const int64_t tile = ur >> 7;
  const int m = (int)(ur & 127);
  uint16_t* h0 = a.h16 + a.tptr[tile] / UK * (2 * PLANE_ELEMS);
  auto put = [&](int slot, float v) {
    __half h, l;
    split_half(v * up, h, l);
    uint16_t* o = h0 + (int64_t)(slot / UK) * (2 * PLANE_ELEMS) + a_elem(m, slot % UK);
    o[0] = __half_as_ushort(h);
    o[PLANE_ELEMS] = __half_as_ushort(l);
  };
  for (int64_t i = a.row_ptr[row] + lane; i < a.row_ptr[row + 1]; i += 32)
    put(a.umma_pos[i], (float)a.v64[(a.rg_gptr[row >> 3] + a.rg_pos[i]) * 8 + (row & 7)]);
  const int64_t s0 = a.tptr[tile], s1 = a.tptr[tile + 1];
  for (int64_t s = s0 + lane; s < s1; s += 32) {
    const int col = a.tcol[s];
    if (col < a.n || (s > s0 && a.tcol[s - 1] == col)) continue;
    const int64_t p = col - a.n;
    for (int64_t i = a.cptr[p]; i < a.cptr[p + 1]; ++i)
      if (a.ccol[i] == row) put((int)(s - s0), a.cval[i]);
  }
  if (lane == 0) a.rscale[ur] = scalbnf(1.f, -e);
}

uint16_t bf16_bits(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)(u >> 16);
  const uint32_t rounding = 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)((u + rounding) >> 16);
}

// FP16 nearest to v (|v| below 65520, an infinity or NaN), to even, and the
// value it has.  Below 2^-14 FP16 counts in units of 2^-24, the last place of
// a float in [0.5, 1): adding 0.5 rounds to them.
uint16_t half_bits(float v, float& back) {
  uint32_t u;
  std::memcpy(&u, &v, 4);
  const uint16_t sign = (uint16_t)((u >> 16) & 0x8000u);
  u &= 0x7fffffffu;
  if (u >= 0x7f800000u) {
    back = v;
    return (uint16_t)(sign | 0x7c00u | (u > 0x7f800000u ? 0x200u : 0u));
  }
  if (u >= 0x38800000u) {                       // 2^-14
    u = (u + 0xfffu + ((u >> 13) & 1u)) & ~0x1fffu;
    std::memcpy(&back, &u, 4);
    back = std::copysign(back, v);
    return (uint16_t)(sign | ((u >> 13) - (112u << 10)));
  }
  const float m = std::fabs(v) + 0.5f;
  back = std::copysign(m - 0.5f, v);
  std::memcpy(&u, &m, 4);
  return (uint16_t)(sign | (u - 0x3f000000u));
}

// largest of |v|s, without infinities and NaN
void raise_max(float& m, float v) {
  v = std::fabs(v);
  if (v <= 3.402823466e38f && v > m) m = v;
}

}  // namespace

bool umma_enabled() {
  const char* e = getenv("TTG_DISABLE_UMMA");
  return !(e && e[0] == '1');
}

ttg_status build_umma_tiles(ttg_op* op, int64_t n, const int64_t* hp, const int32_t* hc,
                            const double* hv, int32_t nproj, const int64_t* cp, const int32_t* cc,
                            const double* cv, const double* d, const int32_t* dims) {
  if (!umma_enabled()) return TTG_OK;
  std::vector<int32_t> rowmap;
  int64_t ntiles;
  if (dims && dims[0] > 0 && dims[1] > 0 && dims[2] > 0 &&
      (int64_t)dims[0] * dims[1] * dims[2] == n) {
    const int rx = dims[0], ry = dims[1], rz = dims[2];
    const int bx = (rx + 3) / 4, by = (ry + 3) / 4, bz = (rz + 7) / 8;
    ntiles = (int64_t)bx * by * bz;
    rowmap.assign(ntiles * UR, -1);
    for (int tz = 0; tz < bz; ++tz)
      for (int ty = 0; ty < by; ++ty)
        for (int tx = 0; tx < bx; ++tx) {
          const int64_t t = tx + (int64_t)bx * (ty + (int64_t)by * tz);
          int slot = 0;
          for (int z = 0; z < 8; ++z)
            for (int y = 0; y < 4; ++y)
              for (int x = 0; x < 4; ++x, ++slot) {
                const int X = 4 * tx + x, Y = 4 * ty + y, Z = 8 * tz + z;
                if (X < rx && Y < ry && Z < rz) rowmap[t * UR + slot] = X + rx * (Y + ry * Z);
              }
        }
  } else {
    ntiles = (n + UR - 1) / UR;
    rowmap.assign(ntiles * UR, -1);
    for (int64_t i = 0; i < n; ++i) rowmap[i] = (int32_t)i;
  }
  // power of two that is at least L1(D_a C_a), so that |W_a| 2^-L <= max |Y|;
  // it goes into the entries of C^T
  std::vector<float> wscale(nproj), cval(nproj > 0 ? cp[nproj] : 0);
  for (int a = 0; a < nproj; ++a) {
    double l1 = 0.0;
    for (int64_t e = cp[a]; e < cp[a + 1]; ++e) l1 += std::fabs(d[a] * cv[e]);
    const int L = l1 > 0.0 && std::isfinite(l1) ? std::min(100, std::max(-100, std::ilogb(l1) + 1)) : 0;
    wscale[a] = std::ldexp(1.f, -L);
    for (int64_t e = cp[a]; e < cp[a + 1]; ++e) cval[e] = (float)std::ldexp(cv[e], L);
  }
  // C^T rows: (n + a, C[a, i]) for each basis row i
  std::vector<int64_t> tp(n + 1, 0);
  std::vector<int32_t> tcv;
  std::vector<double> tvv;
  std::vector<float> tvs;                       // the same times 2^L
  if (nproj > 0) {
    for (int a = 0; a < nproj; ++a)
      for (int64_t e = cp[a]; e < cp[a + 1]; ++e) tp[cc[e] + 1]++;
    for (int64_t i = 0; i < n; ++i) tp[i + 1] += tp[i];
    tcv.resize(tp[n]);
    tvv.resize(tp[n]);
    tvs.resize(tp[n]);
    std::vector<int64_t> f(tp.begin(), tp.end() - 1);
    for (int a = 0; a < nproj; ++a)
      for (int64_t e = cp[a]; e < cp[a + 1]; ++e) {
        tcv[f[cc[e]]] = (int32_t)(n + a);
        tvv[f[cc[e]]] = cv[e];
        tvs[f[cc[e]]] = cval[e];
        f[cc[e]]++;
      }
  }
  auto merge = [&](int64_t t, std::vector<int32_t>& cols) {
    cols.clear();
    for (int s = 0; s < UR; ++s) {
      const int32_t r = rowmap[t * UR + s];
      if (r < 0) continue;
      cols.insert(cols.end(), hc + hp[r], hc + hp[r + 1]);
      if (nproj > 0) cols.insert(cols.end(), tcv.begin() + tp[r], tcv.begin() + tp[r + 1]);
    }
    std::sort(cols.begin(), cols.end());
    cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
  };
  std::vector<int64_t> tptr(ntiles + 1, 0);
#pragma omp parallel
  {
    std::vector<int32_t> cols;
#pragma omp for schedule(dynamic, 4)
    for (int64_t t = 0; t < ntiles; ++t) {
      merge(t, cols);
      tptr[t + 1] = ((int64_t)cols.size() + UK - 1) / UK * UK;
    }
  }
  // Launch order.  While the gathered rows of one column block (two FP16
  // planes of up to 256 states per row) fit in L2, tiles run longest first, so the
  // short ones fill the tail.  Beyond that they run in their spatial order
  // (x fastest, then y, then z): the ~152 tiles resident at a time then
  // cover one slab of the Tucker grid, and the rows their columns gather
  // (the slab plus the band of H around it) stay in L2 while the slab is
  // worked on, instead of being fetched from HBM for every tile.
  std::vector<int32_t> order(ntiles);
  for (int64_t t = 0; t < ntiles; ++t) order[t] = (int32_t)t;
  const int64_t gather_bytes = n * (int64_t)std::min(op->max_k, 256) * 4;
  const bool sorted = gather_bytes <= ((int64_t)64 << 20);
  if (sorted)
    std::stable_sort(order.begin(), order.end(),
                     [&](int32_t a, int32_t b) { return tptr[a + 1] > tptr[b + 1]; });
  // The CTAs' lists: in that order to the CTA with the least to do so far (the
  // spatial order: in turn), CTAs by falling load.
  const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, kMaxCtas));
  std::vector<std::vector<int32_t>> lists(ctas);
  {
    std::vector<int64_t> load(ctas, 0);
    std::vector<int> by(ctas);
    for (int j = 0; j < ctas; ++j) by[j] = j;
    for (int64_t i = 0; i < ntiles; ++i) {
      const int j = sorted ? (int)(std::min_element(load.begin(), load.end()) - load.begin())
                           : (int)(i % ctas);
      lists[j].push_back(order[i]);
      load[j] += tptr[order[i] + 1] / UK + 8;
    }
    std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return load[x] > load[y]; });
    std::vector<std::vector<int32_t>> l(ctas);
    for (int j = 0; j < ctas; ++j) l[j].swap(lists[by[j]]);
    lists.swap(l);
  }
  std::vector<int32_t> lptr(1, 0), litem;
  for (const auto& l : lists) {
    litem.insert(litem.end(), l.begin(), l.end());
    lptr.push_back((int32_t)litem.size());
  }
  for (int64_t t = 0; t < ntiles; ++t) tptr[t + 1] += tptr[t];
  const int64_t slots = tptr[ntiles];
  const int64_t nchunk = slots / UK;
  const bool keep = op->keep_pattern;
  std::vector<int32_t> tcol(std::max<int64_t>(slots, UK), 0);
  // BF16 plane of every chunk, then the two FP16 planes of every chunk
  std::vector<uint16_t> hpl((size_t)std::max<int64_t>(nchunk, 1) * 3 * PLANE_ELEMS, 0);
  uint16_t* h16 = hpl.data() + std::max<int64_t>(nchunk, 1) * PLANE_ELEMS;
  std::vector<float> rscale(ntiles * UR, 1.f), rcmax(ntiles * UR, 0.f);
  std::vector<int32_t> pos(keep ? hp[n] : 0);
#pragma omp parallel
  {
    std::vector<int32_t> cols;
#pragma omp for schedule(dynamic, 4)
    for (int64_t t = 0; t < ntiles; ++t) {
      merge(t, cols);
      const int64_t ns = tptr[t + 1] - tptr[t];
      for (int64_t s = 0; s < ns; ++s)
        tcol[tptr[t] + s] = cols.empty() ? 0 : cols[std::min<int64_t>(s, (int64_t)cols.size() - 1)];
      const int64_t c0 = tptr[t] / UK;
      for (int m = 0; m < UR; ++m) {
        const int32_t r = rowmap[t * UR + m];
        if (r < 0) continue;
        float hmax = 0.f, cmax = 0.f;
        for (int64_t e = hp[r]; e < hp[r + 1]; ++e) raise_max(hmax, (float)hv[e]);
        if (nproj > 0)
          for (int64_t e = tp[r]; e < tp[r + 1]; ++e) raise_max(cmax, tvs[e]);
        const float big = std::max(hmax, cmax);
        const int ex = big > 0.f ? std::min(126, std::max(-126, kRowExp - std::ilogb(big))) : 0;
        const float up = std::ldexp(1.f, ex);
        rscale[t * UR + m] = std::ldexp(1.f, -ex);
        rcmax[t * UR + m] = cmax;
        for (int pass = 0; pass < 2; ++pass) {
          const int32_t* C = pass == 0 ? hc + hp[r] : tcv.data() + (nproj ? tp[r] : 0);
          const double* V = pass == 0 ? hv + hp[r] : tvv.data() + (nproj ? tp[r] : 0);
          const int64_t cnt = pass == 0 ? hp[r + 1] - hp[r] : (nproj ? tp[r + 1] - tp[r] : 0);
          for (int64_t e = 0; e < cnt; ++e) {
            const int64_t slot = std::lower_bound(cols.begin(), cols.end(), C[e]) - cols.begin();
            const int64_t chunk = c0 + slot / UK, at = a_elem(m, (int)(slot % UK));
            hpl[chunk * PLANE_ELEMS + at] = bf16_bits((float)V[e]);
            const float v = (pass == 0 ? (float)V[e] : tvs[tp[r] + e]) * up;
            float back, rest;
            uint16_t* u = h16 + chunk * 2 * PLANE_ELEMS + at;
            u[0] = half_bits(v, back);
            u[PLANE_ELEMS] = half_bits(v - back, rest);
            if (keep && pass == 0) pos[hp[r] + e] = (int32_t)slot;   // slot within the tile
          }
        }
      }
    }
  }
  UmmaOp& U = op->umma;
  U.n_tiles = ntiles;
  U.slots = slots;
  TTG_TRY(U.tptr.alloc((ntiles + 1) * sizeof(int64_t)));
  TTG_TRY(U.tcol.alloc(tcol.size() * sizeof(int32_t)));
  TTG_TRY(U.rowmap.alloc(rowmap.size() * sizeof(int32_t)));
  TTG_TRY(U.order.alloc(order.size() * sizeof(int32_t)));
  TTG_TRY(U.hpl.alloc(hpl.size() * sizeof(uint16_t)));
  TTG_TRY(U.err.alloc(sizeof(int)));
  U.fp16 = U.hpl.as<uint16_t>() + std::max<int64_t>(nchunk, 1) * PLANE_ELEMS;
  auto put = [&](DevBuf& b, const void* p, size_t bytes) -> ttg_status {
    TTG_TRY(b.alloc(std::max<size_t>(bytes, 16)));
    if (bytes) TTG_CUDA_TRY(cudaMemcpyAsync(b.p, p, bytes, cudaMemcpyHostToDevice, op->stream));
    return TTG_OK;
  };
  U.ctas = ctas;
  TTG_TRY(put(U.lptr, lptr.data(), lptr.size() * sizeof(int32_t)));
  TTG_TRY(put(U.litem, litem.data(), litem.size() * sizeof(int32_t)));
  TTG_TRY(put(U.rscale, rscale.data(), rscale.size() * sizeof(float)));
  TTG_TRY(put(U.wscale, wscale.data(), wscale.size() * sizeof(float)));
  if (keep) {
    TTG_TRY(put(U.rcmax, rcmax.data(), rcmax.size() * sizeof(float)));
    TTG_TRY(put(U.rmax, rcmax.data(), rcmax.size() * sizeof(float)));   // set by each update
    TTG_TRY(put(U.cval, cval.data(), cval.size() * sizeof(float)));
  }
  TTG_CUDA_TRY(cudaMemcpyAsync(U.tptr.p, tptr.data(), U.tptr.bytes, cudaMemcpyHostToDevice, op->stream));
  TTG_CUDA_TRY(cudaMemcpyAsync(U.tcol.p, tcol.data(), U.tcol.bytes, cudaMemcpyHostToDevice, op->stream));
  TTG_CUDA_TRY(cudaMemcpyAsync(U.rowmap.p, rowmap.data(), U.rowmap.bytes, cudaMemcpyHostToDevice,
                               op->stream));
  TTG_CUDA_TRY(cudaMemcpyAsync(U.order.p, order.data(), U.order.bytes, cudaMemcpyHostToDevice,
                               op->stream));
  TTG_CUDA_TRY(cudaMemcpyAsync(U.hpl.p, hpl.data(), U.hpl.bytes, cudaMemcpyHostToDevice, op->stream));
  TTG_CUDA_TRY(cudaMemsetAsync(U.err.p, 0, sizeof(int), op->stream));
  if (keep && hp[n] > 0) {
    TTG_TRY(op->pattern.umma_pos.alloc(hp[n] * sizeof(int32_t)));
    TTG_CUDA_TRY(cudaMemcpyAsync(op->pattern.umma_pos.p, pos.data(), hp[n] * sizeof(int32_t),
                                 cudaMemcpyHostToDevice, op->stream));
    // row -> tile * 128 + lane of the row in its tile
    std::vector<int32_t> urow(n, -1);
    for (int64_t t = 0; t < ntiles; ++t)
      for (int m = 0; m < UR; ++m)
        if (rowmap[t * UR + m] >= 0) urow[rowmap[t * UR + m]] = (int32_t)(t * UR + m);
    TTG_TRY(op->pattern.umma_row.alloc(n * sizeof(int32_t)));
    TTG_CUDA_TRY(cudaMemcpyAsync(op->pattern.umma_row.p, urow.data(), n * sizeof(int32_t),
                                 cudaMemcpyHostToDevice, op->stream));
  }
  TTG_CUDA_TRY(cudaStreamSynchronize(op->stream));
  return TTG_OK;
}

namespace {

// Very sparse operators (short tiles, up to 48 entries a row, far from a
// Hamiltonian's 1,500): an FP32 degree's planes of the block and padded tiles cost
// more than the CUDA cores' row groups, unless the rows are long for the block's
// width; the projectors' two launches come on top there.  Fitted to 390 degrees
// of 26 operators (us, here and on the row groups): 40,000 rows of 6.5 entries, 24
// states 28 and 13; 100,000 rows of 16, 24 states 52 and 31; 40,000 rows of 34, 24
// states 28 and 35, 60 states 48 and 37; 20,000 rows of 18 with projectors, 24
// states 25 and 28, 60 states 38 and 30.  None of the 390 gets slower by it.
bool rows_win(const ttg_op* op, int k) {
  const double row = (double)op->nnz_h / (double)op->n;
  if (op->umma.slots > 300 * op->umma.n_tiles || row > 48.0) return false;
  return op->nproj > 0 ? k >= std::max(48.0, 3.0 * row) : k >= std::max(8.0, 1.2 * row);
}

}  // namespace

// BF16 degrees: whole 16-state steps of the MMA, as the block is gathered.
// FP32 degrees have planes of their own, padded with zeros to such steps.
bool umma_supported(const ttg_op* op, int prec, int k) {
  if (op->umma.n_tiles == 0 || op->tc_disabled || k > op->ld) return false;
  if (prec == TTG_PREC_FP32) return k >= 4 && k % 4 == 0 && !rows_win(op, k);
  return prec == TTG_PREC_BF16 && k >= 16 && k % 16 == 0;
}

namespace {

template <bool F32, int NA>
ttg_status launch_umma_na(ttg_op* op, UmmaArgs& a, const void* src, const void* xold, void* dst) {
  UmmaOp& U = op->umma;
  constexpr int P = F32 ? 2 : 1, SC = F32 ? 2 : 4;
  // bytes of a stage: the gathered rows and H (1024 bytes go to alignment)
  constexpr int stage = SC * P * (NA * kAtomBytes + 2 * PLANE_ELEMS);
  constexpr int most = (kSmemBudget - 1024) / stage, half = (kSmemBudget / 2 - 4096) / stage;
  static_assert(most >= 3, "ring");
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.stream = op->stream;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  auto shape = [&](int split) {
    a.split = split;
    // a shared tile: two CTAs an SM where that leaves a ring, as the SMs of a
    // GPC are no multiple of a cluster's
    a.stages = std::min(kMaxStages, split > 1 && half >= 3 ? half : most);
    cfg.gridDim = dim3((unsigned)(split > 1 ? a.n_tiles * a.nblk * split : a.ctas * a.par));
    cfg.dynamicSmemBytes = (size_t)a.stages * stage + 1024;
    at.val.clusterDim.x = (unsigned)split;
    cfg.numAttrs = split > 1 ? 1 : 0;
  };
  // clusters of 2, 4 and 8 that are resident at once (constants of the kernel)
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  static int resident[3] = {0, 0, 0};
  std::call_once(once, [&] {
    attr_err = cudaFuncSetAttribute(k_cheb_umma<F32, NA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBudget);
    for (int i = 0; F32 && i < 3 && attr_err == cudaSuccess; ++i) {
      shape(2 << i);
      attr_err = cudaOccupancyMaxActiveClusters(&resident[i], k_cheb_umma<F32, NA>, &cfg);
    }
  });
  if (attr_err != cudaSuccess) return TTG_CUDA_ERR;
  // CTAs per tile: as many as are resident at once and keep at least four
  // stages of chunks each
  int split = 1;
  for (int i = 0; F32 && i < 3; ++i)
    if (a.n_tiles * a.nblk * (2 << i) <= kMaxCtas && a.n_tiles * a.nblk <= resident[i] &&
        U.slots / UK >= (int64_t)4 * SC * (2 << i) * a.n_tiles)
      split = 2 << i;
  shape(split);
  // two accumulators; a shared tile needs one
  a.tmem_cols = 32;
  while ((int)a.tmem_cols < a.kb) a.tmem_cols <<= 1;
  if (split == 1) a.tmem_cols <<= 1;
  TTG_TRY(kt_begin(op, F32 ? TTG_KT_UMMA_FP32 : TTG_KT_UMMA_BF16));
  TTG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_cheb_umma<F32, NA>, (const UmmaArgs)a, src, xold, dst));
  TTG_COUNT();
  TTG_LAUNCHED(op);
  return kt_end(op);
}

template <bool F32>
ttg_status launch_umma_t(ttg_op* op, UmmaArgs& a, const void* src, const void* xold, void* dst) {
  UmmaOp& U = op->umma;
  const int kp = (a.k + 15) / 16 * 16;
  // column blocks of at most one MMA's 256 states (the reference's
  // num_X_blocks, ChebyShevFilter.cc:97-170, splits its columns the same way)
  const int nblk = (kp + 255) / 256;
  a.kb = ((kp + nblk - 1) / nblk + 15) / 16 * 16;
  a.nblk = (kp + a.kb - 1) / a.kb;
  a.n_tiles = (int)U.n_tiles;
  a.ctas = U.ctas;
  a.par = std::max(1, std::min(a.nblk, kMaxCtas / U.ctas));
  a.tptr = U.tptr.as<int64_t>();
  a.tcol = U.tcol.as<int>();
  a.rowmap = U.rowmap.as<int>();
  a.order = U.order.as<int>();
  a.lptr = U.lptr.as<int>();
  a.litem = U.litem.as<int>();
  a.rscale = U.rscale.as<float>();
  a.ld = op->ld;
  a.err = U.err.as<int>();
  switch ((a.kb + kAtom - 1) / kAtom) {
    case 1: return launch_umma_na<F32, 1>(op, a, src, xold, dst);
    case 2: return launch_umma_na<F32, 2>(op, a, src, xold, dst);
    case 3: return launch_umma_na<F32, 3>(op, a, src, xold, dst);
    default: return launch_umma_na<F32, 4>(op, a, src, xold, dst);
  }
}

}  // namespace

ttg_status launch_cheb_umma(ttg_op* op, int prec, bool first, const void* src, const void* xold,
                            void* dst, int k, double alpha, double beta, double delta) {
  UmmaOp& U = op->umma;
  UmmaArgs a = {};
  a.k = k;
  a.alpha = (float)alpha;
  a.beta = (float)beta;
  a.delta = (float)delta;
  if (prec == TTG_PREC_BF16) {   // the block's rows are gathered as they are (row stride ld)
    a.hpl = U.hpl.as<uint16_t>();
    a.xpl = static_cast<const uint16_t*>(src);
    a.ps = (int)op->ld;
    return launch_umma_t<false>(op, a, src, xold, dst);
  }
  const int64_t rows = op->n + op->nproj;
  const int kp = (k + 15) / 16 * 16;
  PrepareArgs p = {};
  p.groups = (k + 63) / 64;
  // small parts while they are what fills the SMs, larger ones (fewer partial
  // rows and barriers) beyond
  p.chunk = op->C.nnz * p.groups > (int64_t)kPrepChunk * 152 * 4 ? 4 * kPrepChunk : kPrepChunk;
  p.nsplit = (int)((op->C.max_row_nnz + p.chunk - 1) / p.chunk);
  p.proj_blocks = op->nproj * p.nsplit * p.groups;
  auto grow = [&](DevBuf& b, size_t need, bool zero) -> ttg_status {
    if (b.bytes >= need) return TTG_OK;
    TTG_TRY(b.alloc(need));
    if (zero) TTG_CUDA_TRY(cudaMemsetAsync(b.p, 0, need, op->stream));
    return TTG_OK;
  };
  TTG_TRY(grow(U.xpl, (size_t)2 * rows * kp * sizeof(uint16_t), false));
  TTG_TRY(grow(U.cmax, (size_t)2 * op->ld * sizeof(uint32_t), false));
  TTG_TRY(grow(U.ticket, (size_t)std::max(1, op->nproj * p.groups) * sizeof(int), true));
  TTG_TRY(grow(op->wpart, (size_t)op->nproj * p.nsplit * kp * sizeof(float), false));
  uint32_t* cm = U.cmax.as<uint32_t>();
  if (first) {
    U.cside = 0;
    TTG_CUDA_TRY(cudaMemsetAsync(cm, 0, (size_t)k * sizeof(uint32_t), op->stream));
    const int quads = k / 4, gy = (quads + 255) / 256, lines = 256 / std::min(quads, 256);
    const int gx = (int)std::max<int64_t>(
        1, std::min<int64_t>((op->n + 4 * lines - 1) / (4 * lines), 152 * 3 / gy));
    k_colmax<<<dim3(gx, gy), 256, 0, op->stream>>>(static_cast<const float*>(src), op->n, k, op->ld, cm);
    TTG_COUNT();
    TTG_LAUNCHED(op);
  }
  p.src = static_cast<const float*>(src);
  p.n = op->n;
  p.ld = op->ld;
  p.nproj = op->nproj;
  p.k = k;
  p.kp = kp;
  p.pl = U.xpl.as<__half>();
  p.pstride = rows * kp;
  p.cmax = cm + U.cside * op->ld;
  p.cmax_next = cm + (U.cside ^ 1) * op->ld;
  p.cptr = op->C.ptr.as<int64_t>();
  p.ccol = op->C.col.as<int>();
  p.cval = op->C.val.as<double>();
  p.wscale = U.wscale.as<float>();
  p.part = op->wpart.as<float>();
  p.ticket = U.ticket.as<int>();
  const int64_t items = op->n * (kp / 8);
  const int split_blocks = (int)std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, 152 * 16));
  k_umma_prepare<<<(unsigned)(p.proj_blocks + split_blocks), 256, 0, op->stream>>>(p); TTG_COUNT();
  TTG_LAUNCHED(op);
  a.hpl = U.fp16;
  a.xpl = U.xpl.as<uint16_t>();
  a.pstride = p.pstride;
  a.ps = kp;
  a.cmax = p.cmax;
  a.cmax_next = p.cmax_next;
  U.cside ^= 1;
  return launch_umma_t<true>(op, a, src, xold, dst);
}

ttg_status launch_umma_rescale(ttg_op* op) {
  const UmmaOp& U = op->umma;
  const Pattern& P = op->pattern;
  RescaleArgs a = {};
  a.tptr = U.tptr.as<int64_t>();
  a.tcol = U.tcol.as<int>();
  a.rowmap = U.rowmap.as<int>();
  a.rmax = U.rmax.as<float>();
  a.cmax = U.rcmax.as<float>();
  a.rscale = U.rscale.as<float>();
  a.h16 = U.fp16;
  a.row_ptr = P.row_ptr.as<int64_t>();
  a.umma_pos = P.umma_pos.as<int>();
  a.rg_pos = P.rg_pos.as<int>();
  a.rg_gptr = op->rg.gptr.as<int64_t>();
  a.v64 = op->rg.v64.as<double>();
  a.cptr = op->C.ptr.as<int64_t>();
  a.ccol = op->C.col.as<int>();
  a.cval = U.cval.as<float>();
  a.rows = U.n_tiles * UR;
  a.n = op->n;
  k_umma_rescale<<<(unsigned)((a.rows + 7) / 8), 256, 0, op->stream>>>(a); TTG_COUNT();
  TTG_LAUNCHED(op);
  return TTG_OK;
}

ttg_status umma_check_error(ttg_op* op) {
  if (op->umma.n_tiles == 0) return TTG_OK;
  int e = 0;
  TTG_CUDA_TRY(cudaMemcpyAsync(&e, op->umma.err.p, sizeof(int), cudaMemcpyDeviceToHost, op->stream));
  TTG_CUDA_TRY(cudaStreamSynchronize(op->stream));
  if (e) {
    TTG_CUDA_TRY(cudaMemsetAsync(op->umma.err.p, 0, sizeof(int), op->stream));
    return TTG_TIMEOUT;
  }
  return TTG_OK;
}

}  // namespace ttg
