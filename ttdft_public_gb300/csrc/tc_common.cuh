// Building blocks of the tcgen05 kernels (tgemm.cu, ozgemm.cu): shared-memory
// addresses and matrix descriptors, bounded mbarrier waits, TMA tile loads and
// tensor-memory loads.  Every wait is bounded (kTcMaxWait polls).
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cstdint>

namespace ttg {
namespace tc {

constexpr int kTcMaxWait = 1 << 22;

__device__ __forceinline__ uint32_t su32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// canonical K-major layout, no swizzle: core matrices of 8 rows x 16 bytes,
// 128 bytes apart along K (leading byte offset), 256 bytes apart along rows
// (stride byte offset)
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t addr) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)(128 >> 4) << 16;
  d |= (uint64_t)(256 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

__device__ __forceinline__ void bar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count));
}

__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(su32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait; gives up early when another role has aborted
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, volatile int* abort_flag,
                                         int ns) {
  for (int i = 0; i < kTcMaxWait; ++i) {
    if (bar_try(b, parity)) return true;
    if (*abort_flag) return false;
    if (ns) __nanosleep(ns);
  }
  *abort_flag = 1;
  return false;
}

// bounded wait that ignores the abort flag: on the abort path, for copies and
// MMAs already issued to complete before the CTA releases its memory
__device__ __forceinline__ bool bar_drain(uint64_t* b, uint32_t parity) {
  for (int i = 0; i < kTcMaxWait; ++i) {
    if (bar_try(b, parity)) return true;
    __nanosleep(128);
  }
  return false;
}

// non-blocking: has the phase of this parity completed (is the barrier past it)?
__device__ __forceinline__ bool bar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(su32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                         int c2, bool three_d, uint32_t bar) {
  if (three_d)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}

// four 8-column loads and one wait, in one statement (the registers are
// defined only after the wait)
__device__ __forceinline__ void tmem_ld8x4(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                           float* v0, float* v1, float* v2, float* v3) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%34];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%35];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3)
      : "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v0[j] = __uint_as_float(r[j]);
    v1[j] = __uint_as_float(r[8 + j]);
    v2[j] = __uint_as_float(r[16 + j]);
    v3[j] = __uint_as_float(r[24 + j]);
  }
}

}  // namespace tc
}  // namespace ttg
