// tcgen05 helpers (fifth-generation tensor cores): shared-memory matrix
// and instruction descriptors, MMA issue and commit, the tensor-memory
// fences, allocation and loads.
#pragma once

#include <stdint.h>

#include "mbarrier.cuh"

namespace dgfs {

// Shared-memory matrix descriptor of a K-major SWIZZLE_128B tile starting at
// shared address `saddr` (1024-byte aligned, or advanced by a multiple of 32
// bytes inside the swizzle row for the MMA's K step): leading byte offset 16
// (unused by swizzled K-major layouts), stride byte offset 1024 (8-row
// groups), descriptor version 1, layout type 2 (128-byte swizzle).
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of an MN-major SWIZZLE_128B tile: each
// K row holds 64 BF16 of the M (or N) axis in 128 B, 8-row groups of K are
// 1024 B apart (stride byte offset), and the 64-wide M groups `lbo` bytes
// apart (leading byte offset). The MMA's K step of 16 rows advances the
// start by 2048 bytes.
__device__ __forceinline__ uint64_t sdesc_sw128_mn(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// kind::f16 with BF16 operands, FP32 accumulator, M x N; a_mn / b_mn select
// the MN-major layout of A / B (K-major otherwise).
__host__ __device__ constexpr uint32_t idesc_bf16_major(int m, int n, bool a_mn, bool b_mn) {
  return idesc_bf16(m, n) | (a_mn ? (1u << 15) : 0u) | (b_mn ? (1u << 16) : 0u);
}

// 2D tiled TMA load of the box at (x = innermost element, y = row) of the
// tensor map into shared memory, completing on `bar` (no multicast).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// Instruction descriptor of kind::tf32: FP32 accumulator, TF32 A and B
// (FP32 bit patterns whose low 13 mantissa bits the tensor core ignores),
// both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_tf32(int m, int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// Allocate ncols (a power of two >= 32) tensor-memory columns; the base
// address lands in *slot. Whole warp; the CTA then gives up its permit to
// allocate more, so a co-resident CTA never waits on it.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// x rounded to TF32 (nearest, ties away from zero): the low 13 mantissa
// bits of the result are zero.
__device__ __forceinline__ float tf32_round(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// Tensor memory as a warp's scratchpad: each thread owns one lane (the warp's
// quarter, 32 (warp % 4) + lane) and any columns, 32 bits each.  A load's
// registers hold its values after tmem_wait on them, which waits for every
// load of the thread; tmem_store_wait completes the thread's stores.
__device__ __forceinline__ void tmem_load(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]) : : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

__device__ __forceinline__ void tmem_load(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) : : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// n consecutive columns (a multiple of 8) of this thread's lane
template <int n> __device__ __forceinline__ void tm_load(uint32_t col, uint32_t (&t)[n]) {
  static_assert(n % 8 == 0, "columns in steps of 8");
#pragma unroll
  for (int c = 0; c + 16 <= n; c += 16) tmem_load(col + c, *reinterpret_cast<uint32_t(*)[16]>(&t[c]));
  if constexpr (n % 16) tmem_load(col + n / 16 * 16, *reinterpret_cast<uint32_t(*)[8]>(&t[n / 16 * 16]));
}
template <int n> __device__ __forceinline__ void tm_wait(uint32_t (&t)[n]) {
#pragma unroll
  for (int c = 0; c + 16 <= n; c += 16) tmem_wait(*reinterpret_cast<uint32_t(*)[16]>(&t[c]));
  if constexpr (n % 16) tmem_wait(*reinterpret_cast<uint32_t(*)[8]>(&t[n / 16 * 16]));
}
template <int n> __device__ __forceinline__ void tm_store(uint32_t col, const uint32_t (&t)[n]) {
#pragma unroll
  for (int c = 0; c + 16 <= n; c += 16) tmem_store(col + c, *reinterpret_cast<const uint32_t(*)[16]>(&t[c]));
  if constexpr (n % 16) tmem_store(col + n / 16 * 16, *reinterpret_cast<const uint32_t(*)[8]>(&t[n / 16 * 16]));
}
// a real value as words of tensor memory (1 or 2), at compile-time position i
template <int n> __device__ __forceinline__ void tm_put(uint32_t (&t)[n], int i, float v) { t[i] = __float_as_uint(v); }
template <int n> __device__ __forceinline__ void tm_put(uint32_t (&t)[n], int i, double v) {
  t[2 * i] = (uint32_t)__double2loint(v);
  t[2 * i + 1] = (uint32_t)__double2hiint(v);
}
template <int n> __device__ __forceinline__ float tm_get(const uint32_t (&t)[n], int i, float) {
  return __uint_as_float(t[i]);
}
template <int n> __device__ __forceinline__ double tm_get(const uint32_t (&t)[n], int i, double) {
  return __hiloint2double((int)t[2 * i + 1], (int)t[2 * i]);
}

}  // namespace dgfs
