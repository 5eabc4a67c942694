// Fifth-generation tensor-core instructions (tcgen05): operand and instruction descriptors, the multiply-accumulate, and the
// accumulators' way out of tensor memory.  All operands are bf16 tiles of 128-byte rows in shared memory, sixteen-byte pieces
// permuted as the copy engine's 128-byte swizzle leaves them (piece c of row r at c ^ (r % 8)), on 1024-byte boundaries;
// accumulators are fp32.
#pragma once

#include "rglru_device.cuh"

namespace rglru {

// Shared-memory operand descriptor (addresses in units of sixteen bytes): start, leading and stride byte offsets, version 1,
// 128-byte swizzle.
//   contracted axis along the rows' 128 bytes: eight-row groups `stride` = 1024 apart, `lead` unused; the next 16 elements of
//   the axis start 32 bytes further;
//   contracted axis across the rows: eight-row groups 1024 apart along it, 64-element blocks of the other axis `lead` apart;
//   the next 16 elements start 2048 bytes further.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lead = 16) {
  return static_cast<uint64_t>((addr & 0x3ffffu) >> 4) | (static_cast<uint64_t>(lead >> 4) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: fp32 accumulators, bf16 operands, which of them are contracted across their rows, M x N.
__host__ __device__ constexpr uint32_t tc_idesc(int m, int n, bool a_across, bool b_across) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_across) << 15) | (static_cast<uint32_t>(b_across) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
// D[M x N] (+)= A[M x 16] B[N x 16]^T, by one thread.
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(static_cast<uint32_t>(add))
      : "memory");
}
// The barrier completes a phase when everything this thread has issued is done.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// One warp allocates (a power of two of at least 32 columns; the address goes to shared memory) and the same one frees.
template <int COLS>
__device__ __forceinline__ void tc_alloc(uint32_t* where) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(where)), "n"(COLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLS>
__device__ __forceinline__ void tc_free(uint32_t addr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "n"(COLS) : "memory");
}
// 32 columns of the 32 accumulator rows a warp may read (rows 32 (warp % 4) on): thread l gets row l.
__device__ __forceinline__ void tc_load32(uint32_t addr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      " tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace rglru
