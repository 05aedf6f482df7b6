// Warp-level integer matrix instructions (mma.sync, register operands) and the asynchronous 16-byte copies that feed them.
//
// Where they are used: products whose integer sums have to be scaled every 16, 32 or 256 inputs and that have few
// activation rows.  tcgen05 leaves such sums in tensor memory, and what then bounds a kernel is the way from there to the
// scaling threads and the hand-offs (barrier, commit, tcgen05.ld) of every group; here the sums of a group appear in the
// registers of the warp that scales them.  Measured on a B200, cycles per warp instruction and scheduler: m16n8k32 s8 8.05
// (2,035 multiply-adds per clock and SM, a quarter of tcgen05's rate), m16n8k16 s8 8.05 as well, imad 2.0, prmt 2.0, packed
// fp32 2.0, fp32 add 1.0 - several times what streaming a weight byte from HBM needs at up to 32 rows.
#pragma once
#include "common.cuh"

__device__ __forceinline__ void mma_s8_k32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                           uint32_t b1, int c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%10, %10, %10, %10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void mma_s8_k16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
// Four 8 x 16-byte matrices: lane l names row l % 8 of matrix l / 8; a thread receives bytes 4 (lane % 4) .. + 3 of row
// lane / 4 of each - the operand layout of the int8 instructions above, for either operand.
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// 16 bytes global -> shared, past L1; 4 bytes through it.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
