/*
 * tc_common.cuh - the fifth-generation tensor core: PTX wrappers, operand descriptors and the widening of
 * INT4 codes, shared by the kernels that run on it (ffn_tc.cu, ffn_stream_tc.cu).
 */
#pragma once

#include <cuda.h>

#include "stream_common.cuh"

namespace ffn {

constexpr int kTcRows = 128; /* the MMA's M = tensor-memory lanes: one weight row each */

/* ---- tcgen05 wrappers ------------------------------------------------------------------------ */
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
/* D[tmem] (+)= A[tmem] * B[smem]: M = 128 (lane = row), N and the operand types from the instruction
 * descriptor, K = 16; one column of A = two consecutive values of K in BF16 */
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
/* 16 consecutive columns of this thread's lane */
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                   "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
/* 16 consecutive FP32 columns of this thread's lane */
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&d)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
                   "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

/* Shared-memory operand descriptor: K-major, 128-byte swizzle.  A row of the operand is 128 bytes (64
 * values of K); 8 rows form a 1024-byte atom inside which the 16-byte piece c of row r sits at piece
 * c ^ (r & 7); `sbo` is the distance between 8-row atoms.  The leading-dimension field is not used by
 * swizzled K-major layouts (set to 1, as CUTLASS does); bits 46-47 = 1 is the descriptor version of this
 * architecture, layout type 2 (bits 61-63) the 128-byte swizzle.  An MMA's K = 16 (32 bytes) is
 * selected inside the 128-byte row by adding 32 bytes to the start address. */
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t sbo) {
    const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t hi = ((sbo >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
    return ((uint64_t)hi << 32) | lo;
}
/* Instruction descriptor of kind::f16: D = FP32 (bits 4-5 = 1), A = B = BF16 (bits 7-9, 10-12 = 1), both
 * K-major (bits 15, 16 = 0), N / 8 in bits 17-22, M / 16 in bits 24-28. */
__device__ __forceinline__ uint32_t tc_instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTcRows >> 4) << 24);
}
/* nibbles s and s+4 of a word as exact BF16 codes (low half: nibble s, high half: nibble s+4):
 * 0x4300 | n is 128 + n, the xor with 8 turns the two's-complement nibble into code + 8 */
__device__ __forceinline__ uint32_t tc_codes(uint32_t w_shifted) {
    uint32_t v, d;
    asm("lop3.b32 %0, %1, 0x000F000F, 0x43084308, 0x6A;" : "=r"(v) : "r"(w_shifted));
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(0x43084308u));
    return d;
}
__device__ __forceinline__ int tc_permute8(int e) { return ((e & 3) << 1) | (e >> 2); }
/* byte offset of token n's 16-byte piece c inside one K block of the activations' tile order */
__host__ __device__ __forceinline__ int tc_tile_offset(int n, int c) { return (n >> 3) * 1024 + (n & 7) * 128 + ((c ^ (n & 7)) << 4); }

/* Bounded wait of a whole warp: one lane polls, the result reaches the others through a shuffle (which
 * also orders their later accesses after the poll).  Thirty-two lanes polling the same barrier word
 * only multiply the shared-memory traffic that every other warp's loads and arrivals queue behind. */
__device__ __forceinline__ bool tc_warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int lane) {
    int ok = 1;
    if (lane == 0) ok = mbar_wait<32>(bar, parity, abort_flag) ? 1 : 0;
    return __shfl_sync(~0u, ok, 0) != 0;
}

/* One thread of a converged warp.  A tcgen05.mma or commit inside `if (elect_one())` issues in a few
 * cycles; behind `if (lane == 0)`, where the compiler cannot know that one thread is active, each takes
 * about 100 (eight MMAs of 128 x 16 x 16: 167 against 794 cycles). */
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}

}  // namespace ffn
