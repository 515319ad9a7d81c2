// tcgen05 (5th-generation tensor core) pieces for single-CTA kernels: tensor memory allocation, the MMA with
// shared-memory operand descriptors, commit to an mbarrier, and loads of the accumulator from tensor memory.
#pragma once
#include "tma.cuh"

// ncols: a power of two, at least 32; the address of the allocation is written to *dst_smem.  One warp calls it.
__device__ __forceinline__ void kp_tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(kp_smem_u32(dst_smem)), "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
}
__device__ __forceinline__ void kp_tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
__device__ __forceinline__ void kp_tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void kp_tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, bfloat16 operands, float32 accumulator; one thread issues it
__device__ __forceinline__ void kp_umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// The same for a whole warp in step, whose operands are the same in every lane: one elected lane issues it.  (From inside a
// branch that one lane took, the operands pass through general registers: 94 cycles an MMA against 30.)
__device__ __forceinline__ void kp_umma_bf16_warp(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p, e;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// Four MMAs along K over one 128-byte box of a K-major A and B (64 elements), by an elected lane; `accumulate` is that of
// the first.
__device__ __forceinline__ void kp_umma_bf16_box(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool accumulate) {
    asm volatile("{\n .reg .pred p, e;\n .reg .b64 a, b;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n"
                 " add.s64 a, %1, 2;\n add.s64 b, %2, 2;\n setp.eq.b32 p, 0, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, {%5, %5, %5, %5}, p;\n"
                 " add.s64 a, %1, 4;\n add.s64 b, %2, 4;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, {%5, %5, %5, %5}, p;\n"
                 " add.s64 a, %1, 6;\n add.s64 b, %2, 6;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u) : "memory");
}
__device__ __forceinline__ void kp_umma_commit_warp(uint64_t* bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
                 " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(kp_smem_u32(bar)) : "memory");
}
// the mbarrier gets one arrival when every MMA issued so far by this thread has completed
__device__ __forceinline__ void kp_umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(kp_smem_u32(bar)) : "memory");
}
// 32 consecutive columns of this thread's lane of tensor memory (a warp reads the lanes 32 * (warp % 4) ...)
__device__ __forceinline__ void kp_tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The same without the wait: the registers hold the values only after kp_tmem_ld_wait(), so several loads
// can be under way at once.
__device__ __forceinline__ void kp_tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}
// 16 and 8 columns, without the wait
__device__ __forceinline__ void kp_tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void kp_tmem_ld8_issue(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void kp_tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 consecutive columns of this thread's lane written back to tensor memory (complete after kp_tmem_st_wait())
__device__ __forceinline__ void kp_tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
__device__ __forceinline__ void kp_tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- pairs of CTAs (cta_group::2): one MMA over two SMs, M = 256, each CTA with its half of A, of B's rows and of the output.
// One warp of each CTA allocates; the columns are the same in both.
__device__ __forceinline__ void kp_tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(kp_smem_u32(dst_smem)), "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
}
__device__ __forceinline__ void kp_tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
// Four MMAs along K over one 128-byte box of a K-major A and B (64 elements), by an elected lane of the pair's first CTA;
// the descriptors' addresses hold in both CTAs.  `accumulate` is that of the first.
__device__ __forceinline__ void kp_umma_bf16_box_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool accumulate) {
    asm volatile("{\n .reg .pred p, e;\n .reg .b64 a, b;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
                 " @e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
                 " add.s64 a, %1, 2;\n add.s64 b, %2, 2;\n setp.eq.b32 p, 0, 0;\n"
                 " @e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n"
                 " add.s64 a, %1, 4;\n add.s64 b, %2, 4;\n"
                 " @e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n"
                 " add.s64 a, %1, 6;\n add.s64 b, %2, 6;\n"
                 " @e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate ? 1u : 0u) : "memory");
}
// the mbarrier at this place of both CTAs gets one arrival when the pair's MMAs issued so far have completed (elected lane)
__device__ __forceinline__ void kp_umma_commit_pair(uint64_t* bar) {
    asm volatile("{\n .reg .pred e;\n .reg .b16 both;\n elect.sync _|e, 0xffffffff;\n mov.b16 both, 3;\n"
                 " @e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], both;\n}"
                 ::"r"(kp_smem_u32(bar)) : "memory");
}
// the address of this CTA's shared-memory place in the cluster's CTA `rank`
__device__ __forceinline__ uint32_t kp_cluster_addr(const void* p, int rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(kp_smem_u32(p)), "r"(rank));
    return ra;
}
// a box of the 2-D tensor to this CTA's shared memory, its bytes counted at a barrier of either CTA of the pair (elected lane)
__device__ __forceinline__ void kp_tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
                 " @e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}"
                 ::"r"(kp_smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void kp_mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// Shared-memory matrix descriptor of an operand tile whose rows are 128 bytes (64 bf16), stored with the
// 128-byte swizzle in atoms of 8 rows (1024 bytes): start address, leading offset 1 (16 bytes; unused by these
// layouts), stride offset 1024 bytes between 8-row groups, version 1, layout SWIZZLE_128B.  For a K-major
// operand the rows are the M/N index and a step of 16 along K is +2 in the address field (32 bytes); for an
// MN-major operand (rows = the K index, 64 M/N elements a row) a step of 16 along K is +2048 bytes.
__device__ __forceinline__ uint64_t kp_umma_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// The same for an MN-major operand of more than 64 elements along MN: its stretches of 64 lie lead_bytes apart.
__device__ __forceinline__ uint64_t kp_umma_desc_mn(uint32_t smem_addr, uint32_t lead_bytes) {
    return (kp_umma_desc(smem_addr) & ~((uint64_t)0x3FFF << 16)) | ((uint64_t)((lead_bytes >> 4) & 0x3FFF) << 16);
}
// Instruction descriptor: float32 accumulator, bfloat16 A and B, each K-major or (a_mn, b_mn) MN-major,
// N and M of the MMA.
__host__ __device__ constexpr uint32_t kp_umma_idesc(int M, int N, bool b_mn = false, bool a_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? (1u << 15) : 0u) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
