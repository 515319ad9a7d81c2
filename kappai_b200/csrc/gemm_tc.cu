// C[M,N] = A[M,K] * W[N,K]^T (bfloat16 in, float32 accumulation) on the 5th-generation tensor cores:
// tcgen05.mma with the accumulator in tensor memory, operands brought to shared memory by TMA.
// The product of prompt portions, and of few-row steps where it was measured faster than weight streaming.
//
// Persistent CTAs, one an SM; a CTA computes tiles of 128 x BN of C (tile b, b + grid, ...; m runs fastest so
// that the CTAs that run together share W tiles in L2).  BN is 256 to 32, chosen by a small cost model (tc_run).
// Roles by warp:
//   warp 0   : TMA producer.  For every k-block of 64 it waits for a free stage, arms the stage's "full"
//              mbarrier with the byte count and issues the tiled loads of the A box (128 rows x 64, or only
//              the rows there are, rounded up to 8, when M < 128) and the W box (BN rows x 64), both with
//              the 128-byte swizzle, no multicast.  The ring has as many stages as fit shared memory.
//   warp 1   : allocates tensor memory (accumulators for two tiles, if there is room: the epilogue of a tile runs
//              under the main loop of the next), then an elected lane of the warp issues the MMAs: four tcgen05.mma (128 x BN x 16)
//              per k-block, descriptors advanced by 32 bytes inside the swizzled rows (from inside a branch that one lane
//              took, a k-block cost about 0.3 us whatever its width: 128 rows by 2048 x 5632, 17.0 us against 12.4); tcgen05.commit frees the
//              stage ("empty" mbarrier) and, after the last k-block, signals "accumulator full".
//   the rest : epilogue, two warps for each quarter of the 128 lanes of tensor memory (a warp may only read
//              the lanes 32 * (warp % 4) ...), taking pieces of 16 columns in turn so that more loads and
//              stores are in flight.  Each reads its lanes with tcgen05.ld (a piece at a time; 32 columns where sums go to other CTAs), applies
//              bias / residual accumulation / SwiGLU, writes its rows of C and hands the accumulator back.
// A k-block costs the producer and the MMA warp about 0.1 us of waits, arming and commits beside its copies and MMAs, so a
// stage holds two k-blocks where that is at most 64 KB: one copy an operand, of a tensor map with the k-blocks as a
// dimension of its own (gate and up another), where K is a multiple of 64.  64 rows by 6144 x 2048 10.2 us with one, 9.4
// with two; 17 by 2048 x 5632 10.1 and 9.6.
//
// The kernels of a decode step follow one another through the SMs' instruction caches, and what a kernel does not find
// there it waits for, at every launch.  Hence loops that are not unrolled, the long part of a wait out of line, an epilogue
// of 16 columns at a time: 43 to 69 KB of code a kernel became 42 to 59, those of one k-block a stage half of that.  A step
// of 17 requests of the 1.2B shape 803 -> 770 us, of 100 of the 350M shape 729 -> 669; back to back the products hardly differ.
//
// Rows of A beyond M and rows of W beyond N are zero-filled by TMA (out-of-bounds fill) and masked at the
// store; K needs no padding (the tail of the last k-block is zero-filled too) but K % 8 == 0 (16-byte rows).
// Each output sums its k-blocks in order, within its part of K where the product is cut along K (tc_parts).
//
// SwiGLU epilogue: W holds gate rows then up rows (ff apart).  The CTA's W tile is BN/2 gate rows and the
// matching BN/2 up rows (two TMA boxes into one tile), so accumulator columns c and BN/2 + c are the gate and
// up of one output column: the epilogue writes silu(gate) * up.
//
// Split over K (17 to 1024 rows: up to eight rows of tiles; tc_parts): the product is cut along K into parts, whose sums
// are added in the order of the parts.  A CTA runs the parts of its tile one after the other, each into an accumulator of
// its own, and the epilogue adds them up (one commit a tile: a commit a part cost 0.25 us a part, the reading 0.05); or the
// unit of work is (tile, part), all units in one round over the SMs and the parts of a tile one thread-block cluster.
// Then every CTA owns some of the tile's output columns: when its sums are done it sends the other CTAs theirs
// (a bulk copy between the CTAs' rings, counted at a barrier of the owner), and adds up its own, the parts in order of their number -- so the result
// does not depend on timing -- then the epilogue.  The old values of an accumulated output come in under the exchange.
// (Sums left in shared memory and read by the others between two barriers of the cluster took 4.5 us from the last MMA to the
// end: with weights from HBM, 128 rows by 2048 x 5632 16.2 us, this 13.7; 17 rows by 2048 x 2048 6.4 and 5.9.  Sent by single
// stores that count at the barrier, st.async, the two took 8 and 35 % longer; added by the threads that read tensor memory, a few lanes
// of few warps at few rows, 7 and 18 %.)
// With it every SM brings in a part of A only, and wide tiles still keep all SMs streaming.
//
// Every wait on an mbarrier is bounded, and a warp goes on or gives up as one: instructions for a whole warp come next.  A wait
// that gives up sets a status word (kp_tc_status), the CTA stops issuing work, tells the other CTAs of its cluster, lingers until
// what is under way must have come, still frees its tensor memory and returns.
#include "tcgen05.cuh"

#define EPI_STORE 0
#define EPI_STORE_F32 1
#define EPI_ACCUM_F32 2
#define EPI_SWIGLU 3
#define EPI_ACT 6                            // store bf16 behind an ungated activation (common.cuh, kp_act_plain)
#define EPI_GLU 4                            // inside this file only: EPI_SWIGLU whose unit is the one with limits (act code 3)
#define EPI_GATED_RT 5                       // inside this file only: EPI_SWIGLU with an activation other than silu, chosen at run time
#define TC_GATED(E) ((E) == EPI_SWIGLU || (E) == EPI_GLU || (E) == EPI_GATED_RT)

#define TC_BM 128
#define TC_BK 64
#define TC_EPI_PER_Q 2                       // epilogue warps for each quarter of the tensor-memory lanes
#define TC_VI 2
#define TC_PIECE 16                          // columns that an epilogue warp of the one-CTA kernel takes at a time
#define TC_THREADS (64 + TC_EPI_PER_Q * 128) // the producer warp, the MMA warp and the epilogue warps

KP_STATUS_WORD(g_tc_status, tc)          // 0 ok; 1: a bounded wait gave up

struct TcArgs {
    const float* bias;
    void* C; int ldc;
    int M, N, K, ff;
    int act;                                // activation of the gated epilogue (common.cuh)
    float glu_limit, glu_alpha, glu_shift;  // constants of the gated unit with limits (act == KP_ACT_GLU_CLAMPED)
    int vec_ok;                             // rows of C are 16-byte aligned: whole pieces go out in 16-byte stores
    int a_rows;                             // rows of the A box: 128, fewer (a multiple of 8) when M < 128
    int n_stages;                           // stages of the ring
    int kb_stage;                           // k-blocks a stage: 1, or more that one copy an operand brings
    int splits;                             // CTAs that share a tile's parts along K, one each (1: no cluster)
    int inner;                              // parts along K that a CTA (or a pair) runs itself, one after the other (1 beside splits > 1)
    int kb_per_part;                        // k-blocks a part
    int n_sets;                             // sets of `inner` accumulators of BN columns in tensor memory: two, or the one there is room for
    int tmem_cols;                          // columns allocated
    int area;                               // bytes of the ring with its slack, or of what lies there later
    int recv_apart;                         // a split over a cluster: other CTAs' sums have a place of their own behind the barriers
};

// all threads of all CTAs of the cluster; what they wrote to shared memory before is visible to the others after
__device__ __forceinline__ void kp_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void kp_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void kp_cluster_sync() { kp_cluster_arrive(); kp_cluster_wait(); }
__device__ __forceinline__ void kp_cluster_sync_arrive() { kp_cluster_wait(); kp_cluster_arrive(); }   // the end of one round, the next one's start
// `bytes` (16 or a multiple) of this CTA's shared memory to a CTA of the cluster, counted there at a barrier (addresses in
// the cluster's window)
__device__ __forceinline__ void kp_copy_to_cluster(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "r"(kp_smem_u32(src)), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void kp_st_cluster(uint32_t addr, int v) { asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
// the epilogue warps (threads 64 ...) among themselves
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(TC_EPI_PER_Q * 128) : "memory"); }

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
}

// Biases of W sums g (and u: the up half, gated) of the output columns from n_base on, those below n_lim.
template <int EPI, int W>
__device__ __forceinline__ void tc_bias(const TcArgs& p, int n_lim, float (&g)[W], float (&u)[W], int n_base) {
    if (!p.bias) return;
#pragma unroll
    for (int j = 0; j < W; j++) {
        if (n_base + j < n_lim) {
            g[j] += p.bias[n_base + j];
            if TC_GATED(EPI) u[j] += p.bias[p.ff + n_base + j];
        }
    }
}
// What becomes of a sum.  silu has instantiations of its own: with the activation chosen at run time every one of the
// 32 outputs that were unrolled then carried the code of all of them, and the epilogue waited for instructions (200 rows by gate/up
// 11264 x 2048: 24.1 us a product against 20.7; the kernel of pairs 31.6 against 20.2).
template <int EPI>
__device__ __forceinline__ float tc_value(const TcArgs& p, float g, float u) {
    if TC_GATED(EPI) {
        // gate and up are rounded to the storage type first, as the unfused path stores them
        const float gq = to_f32(from_f32<bf16>(g)), uq = to_f32(from_f32<bf16>(u));
        if (EPI == EPI_GLU) return kp_glu_clamped(gq, uq, p.glu_limit, p.glu_alpha, p.glu_shift);
        return (EPI == EPI_SWIGLU ? kp_act<KP_ACT_SILU>(gq) : kp_act_epilogue(p.act, gq)) * uq;
    }
    return EPI == EPI_ACT ? kp_act_plain(p.act, g) : g;
}

// A piece of W output columns (16; 32 behind a pair's float32 store; 4 in the split's reduction) of row m, from its sums g (and u: the up half,
// SwiGLU), to C: bias, SwiGLU or accumulation, and the store (vector stores where rows of C are 16-byte aligned).
template <int EPI, int W>
__device__ __forceinline__ void tc_finish(const TcArgs& p, int n_lim, const float (&g)[W], const float (&u)[W], int m,
                                          int n_base) {
    float v[W];
#pragma unroll
    for (int j = 0; j < W; j++) {
        float x = g[j], up = u[j];
        if (p.bias && n_base + j < n_lim) {
            x += p.bias[n_base + j];
            if TC_GATED(EPI) up += p.bias[p.ff + n_base + j];
        }
        v[j] = tc_value<EPI>(p, x, up);
    }
    const bool whole = p.vec_ok && n_base + W <= n_lim;                  // vector stores of the whole piece
    if (EPI == EPI_STORE || EPI == EPI_ACT || TC_GATED(EPI)) {
        bf16* dst = (bf16*)p.C + (size_t)m * p.ldc + n_base;
        if (whole && W >= 8) {
#pragma unroll
            for (int j = 0; j + 8 <= W; j += 8) {
                uint4 o;
                o.x = pack2(v[j], v[j + 1]); o.y = pack2(v[j + 2], v[j + 3]);
                o.z = pack2(v[j + 4], v[j + 5]); o.w = pack2(v[j + 6], v[j + 7]);
                *reinterpret_cast<uint4*>(dst + j) = o;
            }
        } else if (whole && W == 4) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
        } else {
#pragma unroll
            for (int j = 0; j < W; j++)
                if (n_base + j < n_lim) dst[j] = from_f32<bf16>(v[j]);
        }
    } else {
        float* dst = (float*)p.C + (size_t)m * p.ldc + n_base;
        if (whole) {
#pragma unroll
            for (int j = 0; j < W; j += 4) {
                float4 o = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                if (EPI == EPI_ACCUM_F32) {
                    const float4 c4 = *reinterpret_cast<const float4*>(dst + j);
                    o.x += c4.x; o.y += c4.y; o.z += c4.z; o.w += c4.w;
                }
                *reinterpret_cast<float4*>(dst + j) = o;
            }
        } else {
#pragma unroll
            for (int j = 0; j < W; j++) {
                if (n_base + j < n_lim) {
                    float x = v[j];
                    if (EPI == EPI_ACCUM_F32) x += dst[j];
                    dst[j] = x;
                }
            }
        }
    }
}

// W columns of tensor memory, without the wait
__device__ __forceinline__ void tc_ld_issue(uint32_t at, uint32_t (&r)[32]) { kp_tmem_ld32_issue(at, r); }
__device__ __forceinline__ void tc_ld_issue(uint32_t at, uint32_t (&r)[16]) { kp_tmem_ld16_issue(at, r); }

// The W sums of a lane's row at a place of the unit's accumulators, g (and u: the up half, gated): one part's as they are,
// several parts' added from zero in the order of the parts, as the split over a cluster adds them.
// (PARTS false: there is one, which saves the pairs' gated epilogue the registers that the adding needs.)
template <int EPI, int BN, bool PARTS, int W>
__device__ __forceinline__ void tc_sums(const TcArgs& p, uint32_t at, float (&g)[W], float (&up)[W]) {
    uint32_t r[W], u[W];
    tc_ld_issue(at, r);
    if TC_GATED(EPI) tc_ld_issue(at + BN / 2, u);
    kp_tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < W; j++) {
        g[j] = __uint_as_float(r[j]);
        up[j] = TC_GATED(EPI) ? __uint_as_float(u[j]) : 0.f;
    }
    if (PARTS && p.inner > 1) {
#pragma unroll
        for (int j = 0; j < W; j++) { g[j] = 0.f + g[j]; if TC_GATED(EPI) up[j] = 0.f + up[j]; }
#pragma unroll 1
        for (int i = 1; i < p.inner; i++) {
            at += BN;
            tc_ld_issue(at, r);
            if TC_GATED(EPI) tc_ld_issue(at + BN / 2, u);
            kp_tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < W; j++) { g[j] += __uint_as_float(r[j]); if TC_GATED(EPI) up[j] += __uint_as_float(u[j]); }
        }
    }
}

// What an epilogue warp does when it gave up (whatever gave up, these warps end here): the CTAs of the cluster are told first, so that
// one that has not sent its sums yet does not send them; what is under way to here or from here has come when the warp arrives
// at the cluster's last barrier, before which no CTA leaves.
__device__ __noinline__ void tc_gave_up(int* abort_flag, int n_ctas) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) { *abort_flag = 1; atomicExch(&g_tc_status, 1); }
    if (n_ctas > 1 && lane < n_ctas) kp_st_cluster(kp_cluster_addr(abort_flag, lane), 1);
    kp_linger_after_failure();
}

template <int N> struct TcInt { static constexpr int value = N; };

template <int BN, int EPI>
__global__ void __launch_bounds__(TC_THREADS)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const TcArgs p) {
    constexpr int B_BYTES = BN * TC_BK * 2;
    constexpr int N_OUT_TILE = TC_GATED(EPI) ? BN / 2 : BN;       // output columns of the tile
    const int A_BYTES = p.a_rows * TC_BK * 2;                            // the rows of A that are brought in
    // (a stage: the A tiles of its kb_stage k-blocks, then their W tiles)
    const int STAGES = p.n_stages;
    extern __shared__ unsigned char smem[];
    // STAGES x (A tile | B tile); the swizzled tiles must start on 1024-byte boundaries.  With fewer than 128
    // rows of A a stage is smaller and the ring has more of them; the MMA still reads 128 rows from the
    // stage's start (on into the W tile and beyond: the host leaves room after the last stage), and what it
    // makes of the rest lands in accumulator rows that nobody reads.
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + p.area);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;                                  // [2]: set b holds a finished unit
    uint64_t* acc_empty = acc_full + 2;                                   // [2]: set b has been read out
    uint64_t* recv_full = acc_empty + 2;                                  // (split over a cluster) the other parts' sums are here
    uint64_t* rings_free = recv_full + 1;                                 // ... the other CTAs' rings are free
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rings_free + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned char* recv = p.recv_apart ? tiles + p.area + ((2 * STAGES + 6) * 8 + 8 + 15) / 16 * 16 : tiles + (size_t)min(p.M, TC_BM) * BN * 4;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_kb = (p.K + TC_BK - 1) / TC_BK;
    const int n_out = TC_GATED(EPI) ? p.ff : p.N;
    const int tiles_m = (p.M + TC_BM - 1) / TC_BM, tiles_n = (n_out + N_OUT_TILE - 1) / N_OUT_TILE;
    const int n_tiles = tiles_m * tiles_n;
    const int S = p.splits;                                              // parts along K; a unit of work is (tile, part)
    const int n_units = n_tiles * S;
    // (split over a cluster) the tile's output columns in eights, in which is counted what a CTA owns, and the bytes of a row's
    // sums that an eight takes
    constexpr int U = N_OUT_TILE / 8, EIGHT = TC_GATED(EPI) ? 64 : 32;
    // the CTA is persistent: it takes tiles blockIdx.x, blockIdx.x + gridDim.x, ... ; consecutive tiles
    // share the W tile (m runs fastest), so the CTAs that run together read the same few W tiles from L2

    // set-up that depends on no earlier kernel comes before the wait on it
    if (threadIdx.x == 0) {
        // (the tensor maps are fetched now: the first TMA load through a map that has not been used waits for it)
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmW)) : "memory");
#pragma unroll 1
        for (int s = 0; s < STAGES; s++) { kp_mbar_init(&full[s], 1); kp_mbar_init(&empty[s], 1); }
        for (int b2 = 0; b2 < 2; b2++) { kp_mbar_init(&acc_full[b2], 1); kp_mbar_init(&acc_empty[b2], 4 * TC_EPI_PER_Q); }
        kp_mbar_init(recv_full, 1);
        if (S > 1) kp_mbar_init(rings_free, S - 1);
        *abort_flag = 0;
        kp_mbar_init_fence();
        if (S > 1) {                                                      // (the bytes that the cluster's other CTAs will send)
            const int rank = blockIdx.x % S, R = min(TC_BM, p.M - (int)((blockIdx.x / S) % tiles_m) * TC_BM);
            kp_mbar_expect_tx(recv_full, (S - 1) * (U * (rank + 1) / S - U * rank / S) * EIGHT * R);
        }
    }
    if (warp == 1) kp_tmem_alloc(tmem_slot, p.tmem_cols);
    kp_tc_fence_before();
    __syncthreads();
    kp_tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (S > 1) kp_cluster_arrive();                                       // (waited for in front of the first use of another CTA's memory)

    // (the producer's and the MMA warp's lanes stay in step; one elected lane issues what they issue)
    // (their loops are compiled for each number of k-blocks a stage: they are what a narrow tile's k-blocks wait for)
    const auto produce = [&](auto nb) {
        constexpr int NB = decltype(nb)::value;
        const int STAGE = NB * (A_BYTES + B_BYTES);
        auto load_w = [&](int s, int kb, int n0) {
            unsigned char* b_dst = tiles + (size_t)s * STAGE + NB * A_BYTES;
            if (NB > 1) {
                if TC_GATED(EPI) kp_tma_load_4d_warp(b_dst, &tmW, 0, n0, 0, kb, &full[s]);
                else kp_tma_load_3d_warp(b_dst, &tmW, 0, n0, kb, &full[s]);
            } else if TC_GATED(EPI) {
                kp_tma_load_2d_warp(b_dst, &tmW, kb * TC_BK, n0, &full[s]);                       // gate rows
                kp_tma_load_2d_warp(b_dst + B_BYTES / 2, &tmW, kb * TC_BK, p.ff + n0, &full[s]);  // up rows
            } else {
                kp_tma_load_2d_warp(b_dst, &tmW, kb * TC_BK, n0, &full[s]);
            }
        };
        // The weights depend on no earlier kernel: the W tiles of the first unit's first stages (as many as
        // the ring has) are on their way before the wait on the kernel before; their A tiles follow it.
        int pre = 0;
        if ((int)blockIdx.x < n_units) {
            const int tile = blockIdx.x / S, part = blockIdx.x - tile * S;
            const int n0 = (tile / tiles_m) * N_OUT_TILE;
            const int kb_lo = part * p.kb_per_part, kb_hi = S > 1 ? min(n_kb, kb_lo + p.kb_per_part) : n_kb;
            pre = min(STAGES, (kb_hi - kb_lo + NB - 1) / NB);
#pragma unroll 1
            for (int i = 0; i < pre; i++) {
                kp_mbar_expect_tx_warp(&full[i], STAGE);
                load_w(i, kb_lo + i * NB, n0);
            }
        }
        if (lane == 0) KP_TRACE_MARK_LANE(0);
        pdl_wait();
        if (lane == 0) KP_TRACE_MARK_LANE(1);
        pdl_launch_dependents();
        int s = 0;                                                    // stage, and the parity of its round
        uint32_t ph = 0;
        bool ok = true;
#pragma unroll 1
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
            const int tile = unit / S, part = unit - tile * S;
            const int m0 = (tile % tiles_m) * TC_BM, n0 = (tile / tiles_m) * N_OUT_TILE;
            const int kb_lo = part * p.kb_per_part, kb_hi = S > 1 ? min(n_kb, kb_lo + p.kb_per_part) : n_kb;
#pragma unroll 1
            for (int kb = kb_lo; kb < kb_hi; kb += NB) {
                unsigned char* a_dst = tiles + (size_t)s * STAGE;
                if (pre > 0) {
                    pre--;                                            // armed, W on its way: only A is missing
                } else {
                    ok = __all_sync(0xffffffffu, !*abort_flag && kp_mbar_wait_bounded(&empty[s], ph ^ 1));
                    if (!ok) { *abort_flag = 1; break; }
                    kp_mbar_expect_tx_warp(&full[s], STAGE);
                    load_w(s, kb, n0);
                }
                if (NB > 1) kp_tma_load_3d_warp(a_dst, &tmA, 0, m0, kb, &full[s]);
                else kp_tma_load_2d_warp(a_dst, &tmA, kb * TC_BK, m0, &full[s]);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    };
    const auto multiply = [&](auto nb) {
        constexpr int NB = decltype(nb)::value;
        const int STAGE = NB * (A_BYTES + B_BYTES);
        constexpr uint32_t idesc = kp_umma_idesc(TC_BM, BN);
        int s = 0, b2 = 0;                                                // stage; set of accumulators of this unit
        uint32_t ph = 0, set_ph = 1;                                      // (both sets are empty at first)
        bool ok = true;
#pragma unroll 1
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
            ok = __all_sync(0xffffffffu, !*abort_flag && kp_mbar_wait_bounded(&acc_empty[b2], set_ph));
            if (!ok) { *abort_flag = 1; break; }
            kp_tc_fence_after();
            uint32_t tmem_d = tmem_base + (uint32_t)(b2 * p.inner * BN);
            const int part = unit % S;
            const int kb_lo = part * p.kb_per_part, kb_hi = S > 1 ? min(n_kb, kb_lo + p.kb_per_part) : n_kb;
            int part_kb = 0;                                              // k-blocks in the accumulator so far
#pragma unroll 1
            for (int kb = kb_lo; kb < kb_hi; kb += NB) {
                ok = __all_sync(0xffffffffu, kp_mbar_wait_bounded(&full[s], ph));
                if (!ok) { *abort_flag = 1; break; }
                kp_tc_fence_after();
                const uint32_t a_addr = kp_smem_u32(tiles + (size_t)s * STAGE);
#pragma unroll
                for (int j = 0; j < NB; j++) {
                    if (j > 0 && kb + j >= kb_hi) break;
                    if (part_kb == p.kb_per_part) { part_kb = 0; tmem_d += BN; }
                    // four MMAs of 16 columns (32 bytes along K inside the swizzled row: +2 in the address field)
                    kp_umma_bf16_box(tmem_d, kp_umma_desc(a_addr + j * A_BYTES), kp_umma_desc(a_addr + NB * A_BYTES + j * B_BYTES), idesc, part_kb++ != 0);
                }
                kp_umma_commit_warp(&empty[s]);                           // the stage is free when these MMAs have read it
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            if (ok) kp_umma_commit_warp(&acc_full[b2]);                   // arrives when every MMA of the unit has completed
            if (++b2 == p.n_sets) { b2 = 0; set_ph ^= 1; }
        }
    };
    if (warp == 0) {
        if (p.kb_stage == 1) produce(TcInt<1>{}); else produce(TcInt<2>{});
        if (S > 1) { __syncwarp(); kp_cluster_sync_arrive(); }
    } else if (warp == 1) {
        kp_pdl_begin();
        if (p.kb_stage == 1) multiply(TcInt<1>{}); else multiply(TcInt<2>{});
        if (S > 1) { __syncwarp(); kp_cluster_sync_arrive(); }
    } else {
        kp_pdl_begin();
        // epilogue: warp w reads the 32 lanes (w % 4) * 32 ... of tensor memory; it works on unit i while the
        // MMA warp already fills the other accumulator with unit i + 1
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;                                 // which of the quarter's warps
        int b2 = 0;
        uint32_t set_ph = 0;
        bool ok = true;
#pragma unroll 1
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
            const int tile = unit / S;
            const int m0 = (tile % tiles_m) * TC_BM, n0 = (tile / tiles_m) * N_OUT_TILE;
            ok = __all_sync(0xffffffffu, kp_mbar_wait_bounded(&acc_full[b2], set_ph) && !*abort_flag);
            if (__builtin_expect(!ok, 0)) {
                if (S > 1) { kp_cluster_wait(); epi_sync(); }             // (where the other warps may be waiting for this one)
                break;
            }
            kp_tc_fence_after();
            const int m = m0 + q * 32 + lane;
            const uint32_t lane_base = tmem_base + (uint32_t)(b2 * p.inner * BN) + ((uint32_t)(q * 32) << 16);
            uint64_t* const read_out = &acc_empty[b2];
            if (++b2 == p.n_sets) { b2 = 0; set_ph ^= 1; }
            if (S == 1) {
#pragma unroll 1
                for (int c = half * TC_PIECE; c < N_OUT_TILE; c += TC_PIECE * TC_EPI_PER_Q) {
                    float g[TC_PIECE], up[TC_PIECE];
                    tc_sums<EPI, BN, true>(p, lane_base + c, g, up);
                    if (m < p.M) tc_finish<EPI, TC_PIECE>(p, n_out, g, up, m, n0 + c);
                }
                // this warp has read the accumulators out: hand them back to the MMA warp
                kp_tc_fence_before();
                __syncwarp();
                if (lane == 0) kp_mbar_arrive(read_out);
                continue;
            }
            // Split over K: every CTA of the cluster owns some of the tile's output columns, in eights.  A CTA writes its sums to
            // its ring, which is free, an eight behind the other, each [gate, up][half][row][4]; sends every other owner its
            // eights -- into the owner's ring, behind its sums, once that is free as well, or apart from it -- and adds up its own.
            const int rank = unit - tile * S, R = min(TC_BM, p.M - m0);   // (rows of this tile)
            const int lo = U * rank / S, own = U * (rank + 1) / S - lo;
            kp_cluster_wait();
            if (!p.recv_apart && threadIdx.x < 64 + S && (int)threadIdx.x - 64 != rank) kp_mbar_arrive_cluster(kp_cluster_addr(rings_free, threadIdx.x - 64));
#pragma unroll 1
            for (int c = half * 32; c < BN && q * 32 < R; c += 32 * TC_EPI_PER_Q) {
                uint32_t r[32];
                kp_tmem_ld32(lane_base + c, r);
                const int cu = c / 8, up = cu >= U ? 1 : 0;
                if (m < p.M) {
                    uint4* dst = reinterpret_cast<uint4*>(tiles + ((cu - up * U) * EIGHT + up * 32) * R) + (m - m0);
#pragma unroll
                    for (int k = 0; k < 4; k++, dst += EIGHT / 16 * R) {
                        dst[0] = make_uint4(r[8 * k], r[8 * k + 1], r[8 * k + 2], r[8 * k + 3]);
                        dst[R] = make_uint4(r[8 * k + 4], r[8 * k + 5], r[8 * k + 6], r[8 * k + 7]);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            epi_sync();
            if (warp == 2) {
                // (a CTA that gave up while this one waited here has told so: see tc_gave_up)
                if (!p.recv_apart) ok = __all_sync(0xffffffffu, kp_mbar_try_wait(rings_free, 0) || (kp_mbar_wait_bounded(rings_free, 0) && !*abort_flag));
                const int olo = U * lane / S, bytes = (U * (lane + 1) / S - olo) * EIGHT * R;
                if (ok && lane < S && lane != rank && bytes > 0)
                    kp_copy_to_cluster(kp_cluster_addr(recv, lane) + (rank < lane ? rank : rank - 1) * bytes, tiles + olo * EIGHT * R, bytes,
                                       kp_cluster_addr(recv_full, lane));
                __syncwarp();
            }
            // Its own, by all epilogue threads: VI pieces of four columns of a row at a time; the old values of an accumulated
            // output are asked for before the wait.
            constexpr int VI = TC_VI, NT = TC_EPI_PER_Q * 128;
            const int n_vec = own * 2 * R;
            const bool old_apart = EPI == EPI_ACCUM_F32 && p.vec_ok;
            bool here = false;
#pragma unroll 1
            for (int i0 = (int)threadIdx.x - 64; i0 - lane - (warp - 2) * 32 < n_vec || !here; i0 += VI * NT) {
                int at[VI], col[VI], row[VI];                             // where in an owner's eights; the output's column and row, -1: none
                float4 old[VI];
#pragma unroll
                for (int v = 0; v < VI; v++) {
                    const int idx = i0 + v * NT, piece = idx / R;
                    row[v] = idx < n_vec ? idx - piece * R : -1;
                    col[v] = n0 + lo * 8 + piece * 4;
                    at[v] = ((piece >> 1) * EIGHT + (piece & 1) * 16) * R + row[v] * 16;
                    if (old_apart && row[v] >= 0 && col[v] + 4 <= n_out) old[v] = *reinterpret_cast<const float4*>((const float*)p.C + (size_t)(m0 + row[v]) * p.ldc + col[v]);
                }
                if (!here) {
                    here = true;
                    ok = __all_sync(0xffffffffu, kp_mbar_wait_bounded(recv_full, 0) && ok);
                    if (!ok) break;
                }
                float g[VI][4], up[VI][4];
#pragma unroll
                for (int v = 0; v < VI; v++)
#pragma unroll
                    for (int j = 0; j < 4; j++) g[v][j] = up[v][j] = 0.f;
#pragma unroll 1
                for (int part = 0; part < S; part++) {
                    const unsigned char* src = part == rank ? tiles + lo * EIGHT * R : recv + (part < rank ? part : part - 1) * own * EIGHT * R;
#pragma unroll
                    for (int v = 0; v < VI; v++) {
                        if (row[v] < 0) continue;
                        const float4 a = *reinterpret_cast<const float4*>(src + at[v]);
                        g[v][0] += a.x; g[v][1] += a.y; g[v][2] += a.z; g[v][3] += a.w;
                        if TC_GATED(EPI) {
                            const float4 b = *reinterpret_cast<const float4*>(src + at[v] + 32 * R);
                            up[v][0] += b.x; up[v][1] += b.y; up[v][2] += b.z; up[v][3] += b.w;
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < VI; v++) {
                    if (row[v] < 0) continue;
                    if (old_apart && col[v] + 4 <= n_out) {
                        tc_bias<EPI, 4>(p, n_out, g[v], up[v], col[v]);
                        *reinterpret_cast<float4*>((float*)p.C + (size_t)(m0 + row[v]) * p.ldc + col[v]) =
                            make_float4(g[v][0] + old[v].x, g[v][1] + old[v].y, g[v][2] + old[v].z, g[v][3] + old[v].w);
                    } else {
                        tc_finish<EPI, 4>(p, n_out, g[v], up[v], m0 + row[v], col[v]);
                    }
                }
            }
        }
        if (__builtin_expect(!ok, 0)) tc_gave_up(const_cast<int*>(abort_flag), S);
        if (S > 1) { __syncwarp(); kp_cluster_arrive(); }
    }
    kp_tc_fence_before();
    __syncthreads();
    if (S > 1) kp_cluster_wait();                                         // no CTA leaves before all have what they were sent, or have given up
    if (threadIdx.x == 64) KP_TRACE_MARK_LANE(2);
    if (warp == 1) kp_tmem_dealloc(tmem_base, p.tmem_cols);
}

// ------------------------------------------------------------------------------------------ pairs of CTAs
// Products of many rows: a pair of CTAs (a cluster of two, cta_group::2) computes tiles of 256 x BN, each CTA 128 of the
// rows.  What bounds the one-CTA kernel there is the bytes that an SM brings into shared memory: for 128 x 256 outputs it
// reads 48 KB a k-block, about 770 cycles' worth from L2 for 512 cycles of MMAs.  A pair reads A once a CTA and each half
// of W once a pair: 32 KB an SM.  The roles are those of gemm_tc_kernel; the first CTA's MMA warp issues for both, both
// CTAs' loads count at its "full" barriers, and its commits free the stages and hand over the accumulators in both.
// The sums run in the same order as in gemm_tc_kernel, parts included (the same bits).  Measured, us, one CTA a tile | pairs: 2,048 rows by
// 11264 x 2048 (gated) 77.0 | 67.0, 1.41 PFLOP/s; 2048 x 5632 44.8 | 37.2; 6144 x 2048 46.8 | 37.7; 2048 x 2048 25.3 | 19.3;
// 512 rows by 65536 x 1024 92.8 | 65.1.
//
// The epilogue warps pass their pieces (128 bytes of 32 rows) through shared memory, so that a warp writes, and for an
// accumulated output reads, four whole rows' stretches of 128 bytes at a time instead of 16 bytes of 32 rows; the old
// values of an accumulated output are asked for before the piece is read from tensor memory.  16 columns of
// sums at a time, but for a float32 store (a head) 32.  us, 16 | 32 at a time: float32 999 rows by 65536 x 1024 120.0 | 119.0;
// accumulating 2,048 rows by 2048 x 2048 18.9 | 20.1 (the old values need the registers); gated 999 rows by 9216 x 1024 22.2 | 21.8,
// but 41 KB of code against 98, and in a prompt, where the code comes anew at every launch, the gain is gone (2,048 tokens of the 1.2B
// shape 3.249 | 3.253 ms); stored 999 rows by 3072 x 2048 15.5 | 15.3, but the convolution behind such a product is then no longer resident
// beside it, for the registers, and the product behind that takes the SMs in front of it: a step of 2,048 rows, some of them
// decoded, 3.28 | 3.41 ms (350M shape 2.10 | 2.31).
#define TC_PAIR_STAGES(BN) ((BN) == 256 ? 5 : 7)
#define TC_PAIR_SMEM(BN) ((size_t)TC_PAIR_STAGES(BN) * (128 + (BN) / 2) * TC_BK * 2 + TC_EPI_PER_Q * 4 * 4096 + (2 * TC_PAIR_STAGES(BN) + 4) * 8 + 16 + 1024)

template <int BN, int EPI, bool PARTS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const TcArgs p) {
    constexpr int STAGES = TC_PAIR_STAGES(BN);
    constexpr int A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN / 2 * TC_BK * 2, STAGE = A_BYTES + B_BYTES;
    constexpr int N_OUT_TILE = TC_GATED(EPI) ? BN / 2 : BN;
    extern __shared__ unsigned char smem[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
    unsigned char* pieces = tiles + (size_t)STAGES * STAGE;                // 4 KB an epilogue warp
    uint64_t* full = reinterpret_cast<uint64_t*>(pieces + TC_EPI_PER_Q * 4 * 4096);   // (the first CTA's are used)
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;                                  // [2]
    uint64_t* acc_empty = acc_full + 2;                                   // [2] (the first CTA's are used)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_kb = (p.K + TC_BK - 1) / TC_BK;
    const int n_out = TC_GATED(EPI) ? p.ff : p.N;
    const int tiles_m = (p.M + 2 * TC_BM - 1) / (2 * TC_BM), tiles_n = (n_out + N_OUT_TILE - 1) / N_OUT_TILE;
    const int n_tiles = tiles_m * tiles_n;

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmW)) : "memory");
        for (int s = 0; s < STAGES; s++) { kp_mbar_init(&full[s], 1); kp_mbar_init(&empty[s], 1); }
        for (int b2 = 0; b2 < 2; b2++) { kp_mbar_init(&acc_full[b2], 1); kp_mbar_init(&acc_empty[b2], 2 * 4 * TC_EPI_PER_Q); }
        *abort_flag = 0;
        kp_mbar_init_fence();
    }
    if (warp == 1) kp_tmem_alloc_pair(tmem_slot, p.tmem_cols);
    kp_tc_fence_before();
    __syncthreads();
    kp_cluster_sync();                                                    // both CTAs' barriers and tensor memory are there
    kp_tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        auto load_w = [&](int s, int kb, int n0) {
            // this CTA's half of the W tile: gate rows or up rows, or the first or second BN / 2 rows
            const int row = TC_GATED(EPI) ? rank * p.ff + n0 : n0 + rank * (BN / 2);
            kp_tma_load_2d_pair(tiles + (size_t)s * STAGE + A_BYTES, &tmW, kb * TC_BK, row, kp_cluster_addr(&full[s], 0));
        };
        int pre = 0;
        if (pair < n_tiles) {
            const int n0 = (pair / tiles_m) * N_OUT_TILE;
            pre = min(STAGES, n_kb);
#pragma unroll 1
            for (int i = 0; i < pre; i++) {
                if (rank == 0) kp_mbar_expect_tx_warp(&full[i], 2 * STAGE);
                load_w(i, i, n0);
            }
        }
        if (lane == 0) KP_TRACE_MARK_LANE(0);
        pdl_wait();
        if (lane == 0) KP_TRACE_MARK_LANE(1);
        pdl_launch_dependents();
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
#pragma unroll 1
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int m0 = (tile % tiles_m) * 2 * TC_BM + rank * TC_BM, n0 = (tile / tiles_m) * N_OUT_TILE;
#pragma unroll 1
            for (int kb = 0; kb < n_kb; kb++) {
                if (pre > 0) {
                    pre--;
                } else {
                    ok = __all_sync(0xffffffffu, !*abort_flag && kp_mbar_wait_bounded(&empty[s], ph ^ 1));
                    if (!ok) { *abort_flag = 1; break; }
                    if (rank == 0) kp_mbar_expect_tx_warp(&full[s], 2 * STAGE);
                    load_w(s, kb, n0);
                }
                kp_tma_load_2d_pair(tiles + (size_t)s * STAGE, &tmA, kb * TC_BK, m0, kp_cluster_addr(&full[s], 0));
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        kp_pdl_begin();
        if (rank == 0) {                                                  // (the whole warp in step: one elected lane issues)
            constexpr uint32_t idesc = kp_umma_idesc(2 * TC_BM, BN);
            int s = 0, b2 = 0;
            uint32_t ph = 0, set_ph = 1;
            bool ok = true;
#pragma unroll 1
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                ok = __all_sync(0xffffffffu, !*abort_flag && kp_mbar_wait_bounded(&acc_empty[b2], set_ph));
                if (!ok) { *abort_flag = 1; break; }
                kp_tc_fence_after();
                uint32_t tmem_d = tmem_base + (uint32_t)(b2 * p.inner * BN);
                int part_kb = 0;
#pragma unroll 1
                for (int kb = 0; kb < n_kb; kb++) {
                    if (part_kb == p.kb_per_part) { part_kb = 0; tmem_d += BN; }
                    ok = __all_sync(0xffffffffu, kp_mbar_wait_bounded(&full[s], ph));
                    if (!ok) { *abort_flag = 1; break; }
                    kp_tc_fence_after();
                    const uint32_t a_addr = kp_smem_u32(tiles + (size_t)s * STAGE);
                    kp_umma_bf16_box_pair(tmem_d, kp_umma_desc(a_addr), kp_umma_desc(a_addr + A_BYTES), idesc, part_kb++ != 0);
                    kp_umma_commit_pair(&empty[s]);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (ok) kp_umma_commit_pair(&acc_full[b2]);
                if (++b2 == p.n_sets) { b2 = 0; set_ph ^= 1; }
            }
        }
    } else {
        kp_pdl_begin();
        const int q = warp & 3, half = (warp - 2) >> 2;
        unsigned char* piece = pieces + (size_t)(warp - 2) * 4096;
        constexpr bool NARROW = EPI == EPI_STORE || EPI == EPI_ACT || TC_GATED(EPI);   // 16-bit outputs: a piece is 64 columns
        constexpr int PW = NARROW ? 64 : 32;
        constexpr int PC = EPI == EPI_STORE_F32 ? 32 : 16;                // columns of sums at a time (see above)
        int b2 = 0;
        uint32_t set_ph = 0;
        bool ok = true;
#pragma unroll 1
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int m0 = (tile % tiles_m) * 2 * TC_BM + rank * TC_BM + q * 32, n0 = (tile / tiles_m) * N_OUT_TILE;
            ok = __all_sync(0xffffffffu, kp_mbar_wait_bounded(&acc_full[b2], set_ph) && !*abort_flag);
            if (!ok) break;
            kp_tc_fence_after();
            const uint32_t lane_base = tmem_base + (uint32_t)(b2 * p.inner * BN) + ((uint32_t)(q * 32) << 16);
            const int m = m0 + lane;
#pragma unroll 1
            for (int c = half * PW; c < N_OUT_TILE && m0 < p.M; c += PW * TC_EPI_PER_Q) {
                const bool staged = p.vec_ok && n0 + c + PW <= n_out;     // (the same for the whole warp)
                const int prow = lane >> 3, pch = lane & 7;               // a pass through the piece: rows prow, prow + 4, ...
                float4 old[8];
                if (EPI == EPI_ACCUM_F32 && staged) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int row = m0 + i * 4 + prow;
                        old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (row < p.M) old[i] = *reinterpret_cast<const float4*>((const float*)p.C + (size_t)row * p.ldc + n0 + c + pch * 4);
                    }
                }
#pragma unroll 1
                for (int h = 0; h < PW / PC; h++) {
                    const int n_base = n0 + c + h * PC;
                    float v[PC], up[PC];
                    tc_sums<EPI, BN, PARTS>(p, lane_base + c + h * PC, v, up);
                    if (!staged) {
                        if (m < p.M) tc_finish<EPI, PC>(p, n_out, v, up, m, n_base);
                        continue;
                    }
                    // (rows beyond the last hold zeros, on which the activation's division is slow: they are left alone)
                    if (m < p.M) {
                        tc_bias<EPI, PC>(p, n_out, v, up, n_base);
#pragma unroll
                        for (int j = 0; j < PC; j++) v[j] = tc_value<EPI>(p, v[j], up[j]);
                    }
                    if (NARROW) {
#pragma unroll
                        for (int j = 0; j < PC / 8; j++)
                            *reinterpret_cast<uint4*>(piece + lane * 128 + (((h * (PC / 8) + j) ^ (lane & 7)) * 16)) =
                                make_uint4(pack2(v[8 * j], v[8 * j + 1]), pack2(v[8 * j + 2], v[8 * j + 3]), pack2(v[8 * j + 4], v[8 * j + 5]), pack2(v[8 * j + 6], v[8 * j + 7]));
                    } else {
#pragma unroll
                        for (int j = 0; j < PC / 4; j++)
                            *reinterpret_cast<float4*>(piece + lane * 128 + (((h * (PC / 4) + j) ^ (lane & 7)) * 16)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    }
                }
                if (!staged) continue;
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int row = i * 4 + prow;
                    if (m0 + row >= p.M) continue;
                    const unsigned char* src = piece + row * 128 + ((pch ^ (row & 7)) * 16);
                    if (NARROW) {
                        *reinterpret_cast<uint4*>((bf16*)p.C + (size_t)(m0 + row) * p.ldc + n0 + c + pch * 8) = *reinterpret_cast<const uint4*>(src);
                    } else {
                        float4 o = *reinterpret_cast<const float4*>(src);
                        if (EPI == EPI_ACCUM_F32) { o.x += old[i].x; o.y += old[i].y; o.z += old[i].z; o.w += old[i].w; }
                        *reinterpret_cast<float4*>((float*)p.C + (size_t)(m0 + row) * p.ldc + n0 + c + pch * 4) = o;
                    }
                }
                __syncwarp();
            }
            kp_tc_fence_before();
            __syncwarp();
            if (lane == 0) kp_mbar_arrive_cluster(kp_cluster_addr(&acc_empty[b2], 0));
            if (++b2 == p.n_sets) { b2 = 0; set_ph ^= 1; }
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(&g_tc_status, 1); }
    }
    kp_tc_fence_before();
    __syncthreads();
    if (*abort_flag) kp_linger_after_failure();
    if (threadIdx.x == 64) KP_TRACE_MARK_LANE(2);
    kp_cluster_sync();                                                    // the other CTA may still signal barriers here
    if (warp == 1) kp_tmem_dealloc_pair(tmem_base, p.tmem_cols);
}

// ------------------------------------------------------------------------------------------ host side
#define TC_SMEM_KB 208                       // shared memory for the ring
#define TC_SPLIT_MAX_M_TILES 8               // rows of tiles up to which a product may be cut along K
#define TC_SPLIT_COST (64 * 1024)            // a split over K, in bytes brought into an SM (tc_parts)
// the choice of a tile (tc_choose), in bytes brought into an SM
#define TC_KB_MIN (22 * 1024)                // a k-block at least
#define TC_PAIR_COST (100 * 1024)            // a pair of CTAs

// SMs of the current device (asked once)
static int tc_n_sm() {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    return sms;
}

#define TC_RECV_APART (24 * 1024)            // up to this much has a place of its own, and no CTA has to know that another's ring is free
// Shared memory of a launch: `stages` ring stages with the slack behind a short last stage, or a cluster's exchange of sums if
// that is more (`area`); barriers, alignment, and what other CTAs send apart from that (`apart`).
struct TcSmem { int stages, area, apart; size_t bytes; };
static TcSmem tc_smem(int M, int a_rows, int bn, bool gated, int splits, int kb_stage = 1) {
    TcSmem t = {};
    const int rows = M < TC_BM ? M : TC_BM, stage = kb_stage * (a_rows + bn) * TC_BK * 2;
    const int slack = (TC_BM - a_rows) * TC_BK * 2;            // the MMA's reads past a short last stage
    // the most that a CTA of a cluster is sent: the others' sums of its output columns, which are counted in eights
    const int eights = bn / (gated ? 16 : 8), recv = (splits - 1) * ((eights + splits - 1) / splits) * (gated ? 64 : 32) * rows;
    t.apart = recv <= TC_RECV_APART ? recv : 0;
    t.stages = (TC_SMEM_KB * 1024 - slack - t.apart) / stage;
    if (t.stages > 24) t.stages = 24;
    if (t.stages < 2) t.stages = 2;
    t.area = t.stages * stage + slack;
    const int exchange = splits > 1 ? rows * bn * 4 + recv - t.apart : 0;
    if (t.area < exchange) t.area = (exchange + 1023) / 1024 * 1024;
    t.bytes = (size_t)t.area + (size_t)(2 * t.stages + 6) * 8 + 8 + 16 + t.apart + 1024;
    return t;
}

template <int BN, int EPI>
static int prepare() {
    static std::atomic<unsigned long long> ready{0};
    return kp_smem_limit(gemm_tc_kernel<BN, EPI>, KP_SMEM_MAX, ready);
}

// Clusters of `cluster` CTAs of this kernel that the device runs at once (asked once for each size; 0 if it cannot
// be said): a split over K wants all its tiles' clusters in one round.
template <int BN, int EPI>
static int max_clusters(int cluster, size_t smem) {
    static int known[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (cluster < 2 || cluster > 8) return 0;
    if (known[cluster] == 0) {
        known[cluster] = -1;
        if (prepare<BN, EPI>() == 0) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(cluster * 64); cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr; cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_tc_kernel<BN, EPI>, &cfg) == cudaSuccess && n > 0) known[cluster] = n;
            else cudaGetLastError();
        }
    }
    return known[cluster] > 0 ? known[cluster] : 0;
}

template <int BN, int EPI>
static int launch(const CUtensorMap& ta, const CUtensorMap& tw, TcArgs a, cudaStream_t s) {
    const TcSmem sm = tc_smem(a.M, a.a_rows, BN, TC_GATED(EPI), a.splits, a.kb_stage);
    if (sm.bytes > KP_SMEM_MAX) return KP_ERR_UNSUPPORTED;
    a.n_stages = sm.stages; a.area = sm.area; a.recv_apart = sm.apart > 0;
    const size_t smem = sm.bytes;
    int st = prepare<BN, EPI>();
    if (st) return st;
    const int n_out = TC_GATED(EPI) ? a.ff : a.N;
    const int n_tile = TC_GATED(EPI) ? BN / 2 : BN;
    const int n_units = ((n_out + n_tile - 1) / n_tile) * ((a.M + TC_BM - 1) / TC_BM) * a.splits;
    const int sms = tc_n_sm();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.splits > 1 ? n_units : (n_units < sms ? n_units : sms));   // persistent: one CTA an SM
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
    if (a.splits > 1) {                                        // the parts of a tile: one cluster
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = a.splits; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    cfg.attrs = attr;
    cudaLaunchKernelEx(&cfg, gemm_tc_kernel<BN, EPI>, ta, tw, a);
    return kp_launch_status();
}

template <int BN, int EPI, bool PARTS>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tw, const TcArgs& a, cudaStream_t s) {
    auto kern = gemm_tc_pair_kernel<BN, EPI, PARTS>;
    static std::atomic<unsigned long long> ready{0};
    const int st = kp_smem_limit(kern, TC_PAIR_SMEM(BN), ready);
    if (st) return st;
    const int n_out = TC_GATED(EPI) ? a.ff : a.N, n_tile = TC_GATED(EPI) ? BN / 2 : BN;
    const int n_tiles = ((n_out + n_tile - 1) / n_tile) * ((a.M + 2 * TC_BM - 1) / (2 * TC_BM));
    const int pairs = tc_n_sm() / 2;
    return (int)kp_launch_pdl(kern, dim3(2 * (n_tiles < pairs ? n_tiles : pairs)), dim3(TC_THREADS), TC_PAIR_SMEM(BN), s, ta, tw, a);
}

// Clusters of `cluster` CTAs that run at once, for the tile width and epilogue of a launch.
static int tc_max_clusters(int bn, int epi, int cluster, int a_rows) {
    const size_t smem = tc_smem(TC_BM, a_rows, bn, false, 1).bytes;
#define TC_MC(BN_, EPI_) return max_clusters<BN_, EPI_>(cluster, smem);
#define TC_MC_BN(EPI_)                                             \
    switch (bn) {                                                  \
        case 256: TC_MC(256, EPI_)                                 \
        case 128: TC_MC(128, EPI_)                                 \
        case 64: TC_MC(64, EPI_)                                   \
        default: return 0;                                         \
    }
    switch (epi) {
        case EPI_STORE: TC_MC_BN(EPI_STORE)
        case EPI_STORE_F32: TC_MC_BN(EPI_STORE_F32)
        case EPI_ACCUM_F32: TC_MC_BN(EPI_ACCUM_F32)
        case EPI_ACT: TC_MC_BN(EPI_ACT)
        case EPI_SWIGLU: TC_MC_BN(EPI_SWIGLU)
        default: return 0;
    }
#undef TC_MC_BN
#undef TC_MC
}

// How a product runs: the width of its tiles, its parts along K, and whether the parts of a tile are shared by the CTAs of a
// cluster or run one after the other, by one CTA or a pair of them.
struct TcChoice { int bn, parts; bool cluster, pair; };

// K-blocks a stage (see the top)
#define TC_KB_STAGE_BYTES (64 * 1024)
static int tc_kb_stage(int a_rows, int bn) {
    const int kb = (a_rows + bn) * TC_BK * 2;
    return 2 * kb <= TC_KB_STAGE_BYTES ? 2 : 1;
}

// Sets of accumulators (one a part) that tensor memory's 512 columns have room for: two, so that the epilogue of a tile runs
// under the main loop of the next, one, or none.
static int tc_sets(int bn, int inner) { return 2 * inner * bn <= 512 ? 2 : (inner * bn <= 512 ? 1 : 0); }

static int tc_a_rows(int M) { return M >= TC_BM ? TC_BM : (M + 7) / 8 * 8; }

// Can parts along K of a tile `w` wide run at all: all units in one round, no part under two k-blocks (false for more parts,
// too) ...
static bool tc_split_starts(int K, int sp, int tiles) {
    return tiles * sp <= tc_n_sm() && sp * 2 <= (K + TC_BK - 1) / TC_BK;
}
// ... the clusters all run at once, and no part is empty?
static bool tc_split_runs(int M, int K, int epi, int w, int sp, int tiles) {
    if (tiles > tc_max_clusters(w, epi, sp, tc_a_rows(M))) return false;
    const int n_kb = (K + TC_BK - 1) / TC_BK, kbs = (n_kb + sp - 1) / sp;
    return (n_kb + kbs - 1) / kbs == sp;
}

// Parts along K.  They alone decide an output's bits: its k-blocks are added in order within a part, the parts in order,
// whatever the tile's width and whoever runs it.  And the tensor core cuts the sum off at every addition, so the error of
// a sum grows with the length of its part (float32 sums against 64 bits, 2-norm: 2048 k's in one part 2.1e-6, in two
// 1.0e-6, in four 4.7e-7).  So this rule is not a matter of speed alone: it is kept as it is, and tc_choose looks for the
// fastest way to run what it gives.
//
// It counts the bytes that the busiest SM brings in, about 45 GB/s an SM whatever the source -- its share of W and, for
// every tile, all the rows of A.  Unsplit, a narrow tile reads A once for a few rows of W (64 rows by 2048 x 5632 in
// 32-row tiles: 720 KB of A for 360 KB of W) and wide tiles leave SMs idle.  So products of 17 to 1024 rows are cut where
// the units (tile, part) fill one round over the SMs and a unit brings in fewer bytes; the price of the split (partial
// sums out and in, the wait for the other parts) is counted as TC_SPLIT_COST of traffic.
static int tc_parts(int M, int N, int K, int epi) {
    const bool gated = epi == EPI_SWIGLU;
    const int n_out = gated ? N / 2 : N, sms = tc_n_sm(), n_kb = (K + TC_BK - 1) / TC_BK;
    const int m_tiles = (M + TC_BM - 1) / TC_BM, rows = M < TC_BM ? M : TC_BM, a_rows = tc_a_rows(M);
    if (M <= 16 || m_tiles > TC_SPLIT_MAX_M_TILES) return 1;
    long long best = -1;
    int parts = 1;
    for (int w = 256; w >= 64; w /= 2) {
        const int cols = gated ? w / 2 : w, tiles = (n_out + cols - 1) / cols * m_tiles;
        for (int sp = 1; sp <= 8; sp++) {
            if (sp > 1 && !tc_split_starts(K, sp, tiles)) break;
            if (sp > 1 && !tc_split_runs(M, K, epi, w, sp, tiles)) continue;
            const int kbs = (n_kb + sp - 1) / sp;
            long long cost = (sp == 1 ? (long long)((tiles + sms - 1) / sms) * n_kb : kbs) * (TC_BK * 2) * (w + a_rows);
            if (sp > 1) cost += TC_SPLIT_COST + (long long)rows * w * 4 * (sp - 1) / sp;   // (the sums come in over the same port)
            if (best < 0 || cost < best) { best = cost; parts = sp; }
        }
    }
    return parts;
}

// The fastest way to run the parts that tc_parts gives: the choice that keeps the busiest SM busy for the shortest time,
// counted in bytes brought into it (about 100 a nanosecond, from L2 or, all SMs together, HBM):
//   a k-block: its rows of A and W, but no less than TC_KB_MIN (waiting, issuing, handing on);
//   an epilogue: 0.6 KB a column of the tile, 1 KB gated, under the main loop of the next tile if there is one;
//   parts one after the other: 6 KB a part more and 64 columns, for reading its sums;
//   parts by a cluster (all units in one round): 20 KB and 1.4 KB a CTA for the exchange, five times the sums that are
//   exchanged, a little more for clusters of other than 2 or 4 CTAs;
//   a pair: TC_PAIR_COST for its barriers, and more for parts behind a gated epilogue, which is short of registers.
// It was fitted to all that can run at 17 to 1000 rows of twelve layer products (1,087 timings): within 1 % of the best on average,
// 23 % at worst (128 rows by 3072 x 2048, five parts by a cluster or by one CTA of 32 columns).  Measured, us, the
// choice before the exchange by copies | now: 64 rows by 2048 x 2048 7.8 | 6.7, 128 by 2048 x 5632 16.2 | 13.7, 200 by
// 1024 x 4608 13.7 | 11.3; gated 600 rows by 9216 x 1024 25.2 | 20.9 (weights from HBM).
static TcChoice tc_choose(int M, int N, int K, int epi, int split) {
    const bool gated = epi == EPI_SWIGLU;
    const int n_out = gated ? N / 2 : N, sms = tc_n_sm(), n_kb = (K + TC_BK - 1) / TC_BK;
    const int m_tiles = (M + TC_BM - 1) / TC_BM, rows = M < TC_BM ? M : TC_BM, a_rows = tc_a_rows(M);
    const auto tiles_at = [&](int w) { const int cols = gated ? w / 2 : w; return (long long)((n_out + cols - 1) / cols); };
    const auto kb_cost = [](long long r) { const long long bytes = r * TC_BK * 2; return bytes > TC_KB_MIN ? bytes : (long long)TC_KB_MIN; };
    const auto epi_cost = [&](int w) { return (long long)w * (gated ? 1000 : 614); };
    const auto run_cost = [&](long long rounds, long long main, int w) {
        return rounds * (main > epi_cost(w) ? main : epi_cost(w)) + epi_cost(w);
    };
    const int parts = split ? tc_parts(M, N, K, epi) : 1;
    const auto parts_cost = [&](int w) { return (parts - 1LL) * 6 * 1024 * (w > 64 ? w / 64 : 1); };
    TcChoice ch = {0, parts, false, false};
    long long best = -1;
    for (int w = 256; w >= (gated ? 64 : 32); w /= 2) {
        if (!tc_sets(w, parts)) continue;
        const long long tiles = tiles_at(w) * m_tiles;
        const long long cost = run_cost((tiles + sms - 1) / sms, n_kb * kb_cost(w + a_rows), w) + parts_cost(w);
        if (best < 0 || cost < best) { best = cost; ch = {w, parts, false, false}; }
    }
    for (int w = 256; parts > 1 && w >= 64; w /= 2) {
        const int tiles = (int)(tiles_at(w) * m_tiles), kbs = (n_kb + parts - 1) / parts;
        if (!tc_split_starts(K, parts, tiles) || !tc_split_runs(M, K, epi, w, parts, tiles) || tc_smem(M, a_rows, w, gated, parts).bytes > KP_SMEM_MAX) continue;
        const long long cost = kbs * kb_cost(w + a_rows) + epi_cost(w) / parts + 20 * 1024 + tiles * parts * 1434LL +
                               5LL * rows * w * 4 * (parts - 1) / parts + (parts != 2 && parts != 4 ? 20 * 1024 : 0);
        if (cost < best) { best = cost; ch = {w, parts, true, false}; }
    }
    for (int w = 256; m_tiles > 1 && w >= 128; w /= 2) {
        if (!tc_sets(w, parts)) continue;
        const long long tiles = tiles_at(w) * ((M + 2 * TC_BM - 1) / (2 * TC_BM));
        const long long cost = run_cost((tiles + sms / 2 - 1) / (sms / 2), n_kb * kb_cost(w / 2 + TC_BM), w) + TC_PAIR_COST +
                               parts_cost(w) + (gated && parts > 1 ? 150 * 1024 : 0);
        if (cost < best) { best = cost; ch = {w, parts, false, true}; }
    }
    return ch;
}

extern "C" {

// epi: 0 store bf16, 1 store f32, 2 accumulate into f32, 3 SwiGLU (W = [gate; up], N = 2*ff, output [M, ff] bf16),
// 6 store bf16 behind the activation of bits 8 and up.
// split: products of 17 to 1024 rows may be cut along K (0: never).
// glu: limit, alpha and shift of the gated unit with limits (activation code 3 in epi), else null.
static int tc_run(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N,
                  int K, int epi, int split, const float* glu, const TcChoice* as, void* stream);

int kp_gemm_tc_split(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N,
                     int K, int epi, int split, void* stream) {
    return tc_run(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, split, nullptr, nullptr, stream);
}

int kp_gemm_tc_split_glu(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N,
                         int K, int epi, int split, float limit, float alpha, float shift, void* stream) {
    const float glu[3] = {limit, alpha, shift};
    return tc_run(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, split, glu, nullptr, stream);
}

// out[0..3]: the tile width, the parts along K, whether a cluster shares them and whether pairs of CTAs run a product (epi:
// its kind, without an activation)
int kp_gemm_tc_choice(int M, int N, int K, int epi, int split, int* out) {
    if (M <= 0 || N <= 0 || K < 8 || (K & 7)) return KP_ERR_BAD_ARG;
    const TcChoice ch = tc_choose(M, N, K, epi, split);
    out[0] = ch.bn; out[1] = ch.parts; out[2] = ch.cluster ? 1 : 0; out[3] = ch.pair ? 1 : 0;
    return 0;
}

// kp_gemm_tc_split_glu (limit 0: the activation of epi) with all that given, where it can run
int kp_gemm_tc_as(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N, int K,
                  int epi, int bn, int parts, int cluster, int pair, float limit, float alpha, float shift, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int kind = KP_EPI_KIND(epi), n_kb = (K + TC_BK - 1) / TC_BK;
    const bool gated = kind == EPI_SWIGLU;
    const int cols = gated ? bn / 2 : bn, n_out = gated ? N / 2 : N, m_tiles = (M + TC_BM - 1) / TC_BM;
    if (bn != 256 && bn != 128 && bn != 64 && !(bn == 32 && !gated)) return KP_ERR_BAD_ARG;
    if (parts < 1 || parts > 8 || (cluster && (pair || parts == 1 || bn < 64))) return KP_ERR_BAD_ARG;
    if (pair && (bn < 128 || m_tiles < 2)) return KP_ERR_UNSUPPORTED;
    if (cluster) {
        const long long tiles = (long long)((n_out + cols - 1) / cols) * m_tiles;
        if (tiles > 65535 || !tc_split_starts(K, parts, (int)tiles) || !tc_split_runs(M, K, kind, bn, parts, (int)tiles)) return KP_ERR_UNSUPPORTED;
        // Five parts or more of 256 columns by 121 rows and more: the sums that go out and come in do not fit beside one another.
        // The same parts, and so the same bits, by a cluster for each half of the columns, or one after the other.
        if (tc_smem(M, tc_a_rows(M), bn, gated, parts).bytes > KP_SMEM_MAX) {
            const long long halves = (long long)((n_out + cols / 2 - 1) / (cols / 2)) * m_tiles;
            cluster = halves <= 65535 && tc_split_starts(K, parts, (int)halves) && tc_split_runs(M, K, kind, bn / 2, parts, (int)halves);
            bn = cluster ? bn / 2 : 64;
        }
    } else {
        const int kbs = (n_kb + parts - 1) / parts;
        if (!tc_sets(bn, parts) || (n_kb + kbs - 1) / kbs != parts) return KP_ERR_UNSUPPORTED;
    }
    const TcChoice ch = {bn, parts, cluster != 0, pair != 0};
    const float glu[3] = {limit, alpha, shift};
    return tc_run(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, 1, limit > 0.f ? glu : nullptr, &ch, stream);
}

static int tc_run(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N,
                  int K, int epi, int split, const float* glu, const TcChoice* as, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int act = KP_EPI_ACT(epi);
    epi = KP_EPI_KIND(epi);
    if (act != KP_ACT_SILU && act != KP_ACT_RELU && act != KP_ACT_GELU_TANH && !(act == KP_ACT_GLU_CLAMPED && glu) &&
        !(act == KP_ACT_RELU_SQ && epi == EPI_ACT)) return KP_ERR_UNSUPPORTED;
    if (K < 8 || (K & 7) || (lda & 7) || (ldw & 7) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return KP_ERR_UNSUPPORTED;
    if ((long long)((M + TC_BM - 1) / TC_BM) > 65535) return KP_ERR_UNSUPPORTED;
    TcArgs a = {};
    a.bias = bias; a.C = C; a.ldc = ldc; a.M = M; a.N = N; a.K = K; a.ff = 0; a.act = act;
    if (glu) { a.glu_limit = glu[0]; a.glu_alpha = glu[1]; a.glu_shift = glu[2]; }
    {
        const int esz = (epi == EPI_STORE || epi == EPI_SWIGLU || epi == EPI_ACT) ? 2 : 4;
        a.vec_ok = (((uintptr_t)C & 15) == 0 && ((size_t)ldc * esz) % 16 == 0) ? 1 : 0;
    }
    if (epi == EPI_SWIGLU) {
        if (N & 1) return KP_ERR_BAD_ARG;
        a.ff = N / 2;
    }
    const TcChoice ch = as ? *as : tc_choose(M, N, K, epi, split);
    const int bn = ch.bn, pair_bn = ch.pair ? ch.bn : 0, n_kb = (K + TC_BK - 1) / TC_BK;
    a.splits = ch.cluster ? ch.parts : 1;
    a.inner = ch.cluster ? 1 : ch.parts;
    a.kb_per_part = (n_kb + ch.parts - 1) / ch.parts;
    a.n_sets = tc_sets(bn, a.inner);
    for (a.tmem_cols = 32; a.tmem_cols < a.n_sets * a.inner * bn;) a.tmem_cols *= 2;
    a.a_rows = tc_a_rows(M);
    cudaStream_t s = (cudaStream_t)stream;
    a.kb_stage = !ch.pair && K % TC_BK == 0 && n_kb > 1 ? tc_kb_stage(a.a_rows, bn) : 1;
    alignas(64) CUtensorMap ta, tw;
    int st;
    if (a.kb_stage > 1) {
        st = kp_make_map_bf16_groups(&ta, A, (unsigned long long)M, n_kb, lda, a.a_rows, a.kb_stage);
        if (!st) st = epi == EPI_SWIGLU ? kp_make_map_bf16_halves(&tw, W, (unsigned long long)a.ff, n_kb, ldw, bn / 2, a.kb_stage)
                                        : kp_make_map_bf16_groups(&tw, W, (unsigned long long)N, n_kb, ldw, bn, a.kb_stage);
    } else {
        st = kp_make_map_bf16_2d(&ta, A, (unsigned long long)M, K, lda, TC_BK, a.a_rows);
        if (!st) st = kp_make_map_bf16_2d(&tw, W, (unsigned long long)N, K, ldw, TC_BK, pair_bn ? pair_bn / 2 : (epi == EPI_SWIGLU ? bn / 2 : bn));
    }
    if (st) return st;
    if (pair_bn) {
#define TC_PAIR_BN(EPI, PARTS) return pair_bn == 256 ? launch_pair<256, EPI, PARTS>(ta, tw, a, s) : launch_pair<128, EPI, PARTS>(ta, tw, a, s)
#define TC_PAIR(EPI) do { if (a.inner > 1) TC_PAIR_BN(EPI, true); TC_PAIR_BN(EPI, false); } while (0)
        switch (epi) {
            case EPI_STORE: TC_PAIR(EPI_STORE);
            case EPI_STORE_F32: TC_PAIR(EPI_STORE_F32);
            case EPI_ACCUM_F32: TC_PAIR(EPI_ACCUM_F32);
            case EPI_ACT: TC_PAIR(EPI_ACT);
            case EPI_SWIGLU:
                if (a.act == KP_ACT_GLU_CLAMPED) TC_PAIR(EPI_GLU);
                if (a.act != KP_ACT_SILU) TC_PAIR(EPI_GATED_RT);
                TC_PAIR(EPI_SWIGLU);
            default: return KP_ERR_BAD_ARG;
        }
#undef TC_PAIR
#undef TC_PAIR_BN
    }
#define TC_PICK(EPI)                                               \
    switch (bn) {                                                  \
        case 256: return launch<256, EPI>(ta, tw, a, s);           \
        case 128: return launch<128, EPI>(ta, tw, a, s);           \
        case 64: return launch<64, EPI>(ta, tw, a, s);             \
        default: return launch<32, EPI>(ta, tw, a, s);             \
    }
    switch (epi) {
        case EPI_STORE: TC_PICK(EPI_STORE)
        case EPI_STORE_F32: TC_PICK(EPI_STORE_F32)
        case EPI_ACCUM_F32: TC_PICK(EPI_ACCUM_F32)
        case EPI_ACT: TC_PICK(EPI_ACT)
        case EPI_SWIGLU:
#define TC_PICK_GATED(EPI)                                         \
    switch (bn) {                                                  \
        case 256: return launch<256, EPI>(ta, tw, a, s);           \
        case 128: return launch<128, EPI>(ta, tw, a, s);           \
        default: return launch<64, EPI>(ta, tw, a, s);             \
    }
            if (a.act == KP_ACT_GLU_CLAMPED) TC_PICK_GATED(EPI_GLU)
            if (a.act != KP_ACT_SILU) TC_PICK_GATED(EPI_GATED_RT)
            TC_PICK_GATED(EPI_SWIGLU)
        default: return KP_ERR_BAD_ARG;
    }
#undef TC_PICK_GATED
#undef TC_PICK
}

int kp_gemm_tc(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N,
               int K, int epi, void* stream) {
    return kp_gemm_tc_split(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, 0, stream);
}

}  // extern "C"
