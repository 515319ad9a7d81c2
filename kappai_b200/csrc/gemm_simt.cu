// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) on the CUDA cores, float32 FMA.
//
// This is the matrix product of the true 32-bit path (no tensor-core mode of
// reduced precision is involved) and the general fallback of the bfloat16 path
// for shapes the tensor-core kernels refuse.  W is row-major [out][in] as in
// the reference (src/backend/cpu/scalar/quants.c:1367-1414).
//
// float32 operands with 16-byte rows run one of two kernels.  Both add an output's products in the same order,
// whatever M is: k is cut into stretches of 256, a stretch's even and odd k are two chains of FMAs from zero that are added
// at its end, and the stretches' sums are added in the order of k.  So a row's result does not depend on the rows beside it, the rows of a step can be
// cut anywhere, and long sums lose less than in one chain of K.
//
//  * gemm_f32_rows_kernel: few rows.  Bound by reading W once (4 bytes a weight).
//  * gemm_f32_tile_kernel: many rows.  Bound by the FMA rate (about 70 TFLOP/s of scalar FMA was measured on B200; the
//    packed two-element form gains nothing in rate but takes half the issue slots).
//
// Everything else (bfloat16 operands, rows that are not 16-byte aligned) runs gemm_nt_simt_kernel, which sums
// k = 0..K-1 in order.  The choice between the orders depends on type and alignment only, never on M.
#include "common.cuh"

#define EPI_STORE 0      // C (type T) = acc
#define EPI_STORE_F32 1  // C (float)  = acc
#define EPI_ACCUM_F32 2  // C (float) += acc        (residual sum in 32-bit)

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename T, int EPI>
__global__ void __launch_bounds__(256)
gemm_nt_simt_kernel(const T* __restrict__ A, const T* __restrict__ W, const float* __restrict__ bias,
                    void* __restrict__ Cv, int M, int N, int K, int lda, int ldw, int ldc) {
    kp_pdl_begin();
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;          // 16 x 16 threads, 4x4 outputs each
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64x16 elements per operand, 256 threads: 4 each
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e = tid + i * 256;
            const int r = e / BK, c = e % BK;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
            As[c][r] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.f;
            Ws[c][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; i++) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; j++) b[j] = Ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int gn = n0 + tx * TN + j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[gn];
            const size_t o = (size_t)gm * ldc + gn;
            if (EPI == EPI_STORE) ((T*)Cv)[o] = from_f32<T>(v);
            else if (EPI == EPI_STORE_F32) ((float*)Cv)[o] = v;
            else ((float*)Cv)[o] += v;
        }
    }
}

template <typename T>
static int launch(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, int lda, int ldw,
                  int ldc, int epi, cudaStream_t s) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (epi == EPI_STORE)
        kp_launch_pdl(gemm_nt_simt_kernel<T, EPI_STORE>, dim3(grid), dim3(256), 0, s, (const T*)A, (const T*)W, bias, C, M, N, K, lda, ldw, ldc);
    else if (epi == EPI_STORE_F32)
        kp_launch_pdl(gemm_nt_simt_kernel<T, EPI_STORE_F32>, dim3(grid), dim3(256), 0, s, (const T*)A, (const T*)W, bias, C, M, N, K, lda, ldw, ldc);
    else if (epi == EPI_ACCUM_F32)
        kp_launch_pdl(gemm_nt_simt_kernel<T, EPI_ACCUM_F32>, dim3(grid), dim3(256), 0, s, (const T*)A, (const T*)W, bias, C, M, N, K, lda, ldw, ldc);
    else
        return KP_ERR_BAD_ARG;
    return kp_launch_status();
}

// ------------------------------------------------------------------------------------------ float32, aligned rows

constexpr int F32_GROUP = 256;                       // k's of one chain of FMAs (see above)

struct F32Args {
    const float* A; const float* W; const float* bias; float* C;
    int M, N, K, lda, ldw, ldc;
    int w_settled;                                   // W is written by nothing that may still run: it may be read before the wait
};

// 16 bytes to shared memory without a register between; `ok` false: zeros, nothing is read
__device__ __forceinline__ void f32_cp16(void* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void f32_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void f32_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// two FMAs in one instruction: the chains of the even and of the odd k's
typedef unsigned long long f32x2;
__device__ __forceinline__ void f32_fma2(f32x2& d, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float f32_halves(f32x2 v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

template <int EPI> __device__ __forceinline__ void f32_store(const F32Args& p, int m, int n, float v) {
    if (p.bias) v += p.bias[n];
    float* c = p.C + (size_t)m * p.ldc + n;
    *c = EPI == EPI_ACCUM_F32 ? *c + v : v;
}

// Few rows.  A CTA owns 8 R rows of W; its warps cut K into jobs of 1024 columns = 4 stretches, and a lane (r, q) of a job
// sums stretch q of the rows r, r + 8, ... for MB rows of A, so that every chain stays in one lane.  A warp brings its
// job's W (and A) through a ring of its own in stages of 32 columns, by cp.async; nothing in the main loop waits for
// another warp.  The stages of a settled W that the ring holds are on their way before the wait on the kernel before
// (a decode step of the 350M shape: 2 % of its time), those of A behind it.  In shared memory the eight 16-byte chunks of a row's stage are permuted
// by the row (chunk c of row r at c ^ r), so the eight rows of a quarter warp read all banks once.
//
// SHARE: warps that share a job, each for MB / SHARE of the rows (see f32_rows).
//
// More rows than MB take the grid's y; W then comes from L2.  Measured (W from HBM): 8 rows by 2048 x 5632 in 13.3 us
// (3.5 TB/s; 608 us with tiles of 64 x 64 and a chain of K), 11264 x 2048 in 23 us, 65536 x 2048 in 93 us (5.8 TB/s); one
// row 10.6, 15.7 and 78 us (6.9 TB/s).  R = 4, MB = 16 reads shared memory least for its FMAs: 64 rows by 2048 x 5632 in
// 77 us against 84 with R = 2, MB = 8.
#define F32R_COLS 32                                  // columns of a stage
#define F32R_JOB (4 * F32_GROUP)                      // columns of a job
#define F32R_MAX_WARPS 8

template <int R, int MB, int EPI, int SHARE>
__global__ void __launch_bounds__(F32R_MAX_WARPS * SHARE * 32)
gemm_f32_rows_kernel(const F32Args p, int n_stages) {
    constexpr int W_BYTES = 8 * R * 4 * F32R_COLS * 4, A_BYTES = MB * 4 * F32R_COLS * 4, STAGE = W_BYTES + A_BYTES;
    constexpr int PER_JOB = F32_GROUP / F32R_COLS;    // stages of a job
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int MS = MB / SHARE;                    // rows of A that a warp sums
    const int part = (threadIdx.x >> 5) % SHARE, warp = (threadIdx.x >> 5) / SHARE;       // part: which of the warps that share a job
    const int lane = threadIdx.x & 31, n_warps = (blockDim.x >> 5) / SHARE;
    const int r = lane & 7, q = lane >> 3;
    const auto job_sync = [&]() {
        if (SHARE == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + warp), "n"(SHARE * 32) : "memory");
    };
    const int n0 = blockIdx.x * 8 * R, m0 = blockIdx.y * MB;
    const int K = p.K, n_jobs = (K + F32R_JOB - 1) / F32R_JOB;
    unsigned char* ring = smem + (size_t)warp * n_stages * STAGE;
    float* red = reinterpret_cast<float*>(smem + (size_t)n_warps * n_stages * STAGE);     // [stretch][MB][8 R]
    const int mine = n_jobs > warp ? (n_jobs - warp - 1) / n_warps + 1 : 0;               // jobs of this warp
    const int total = mine * PER_JOB;

    auto col_of = [&](int it) { return (warp + (it / PER_JOB) * n_warps) * F32R_JOB + (it % PER_JOB) * F32R_COLS; };
    // (a warp's 32 copies are 4 rows of a stretch by 8 chunks)
    const int cr = lane >> 3, cc = lane & 7;
    auto load_w = [&](int it) {
        unsigned char* dst = ring + (size_t)(it % n_stages) * STAGE;
        const int k0 = col_of(it) + cc * 4;
#pragma unroll
        for (int g = 0; g < 4; g++)
#pragma unroll
            for (int i = 0; i < 2 * R; i++) {
                if ((g * 2 * R + i) % SHARE != part) continue;
                const int row = i * 4 + cr, k = k0 + g * F32_GROUP;                       // row of the CTA's 8 R
                const float* src = p.W + (size_t)min(n0 + row, p.N - 1) * p.ldw + k;
                f32_cp16(dst + ((((row >> 3) * 4 + g) * 8 + (row & 7)) * 8 + (cc ^ (row & 7))) * 16, src, k < K);
            }
    };
    auto load_a = [&](int it) {
        unsigned char* dst = ring + (size_t)(it % n_stages) * STAGE + W_BYTES;
        const int k = col_of(it) + cc * 4 + cr * F32_GROUP;                               // stretch cr, chunk cc
#pragma unroll
        for (int i = 0; i < MS; i++) {
            const int m = part * MS + i;
            f32_cp16(dst + ((m * 4 + cr) * 8 + ((cc + 2 * cr) & 7)) * 16, p.A + (size_t)min(m0 + m, p.M - 1) * p.lda + k, k < K);
        }
    };

    const int ahead = n_stages - 1;
    KP_TRACE_MARK(0);
    if (!p.w_settled) pdl_wait();
#pragma unroll 1
    for (int it = 0; it < ahead && it < total; it++) load_w(it);
    pdl_wait();
    KP_TRACE_MARK(1);
    pdl_launch_dependents();
    // (the first stages' W is part of the first stage's group: it was asked for first and comes first)
#pragma unroll 1
    for (int it = 0; it < ahead; it++) {
        if (it < total) load_a(it);
        f32_cp_commit();
    }

    f32x2 acc[R][MS];
#pragma unroll 1
    for (int it = 0; it < total; it++) {
        if (it % PER_JOB == 0) {
#pragma unroll
            for (int i = 0; i < R; i++)
#pragma unroll
                for (int m = 0; m < MS; m++) acc[i][m] = 0;
        }
        // stage `it` has come: all but the ahead - 1 groups behind it
        switch (ahead) {
            case 1: f32_cp_wait<0>(); break;
            case 2: f32_cp_wait<1>(); break;
            case 3: f32_cp_wait<2>(); break;
            case 4: f32_cp_wait<3>(); break;
            case 5: f32_cp_wait<4>(); break;
            case 6: f32_cp_wait<5>(); break;
            default: f32_cp_wait<6>(); break;
        }
        job_sync();
        if (it + ahead < total) { load_w(it + ahead); load_a(it + ahead); }
        f32_cp_commit();
        const unsigned char* st = ring + (size_t)(it % n_stages) * STAGE;
        const ulonglong2* wr = reinterpret_cast<const ulonglong2*>(st) + (q * 8 + r) * 8;
        const ulonglong2* ar = reinterpret_cast<const ulonglong2*>(st + W_BYTES) + part * MS * 32 + q * 8;
#pragma unroll
        for (int c = 0; c < F32R_COLS / 4; c++) {
            ulonglong2 w[R];
#pragma unroll
            for (int i = 0; i < R; i++) w[i] = wr[i * 256 + (c ^ r)];
#pragma unroll
            for (int m = 0; m < MS; m++) {
                const ulonglong2 a = ar[m * 32 + ((c + 2 * q) & 7)];
#pragma unroll
                for (int i = 0; i < R; i++) { f32_fma2(acc[i][m], a.x, w[i].x); f32_fma2(acc[i][m], a.y, w[i].y); }
            }
        }
        if (it % PER_JOB == PER_JOB - 1) {
            const int g = (warp + (it / PER_JOB) * n_warps) * 4 + q;
#pragma unroll
            for (int i = 0; i < R; i++)
#pragma unroll
                for (int m = 0; m < MS; m++) red[((size_t)g * MB + part * MS + m) * 8 * R + i * 8 + r] = f32_halves(acc[i][m]);
        }
    }
    __syncthreads();
    const int n_groups = (K + F32_GROUP - 1) / F32_GROUP;
#pragma unroll 1
    for (int e = threadIdx.x; e < MB * 8 * R; e += blockDim.x) {
        const int m = m0 + e / (8 * R), n = n0 + e % (8 * R);
        if (m >= p.M || n >= p.N) continue;
        float v = 0.f;
        for (int g = 0; g < n_groups; g++) v += red[(size_t)g * MB * 8 * R + e];
        f32_store<EPI>(p, m, n, v);
    }
}

// Many rows.  A CTA of 256 threads computes 64 x 64 of C, a thread 4 x 4 of it (rows ty + 16 i, columns tx + 16 j).
// Stages of 32 columns of A and W come by cp.async as they lie in memory; a thread reads four k's of a row at a time (no
// transposed copy is needed), chunks permuted by the row as above.  A 16-byte read that neighbouring lanes share costs
// two slots of shared memory, one that lanes eight apart share four (measured), so lane bits 1 to 3 choose the row of A
// and bits 0 and 4 that of W.  Two CTAs an SM.
// Measured: 2,048 rows by 6144 x 2048 in 1.21 ms, 43 TFLOP/s, 513 rows by 2048 x 5632 in 325 us (one thread a 4 x 4 of a
// tile read with scalar, transposed copies: 647 us).  What is left is the dispatch of FMAs with three operands from
// registers of the same bank; 128 x 64 tiles (8 x 4 a thread) were within 4 % either way.
#define F32T_COLS 32
#define F32T_STAGES 3
#define F32T_SMEM (F32T_STAGES * 128 * F32T_COLS * 4 + 4 * 256 * 16)
template <int EPI>
__global__ void __launch_bounds__(256, 2)
gemm_f32_tile_kernel(const F32Args p) {
    constexpr int TMt = 4, ROWS = 16 * TMt, STAGE = (ROWS + 64) * F32T_COLS * 4;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ty = (warp & 1) * 8 + ((lane >> 1) & 7), tx = (warp >> 1) * 4 + (lane & 1) + ((lane >> 4) << 1);
    const int m0 = blockIdx.y * ROWS, n0 = blockIdx.x * 64;
    const int K = p.K, n_st = (K + F32T_COLS - 1) / F32T_COLS;
    const int lr = threadIdx.x >> 3, lc = threadIdx.x & 7;               // copies: 32 rows by 8 chunks at a time
    auto load = [&](int it, bool a, bool w) {
        unsigned char* dst = smem + (it % F32T_STAGES) * STAGE;
        const int k = it * F32T_COLS + lc * 4;
        if (a) {
#pragma unroll
            for (int i = 0; i < ROWS / 32; i++) {
                const int row = i * 32 + lr;
                f32_cp16(dst + (row * 8 + (lc ^ (row & 7))) * 16, p.A + (size_t)min(m0 + row, p.M - 1) * p.lda + k, k < K);
            }
        }
        if (w) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int row = i * 32 + lr;
                f32_cp16(dst + ((ROWS + row) * 8 + (lc ^ (row & 7))) * 16, p.W + (size_t)min(n0 + row, p.N - 1) * p.ldw + k, k < K);
            }
        }
    };
    KP_TRACE_MARK(0);
    if (!p.w_settled) pdl_wait();
    for (int it = 0; it < F32T_STAGES - 1 && it < n_st; it++) load(it, false, true);
    pdl_wait();
    KP_TRACE_MARK(1);
    pdl_launch_dependents();
    for (int it = 0; it < F32T_STAGES - 1; it++) {
        if (it < n_st) load(it, true, false);
        f32_cp_commit();
    }
    f32x2 acc[TMt][4];
    // the outputs' sums over the stretches so far lie in shared memory (registers are short), each thread's its own
    float4* sum = reinterpret_cast<float4*>(smem + F32T_STAGES * STAGE) + threadIdx.x;
#pragma unroll
    for (int i = 0; i < TMt; i++) {
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0;
        sum[i * 256] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int it = 0; it < n_st; it++) {
        f32_cp_wait<F32T_STAGES - 2>();
        __syncthreads();                                                 // the stage has come; the one before has been read
        if (it + F32T_STAGES - 1 < n_st) load(it + F32T_STAGES - 1, true, true);
        f32_cp_commit();
        const ulonglong2* as = reinterpret_cast<const ulonglong2*>(smem + (it % F32T_STAGES) * STAGE);
        const ulonglong2* ws = as + ROWS * 8;
#pragma unroll
        for (int c = 0; c < F32T_COLS / 4; c++) {
            ulonglong2 w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = ws[(tx + 16 * j) * 8 + (c ^ (tx & 7))];
#pragma unroll
            for (int i = 0; i < TMt; i++) {
                const ulonglong2 a = as[(ty + 16 * i) * 8 + (c ^ (ty & 7))];
#pragma unroll
                for (int j = 0; j < 4; j++) f32_fma2(acc[i][j], a.x, w[j].x);
#pragma unroll
                for (int j = 0; j < 4; j++) f32_fma2(acc[i][j], a.y, w[j].y);
            }
        }
        if (it % (F32_GROUP / F32T_COLS) == F32_GROUP / F32T_COLS - 1 || it == n_st - 1) {
#pragma unroll
            for (int i = 0; i < TMt; i++) {
                float4 v = sum[i * 256];
                v.x += f32_halves(acc[i][0]); v.y += f32_halves(acc[i][1]); v.z += f32_halves(acc[i][2]); v.w += f32_halves(acc[i][3]);
                sum[i * 256] = v;
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = 0;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TMt; i++) {
        const int m = m0 + ty + 16 * i;
        if (m >= p.M) continue;
        const float4 v = sum[i * 256];
        const float out[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx + 16 * j;
            if (n < p.N) f32_store<EPI>(p, m, n, out[j]);
        }
    }
}

static int f32_n_sm() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

// Which kernel runs, and how: R, MB, warps and ring stages of the few-row kernel, or tiles (R 0).
struct F32Choice { int R, MB, warps, stages; size_t smem; };

// The few-row kernel's warps and ring; `fits` false: not even one warp's ring and the stretches' sums have room.
static bool f32_rows_fit(int M, int N, int K, int R, int MB, F32Choice* c) {
    const int n_jobs = (K + F32R_JOB - 1) / F32R_JOB, stage = (8 * R + MB) * 4 * F32R_COLS * 4;
    const int most = R == 4 ? 4 : F32R_MAX_WARPS;
    const size_t red = (size_t)n_jobs * 4 * MB * 8 * R * 4;
    int warps = n_jobs < most ? n_jobs : (n_jobs + (n_jobs + most - 1) / most - 1) / ((n_jobs + most - 1) / most);
    while (warps > 1 && (size_t)warps * 2 * stage + red > KP_SMEM_MAX) warps--;      // (the order of the sums is the same)
    const long long ctas = (long long)((N + 8 * R - 1) / (8 * R)) * ((M + MB - 1) / MB);
    // one CTA an SM: all the ring that pays (a job has 8 stages); more: a third of the SM's memory each, or a sixth where a
    // CTA is a single warp (8 rows by 9216 x 1024: 19.5 us with a third, 11.5 with a sixth; 65536 x 1024 95 and 52; one row by
    // 6144 x 2048, two warps: 8.9 and 11.1)
    const size_t room = ctas <= f32_n_sm() ? 200 * 1024 : (warps == 1 ? 36 : 74) * 1024;
    int stages = red < room ? (int)((room - red) / ((size_t)warps * stage)) : 0;
    if (stages > 8) stages = 8;
    if (stages < 2) stages = 2;
    *c = {R, MB, warps, stages, (size_t)warps * stages * stage + red};
    return c->smem <= KP_SMEM_MAX && (M + MB - 1) / MB <= 65535;                     // (more rows of A than a grid has)
}

// K counts in every kernel alike, so the rule compares rounds over the SMs; measured at widths of 1024 to 11264, us, with
// rows of 8 | rows of 16 | tiles:
//   up to 24 rows: rows of 8 (16 rows by 2048 x 5632: 25 | 38 | 172; by 1024 x 1024: 8 | 19 | 32), but not for a wide W
//   with one job of K, whose CTAs are single warps (16 rows by 9216 x 1024: 30 | 21 | 40);
//   a round of rows of 16 takes 7.2 us for 1,000 k, one of tiles 30.5 (128 rows by 2048 x 5632: 165 | 152 | 172; 160 rows:
//   - | 190 | 173; 96 rows by 6144 x 2048: 98 | 82 | 121; 256 rows by 1024 x 1024: - | 22 | 33; 400 rows: - | 42 | 33);
//   where the sums leave room for fewer than four warps, a round of rows of 16 takes 18 us a turn of them (32 rows by
//   4096 x 4096, four warps: - | 41 | 127; x 7168, three: - | 111 | 219; 128 rows by 2048 x 12288, two: - | 422 | 375).
// A K whose stretches' sums leave no room for a ring (some 100,000 at 8 rows, 20,000 at rows of 16) goes to tiles.
static F32Choice f32_choose(int M, int N, int K) {
    const int sms = f32_n_sm();
    const auto rounds = [&](long long ctas) { return (ctas + sms - 1) / sms; };
    const auto cuts = [](int n, int size) { return (long long)((n + size - 1) / size); };
    F32Choice c;
    if (M <= 8 || (M <= 24 && (K > F32R_JOB || N <= 32 * sms))) {
        const int R = cuts(N, 16) < sms ? 1 : 2;                                     // 8 rows of W a CTA where 16 leave SMs idle
        if (f32_rows_fit(M, N, K, R, M == 1 ? 1 : M == 2 ? 2 : M <= 4 ? 4 : 8, &c)) return c;
    } else if (f32_rows_fit(M, N, K, 4, 16, &c)) {
        const long long jobs = (K + F32R_JOB - 1) / F32R_JOB, turns = (jobs + c.warps - 1) / c.warps;
        const long long row = turns > (jobs + 3) / 4 && 180000 * turns > 72LL * K ? 180000 * turns : 72LL * K;
        if (rounds(cuts(M, 16) * cuts(N, 32)) * row < rounds(cuts(M, 64) * cuts(N, 64)) * 305 * K) return c;
    }
    return {0, 0, 0, 0, 0};
}

template <int R, int MB, int EPI, int SHARE>
static int f32_rows_shared(const F32Args& p, const F32Choice& c, cudaStream_t s) {
    static std::atomic<unsigned long long> ready{0};
    const int st = kp_smem_limit(gemm_f32_rows_kernel<R, MB, EPI, SHARE>, KP_SMEM_MAX, ready);
    if (st) return st;
    const dim3 grid((p.N + 8 * R - 1) / (8 * R), (p.M + MB - 1) / MB);
    return (int)kp_launch_pdl(gemm_f32_rows_kernel<R, MB, EPI, SHARE>, grid, dim3(c.warps * SHARE * 32), c.smem, s, p, c.stages);
}

// Where K is one job, a CTA of up to 8 rows is a single warp, and few CTAs leave an SM with few warps: two warps then share the
// job (half of the rows each).  8 rows, us, one warp | two: 1024 x 1024 7.6 | 6.5, 3072 x 1024 10.0 | 9.2, 9216 x 1024 11.5 | 11.0;
// but 65536 x 1024 51.6 | 70.5, as W is then read twice from shared memory, which is what bounds many CTAs, and with several
// jobs as well: 2048 x 5632 13.1 | 16.0.
template <int R, int MB, int EPI>
static int f32_rows(const F32Args& p, const F32Choice& c, cudaStream_t s) {
    if constexpr (MB == 4 || MB == 8) {
        const long long ctas = (long long)((p.N + 8 * R - 1) / (8 * R)) * ((p.M + MB - 1) / MB);
        if (p.K <= F32R_JOB && ctas <= 4LL * f32_n_sm()) return f32_rows_shared<R, MB, EPI, 2>(p, c, s);
    }
    return f32_rows_shared<R, MB, EPI, 1>(p, c, s);
}

template <int EPI>
static int f32_run(const F32Args& p, cudaStream_t s) {
    const F32Choice c = f32_choose(p.M, p.N, p.K);
    if (c.R == 4) return f32_rows<4, 16, EPI>(p, c, s);
#define F32_ROWS(MB_) return c.R == 1 ? f32_rows<1, MB_, EPI>(p, c, s) : f32_rows<2, MB_, EPI>(p, c, s)
    switch (c.MB) {
        case 1: F32_ROWS(1);
        case 2: F32_ROWS(2);
        case 4: F32_ROWS(4);
        case 8: F32_ROWS(8);
    }
#undef F32_ROWS
    static std::atomic<unsigned long long> ready{0};
    const int st = kp_smem_limit(gemm_f32_tile_kernel<EPI>, F32T_SMEM, ready);
    return st ? st : (int)kp_launch_pdl(gemm_f32_tile_kernel<EPI>, dim3((p.N + 63) / 64, (p.M + 63) / 64), dim3(256), F32T_SMEM, s, p);
}

// out[0..3]: R, MB, warps and stages of the few-row kernel that runs a float32 product with 16-byte rows; R 0: tiles
extern "C" int kp_gemm_f32_choice(int M, int N, int K, int* out) {
    const F32Choice c = f32_choose(M, N, K);
    out[0] = c.R; out[1] = c.MB; out[2] = c.warps; out[3] = c.stages;
    return 0;
}

// w_settled: see F32Args (the general kernel waits first in any case)
extern "C" int kp_gemm_nt_simt(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, int lda,
                               int ldw, int ldc, int epi, int dtype, int w_settled, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return KP_ERR_BAD_ARG;
    if ((long long)((M + BM - 1) / BM) > 65535) return KP_ERR_UNSUPPORTED;
    if (dtype == KP_DTYPE_F32 && !((K | lda | ldw) & 3) && !(((uintptr_t)A | (uintptr_t)W) & 15)) {
        const F32Args p = {(const float*)A, (const float*)W, bias, (float*)C, M, N, K, lda, ldw, ldc, w_settled};
        if (epi == EPI_STORE || epi == EPI_STORE_F32) return f32_run<EPI_STORE>(p, (cudaStream_t)stream);
        if (epi == EPI_ACCUM_F32) return f32_run<EPI_ACCUM_F32>(p, (cudaStream_t)stream);
        return KP_ERR_BAD_ARG;
    }
    KP_DISPATCH_DTYPE(dtype, T, return launch<T>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, (cudaStream_t)stream));
    return 0;
}
