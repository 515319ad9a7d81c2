// C[M,N] = A[M,K] * W[N,K]^T for up to 8 rows of bfloat16: the products of a decode step.
//
// Such a product is a few microseconds long, and a step is a chain of a hundred of them.  Back to back, the time of
// gemm_stream.cu hardly depends on whether the weights come from HBM or lie in L2 (2048 x 5632: 8.3 us against 8.1), nor on
// its loads of A or its epilogue: what it waits for is the hand over of its rings between a producer and eight warps, a
// stage of 8 rows at a time, on two or three CTAs an SM.  Here nothing is handed over:
//
//  * Persistent CTAs of 256 threads, one an SM, walk tiles of W rows: 16 rows, or 8 where that spreads the rows more evenly; 8 gate and
//    the 8 matching up rows (gated epilogue); the 8 matching rows of B, C and X (conv step).
//  * The eight warps cut K: of every 512 columns warp w takes the blocks of 32 at w and w + 8.  Each brings its blocks of
//    the tile's rows (and of A) through a ring of its own by cp.async; no warp waits for another inside a tile.  The
//    rings are filled with weights, which depend on no earlier kernel, before the wait on the kernel before.
//  * W rows are the m side of mma.m16n8k16, the batch rows the n side.  A lane's operands are 16 bytes of one row (the
//    same permutation of k on both sides); the 16-byte chunks of odd rows are stored four places on, so that the eight
//    lanes of a quarter warp read all banks once.
//  * At a tile's end the warps' partial sums are added in warp order from zero.  The order of every sum is that of
//    gemm_stream.cu, so a row's result does not depend on which of the two ran.
//  * Behind an RMS norm (the normed form) a CTA brings the float32 rows in itself, norms them with the arithmetic of the norm
//    kernel for that many columns (rowwise.cu: the same order of the squares' sum, x times the scale times the weight, rounded
//    to bfloat16) and holds them beside the rings for all its tiles: the bits of the norm kernel and the product, without a
//    launch between the product in front and this one.  (The weighted rows rounded before the scale, which then goes to the sums,
//    saves two barriers a CTA but rounds a row elsewhere than with nine rows and more, and makes NaN of rows whose squares
//    overflow; and with a warp's own columns read by itself, 128 bytes at a time, it was slower: rounds of one request of the
//    1.2B shape 31.5 ms, this 31.1, of a short chat 8.12 and 7.83, of eight requests 44.3 and 43.8.  Left to the product in
//    front -- it writes the weighted rows and sums of squares, this one reads both -- a step took 3 % longer.)
//
// Measured back to back, us, gemm_stream | this, one row and 8: 2048 x 5632 7.8 | 6.5, 7.9 | 7.1; 6144 x 2048 6.8 | 5.2,
// 6.9 | 5.7; 2048 x 2048 3.8 | 2.6, 3.8 | 2.8; at 16 rows it loses (8.2 | 9.0), as A then weighs as much as W.
//
// Two CTAs an SM, of two products that follow one another: the next product's rings fill while this one still streams.  That
// pays only if every SM gets one of each, so accumulating products have small CTAs and the others, between which they
// stand, big ones of more than half an SM; and only if the SM's split between cache and shared memory allows it (it is
// set for the kernel that comes first: without the preference asked for in kp_smem_limit the second never came in).
// A decode step through eight layers, us, norms apart and a CTA an SM | norms apart, two | norms inside, two (five to eight rows: see
// rows_run): one request, 1024 columns 182 | 180 | 159, 1536 221 | 222 | 198, 2048 272 | 273 | 246, 2560 415 | 424 | 377; eight
// 191 | 189 | 173, 232 | 224 | 216, 293 | 285 | 273, 451 | 441 | 425.
// Big and small, KB, 64 steps of one request, 1.2B shape, ms: 148 + 78 32.1, 128 + 96 31.9, 116 + 110 32.2, 164 + 62 33.2.
//
// Epilogues as in gemm_stream.cu.  K a multiple of 512.  Loops are not unrolled where that gains nothing back to back: in a step
// the kernels' code is fetched anew at every launch.
#include "mma.cuh"

#define EPI_STORE 0
#define EPI_STORE_F32 1
#define EPI_ACCUM_F32 2
#define EPI_SWIGLU 3
#define EPI_CONV_STEP 4
#define EPI_ACT 6
#define EPI_CONV_ANY 7                       // inside this file only: EPI_CONV_STEP with other than three taps

#define RW_WARPS 8
#define RW_NORM_MAX_K 4096                   // columns up to which the normed form holds A (8 rows: 64 KB)
// Shared memory of a CTA: with a big ring, with a small ring, and of one that has the SM to itself.
#define RW_BIG (128 * 1024)
#define RW_SMALL (96 * 1024)
#define RW_ALONE (155 * 1024)
#define RW_MAX_STAGES 12

struct RowsArgs {
    const bf16* A; int lda;
    const bf16* W; int ldw;
    const float* bias;
    void* C; int ldc;
    int M, N, K, ff;                         // ff: output columns of an epilogue that joins rows of W (gated: N / 2; conv step: N / 3)
    int act;
    float glu_limit, glu_alpha, glu_shift;
    const float* conv_w; const float* conv_bias; float* conv_state;
    const int* seg_pos; const int* seg_slot;
    int conv_k;
    const float* X; int ldx;                 // the normed form: float32 rows, the norm's weight and eps
    const float* gamma; float eps;
};

// How a launch runs.  WR: rows of W a tile (8, 16, or 24: the conv step).  R: rows of A that are kept, at least M (1, 4 or 8).
// NORM: A is normed by the kernel and held beside the rings, which are of W alone.  ROOM: a size of the three above.
template <int WR, int R, bool NORM, int ROOM> struct RowsShape {
    static constexpr int MT = (WR + 15) / 16;                            // m16 tiles (of a 24-row tile's second one half is empty)
    static constexpr int W_BYTES = WR * 128, STAGE = W_BYTES + (NORM ? 0 : R * 128);
    static constexpr int SUMS = 2 * RW_WARPS * MT * 128 * 4 + 128;
    static constexpr int FIT = (ROOM - SUMS - (NORM ? 2048 * 2 * R : 0)) / (RW_WARPS * STAGE);
    static constexpr int S = FIT > RW_MAX_STAGES ? RW_MAX_STAGES : FIT;  // ring stages of a warp
    static_assert(S >= 2, "a ring of two stages at least");
    static constexpr size_t bytes(int K) {
        const size_t need = (size_t)RW_WARPS * S * STAGE + SUMS + (NORM ? (size_t)K * 2 * R : 0);
        return ROOM != RW_SMALL && need < ROOM ? (size_t)ROOM : need;   // (more than half an SM: two of one product never share one)
    }
};

// LONG: the normed form of more than 2048 columns.  EPI_CONV_STEP has three taps, EPI_CONV_ANY any number.
template <int WR, int EPI, int R, bool NORM, int ROOM, bool LONG>
__global__ void __launch_bounds__(RW_WARPS * 32, 1)
gemm_rows_kernel(const RowsArgs p) {
    using Shape = RowsShape<WR, R, NORM, ROOM>;
    constexpr int MT = Shape::MT, W_BYTES = Shape::W_BYTES, STAGE = Shape::STAGE, S = Shape::S;
    constexpr bool CONV = EPI == EPI_CONV_STEP || EPI == EPI_CONV_ANY;
    constexpr int JOINS = CONV ? 3 : (EPI == EPI_SWIGLU ? 2 : 1);
    constexpr int TROWS = WR / JOINS;                                    // output columns a tile
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int M = p.M, n_out = JOINS > 1 ? p.ff : p.N;
    const int n_tiles = (n_out + TROWS - 1) / TROWS, n_ch = p.K / 512;   // chunks of 64 columns a warp and tile
    unsigned char* ring = smem + (size_t)warp * S * STAGE;
    float* red = reinterpret_cast<float*>(smem + (size_t)RW_WARPS * S * STAGE);   // [2][warp][MT][4][32]
    // (NORM) the rows' 1 / root mean square, then for every warp its columns of A [chunk][row][64], laid out as a stage's
    float* scales = red + 2 * RW_WARPS * MT * 128;
    unsigned char* held0 = reinterpret_cast<unsigned char*>(scales + 32);
    const unsigned char* held = held0 + (size_t)warp * n_ch * (R * 128);
    const int ga = g < R ? g : R - 1;                                    // the row of A this lane's fragments are of
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - blockIdx.x - 1) / gridDim.x + 1 : 0;
    const int total = my_tiles * n_ch;

    const int cr = lane >> 3, cc = lane & 7;                             // copies: 4 rows by 8 chunks at a time
    const int col0 = warp * 32 + (cc >> 2) * 256 + (cc & 3) * 8;         // this lane's column of a warp's chunk 0
    int ld_tile = blockIdx.x, ld_c = 0, ld_s = 0;                        // the next stage to be asked for
    auto load_w = [&](int tile, int c, int s) {
        unsigned char* dst = ring + (size_t)s * STAGE;
        const int n0 = tile * TROWS;
#pragma unroll
        for (int i = 0; i < WR / 4; i++) {
            const int row = i * 4 + cr;                                  // row of the tile
            const int wrow = JOINS > 1 ? (row >> 3) * p.ff + min(n0 + (row & 7), n_out - 1) : min(n0 + row, n_out - 1);
            cp_async16(dst + row * 128 + ((cc ^ ((row & 1) << 2)) * 16), p.W + (size_t)wrow * p.ldw + c * 512 + col0, true);
        }
    };
    auto load_a = [&](int c, int s) {
        unsigned char* dst = ring + (size_t)s * STAGE + W_BYTES;
#pragma unroll
        for (int i = 0; i < (R + 3) / 4; i++) {
            const int row = i * 4 + cr;
            if (row < M) cp_async16(dst + row * 128 + ((cc ^ ((row & 1) << 2)) * 16), p.A + (size_t)row * p.lda + c * 512 + col0, true);
        }
    };
    auto advance = [&]() {
        if (++ld_c == n_ch) { ld_c = 0; ld_tile += gridDim.x; }
        if (++ld_s == S) ld_s = 0;
    };

    KP_TRACE_MARK(0);
    pdl_launch_dependents();                                             // (what comes next reads nothing before its own wait)
#pragma unroll 1
    for (int i = 0; i < S; i++) {
        if (i < total) { load_w(ld_tile, ld_c, ld_s); advance(); }
        cp_async_commit();
    }
    if constexpr (NORM) {
        // A thread has the float4s threadIdx.x, + 256, ... of every row; the first KEEP of each stay in registers (all of them, but
        // for more than 2048 columns of more than four rows: 128 registers).
        constexpr int KEEP = LONG && R <= 4 ? 4 : 2;
        const int tid = threadIdx.x, n4 = p.K >> 2;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const auto x_at = [&](int r, int i) { return r < M && i < n4 ? *reinterpret_cast<const float4*>(p.X + (size_t)r * p.ldx + i * 4) : zero; };
        const auto gamma_at = [&](int i) { return i < n4 ? *reinterpret_cast<const float4*>(p.gamma + i * 4) : zero; };
        const auto squares = [](const float4& x, float ss) { return fmaf(x.w, x.w, fmaf(x.z, x.z, fmaf(x.y, x.y, fmaf(x.x, x.x, ss)))); };
        pdl_wait();
        KP_TRACE_MARK(1);
        float4 v[R][KEEP], gm[KEEP];
#pragma unroll
        for (int j = 0; j < KEEP; j++) {
#pragma unroll
            for (int r = 0; r < R; r++) v[r][j] = x_at(r, tid + j * 256);
            gm[j] = gamma_at(tid + j * 256);
        }
        float ss[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            ss[r] = 0.f;
#pragma unroll
            for (int j = 0; j < KEEP; j++) ss[r] = squares(v[r][j], ss[r]);
        }
        if (LONG && R > 4) {
#pragma unroll 1
            for (int j = KEEP; j * 256 < n4; j++)
#pragma unroll
                for (int r = 0; r < R; r++) ss[r] = squares(x_at(r, tid + j * 256), ss[r]);
        }
        // the sum over the threads, as the norm kernel of that size has it: up to 2048 columns the warps' values lane by lane, in
        // the order of the warps, then the lanes; beyond, the lanes of a warp, then the warps
        constexpr bool by_lane = !LONG;
        float* part = red;                                               // [row][warp][lane], or [row][256] by warp
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float q = by_lane ? ss[r] : warp_sum(ss[r]);
            if (by_lane || lane == 0) part[r * 256 + (by_lane ? tid : warp)] = q;
        }
        __syncthreads();
        const auto scale_of = [&](int r) {
            float q;
            if (by_lane) {
                q = part[r * 256 + lane];
#pragma unroll
                for (int w8 = 1; w8 < RW_WARPS; w8++) q += part[r * 256 + w8 * 32 + lane];
            } else {
                q = lane < RW_WARPS ? part[r * 256 + lane] : 0.f;
            }
            return 1.0f / sqrtf(warp_sum(q) / (float)p.K + p.eps);
        };
        float scale[R];
        if (R == 1) {
            scale[0] = scale_of(0);                                      // (every warp: that saves a barrier)
        } else {
            if (warp < R) scales[warp] = scale_of(warp);
            __syncthreads();
#pragma unroll
            for (int r = 0; r < R; r++) scale[r] = scales[r];
        }
        // column 4 i is of chunk i / 128, there of half i / 64 % 2, there of warp i / 8 % 8 (see load_a)
        const auto hold = [&](int r, int i, const float4& x, const float4& g4) {
            if (r >= M || i >= n4) return;
            const int j = (i >> 6 & 1) * 8 + (i & 7);
            *reinterpret_cast<uint2*>(held0 + (size_t)((i >> 3 & 7) * n_ch + (i >> 7)) * (R * 128) + r * 128 + (((j >> 1) ^ ((r & 1) << 2)) * 16) + (j & 1) * 8) =
                make_uint2(pack_bf16((x.x * scale[r]) * g4.x, (x.y * scale[r]) * g4.y), pack_bf16((x.z * scale[r]) * g4.z, (x.w * scale[r]) * g4.w));
        };
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int j = 0; j < KEEP; j++) hold(r, tid + j * 256, v[r][j], gm[j]);
        if (LONG && R > 4) {
#pragma unroll 1
            for (int j = KEEP; j * 256 < n4; j++) {
                const float4 g4 = gamma_at(tid + j * 256);
#pragma unroll
                for (int r = 0; r < R; r++) hold(r, tid + j * 256, x_at(r, tid + j * 256), g4);
            }
        }
        __syncthreads();
    } else {
        pdl_wait();
        KP_TRACE_MARK(1);
#pragma unroll 1
        for (int i = 0; i < S; i++) {
            if (i < total) load_a(i % n_ch, i);
            cp_async_commit();
        }
    }

    int s = 0, buf = 0;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, buf ^= 1) {
        const int n0 = tile * TROWS;
        // what the epilogue needs beside the sums is asked for now: its trips to L2 run under the main loop
        constexpr int PRE = EPI == EPI_CONV_STEP ? 2 : 3;                // kept inputs fetched ahead, with their taps, and the last tap
        float pre_c = 0.f, pre_hist[PRE] = {}, pre_cw[PRE] = {}, pre_last = 0.f;
        bool pre_fresh = false;
        const int om = threadIdx.x / TROWS, on = n0 + threadIdx.x % TROWS;   // this thread's output (the first TROWS * M threads)
        const bool mine = om < M && on < n_out;
        const int Kc = EPI == EPI_CONV_STEP ? 3 : p.conv_k;
        if (mine) {
            if (EPI == EPI_ACCUM_F32) pre_c = ((const float*)p.C)[(size_t)om * p.ldc + on];
            if (CONV) {                                                  // (a new request's kept inputs count as zeros below, so that
                pre_fresh = p.seg_pos[om] == 0;                          //  nothing here waits for its position)
                const float* st = p.conv_state + (size_t)p.seg_slot[om] * (Kc - 1) * p.ff + on;
                const float* cw = p.conv_w + (size_t)on * Kc;
#pragma unroll
                for (int k = 0; k < PRE; k++) {
                    const int kk = min(k, Kc - 2);
                    pre_hist[k] = st[(size_t)kk * p.ff];
                    pre_cw[k] = cw[kk];
                }
                pre_last = cw[Kc - 1];
            }
        }
        float acc[MT][4];
#pragma unroll
        for (int a = 0; a < MT; a++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[a][i] = 0.f;
#pragma unroll 1
        for (int c = 0; c < n_ch; c++) {
            cp_async_wait<S - 1>();                                      // this stage has come, all but the S - 1 behind it
            __syncwarp();
            const unsigned char* st = ring + (size_t)s * STAGE;
#pragma unroll
            for (int b = 0; b < 2; b++) {                                // the blocks of 32 columns
                const int at = ((b * 4 + t) ^ ((g & 1) << 2)) * 16;
                uint4 w[2 * MT];
#pragma unroll
                for (int i = 0; i < 2 * MT; i++) w[i] = i * 8 < WR ? *reinterpret_cast<const uint4*>(st + (i * 8 + g) * 128 + at) : make_uint4(0, 0, 0, 0);
                const uint4 x = *reinterpret_cast<const uint4*>((NORM ? held + (size_t)c * (R * 128) : st + W_BYTES) + ga * 128 + ((b * 4 + t) ^ ((ga & 1) << 2)) * 16);   // (rows beyond M: any values, nobody reads their sums)
#pragma unroll
                for (int a = 0; a < MT; a++) {
                    mma_bf16(acc[a], w[2 * a].x, w[2 * a + 1].x, w[2 * a].y, w[2 * a + 1].y, x.x, x.y);
                    mma_bf16(acc[a], w[2 * a].z, w[2 * a + 1].z, w[2 * a].w, w[2 * a + 1].w, x.z, x.w);
                }
            }
            __syncwarp();                                                // the stage has been read
            if (ld_tile < n_tiles) {
                load_w(ld_tile, ld_c, ld_s);
                if (!NORM) load_a(ld_c, ld_s);
                advance();
            }
            cp_async_commit();
            if (++s == S) s = 0;
        }
        // acc[a]: rows of W 16 a + g (elements 0, 1) and 16 a + g + 8 (2, 3), batch rows 2 t, 2 t + 1
        float* r = red + (size_t)buf * RW_WARPS * MT * 128;
#pragma unroll
        for (int a = 0; a < MT; a++)
#pragma unroll
            for (int i = 0; i < 4; i++) r[(warp * MT + a) * 128 + i * 32 + lane] = acc[a][i];
        __syncthreads();                                                 // (the other half of `red` is free: its readers were here)
        if (mine) {
            // the sum of W row `row` of the tile for this thread's batch row, over the warps in order
            auto sum_of = [&](int row) {
                const int a = row >> 4, i = ((row & 8) ? 2 : 0) + (om & 1), l = (row & 7) * 4 + (om >> 1);
                float v = 0.f;
#pragma unroll
                for (int w8 = 0; w8 < RW_WARPS; w8++) v += r[(w8 * MT + a) * 128 + i * 32 + l];
                return v;
            };
            const int m = om, n = on, lr = on - n0;
            float v = sum_of(lr);
            if (p.bias) v += p.bias[n];
            const size_t o = (size_t)m * p.ldc + n;
            if (CONV) {
                float cg = sum_of(8 + lr), xv = sum_of(16 + lr);
                if (p.bias) { cg += p.bias[p.ff + n]; xv += p.bias[2 * p.ff + n]; }
                // B, C and X as the separate product stores them, then shortconv.cu's decode step: every product and
                // sum rounded on its own (src/backend/cpu/common.c:2393-2431)
                const float b = to_f32(from_f32<bf16>(v)), cq = to_f32(from_f32<bf16>(cg)), xq = to_f32(from_f32<bf16>(xv));
                const int d = p.ff;
                float* st = p.conv_state + (size_t)p.seg_slot[m] * (Kc - 1) * d;
                const float bx = __fmul_rn(b, xq);
                float sum;
#pragma unroll
                for (int k = 0; k < PRE; k++) pre_hist[k] = pre_fresh ? 0.f : pre_hist[k];
                if (EPI == EPI_CONV_STEP || Kc == 3) {
                    sum = __fadd_rn(__fadd_rn(__fmul_rn(pre_hist[0], pre_cw[0]), __fmul_rn(pre_hist[1], pre_cw[1])), __fmul_rn(bx, pre_last));
                } else {
                    sum = __fmul_rn(bx, pre_last);
#pragma unroll
                    for (int k = 0; k < PRE; k++)
                        if (k < Kc - 1) sum = __fadd_rn(sum, __fmul_rn(pre_hist[k], pre_cw[k]));
                }
#pragma unroll
                for (int k = 1; k < PRE; k++)
                    if (k < Kc - 1) st[(size_t)(k - 1) * d + n] = pre_hist[k];
                if (EPI == EPI_CONV_ANY && Kc > 4) {                     // more taps: four at a time, their loads in front of the stores
                    const float* cw = p.conv_w + (size_t)n * Kc;
#pragma unroll 1
                    for (int k0 = PRE; k0 < Kc - 1; k0 += 4) {
                        float h[4], t4[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const bool in = k0 + k < Kc - 1;
                            h[k] = in && !pre_fresh ? st[(size_t)(k0 + k) * d + n] : 0.f;
                            t4[k] = in ? cw[k0 + k] : 0.f;
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (k0 + k < Kc - 1) { sum = __fadd_rn(sum, __fmul_rn(h[k], t4[k])); st[(size_t)(k0 + k - 1) * d + n] = h[k]; }
                    }
                }
                st[(size_t)(Kc - 2) * d + n] = bx;
                if (p.conv_bias) sum = __fadd_rn(sum, p.conv_bias[n]);
                ((bf16*)p.C)[o] = from_f32<bf16>(__fmul_rn(cq, sum));
            } else if (EPI == EPI_SWIGLU) {
                float u = sum_of(8 + lr);
                if (p.bias) u += p.bias[p.ff + n];
                // gate and up are rounded to the storage type before the activation, as the unfused path stores them
                const float gq = to_f32(from_f32<bf16>(v)), uq = to_f32(from_f32<bf16>(u));
                ((bf16*)p.C)[o] = from_f32<bf16>(kp_gated_epilogue(p.act, gq, uq, p.glu_limit, p.glu_alpha, p.glu_shift));
            } else if (EPI == EPI_STORE) {
                ((bf16*)p.C)[o] = from_f32<bf16>(v);
            } else if (EPI == EPI_ACT) {
                ((bf16*)p.C)[o] = from_f32<bf16>(kp_act_plain(p.act, v));
            } else if (EPI == EPI_STORE_F32) {
                ((float*)p.C)[o] = v;
            } else {
                ((float*)p.C)[o] = pre_c + v;
            }
        }
    }
    KP_TRACE_MARK(2);
}

static int rw_n_sm() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

template <int WR, int EPI, int R, bool NORM, int ROOM, bool LONG>
static int rows_launch_as(const RowsArgs& a, cudaStream_t s) {
    using Shape = RowsShape<WR, R, NORM, ROOM>;
    constexpr int JOINS = EPI == EPI_CONV_STEP || EPI == EPI_CONV_ANY ? 3 : (EPI == EPI_SWIGLU ? 2 : 1);
    auto kern = gemm_rows_kernel<WR, EPI, R, NORM, ROOM, LONG>;
    static std::atomic<unsigned long long> ready{0};
    const int st = kp_smem_limit(kern, Shape::bytes(RW_NORM_MAX_K), ready, true);
    if (st) return st;
    const int n_out = JOINS > 1 ? a.ff : a.N, n_tiles = (n_out + WR / JOINS - 1) / (WR / JOINS);
    return (int)kp_launch_pdl(kern, dim3(n_tiles < rw_n_sm() ? n_tiles : rw_n_sm()), dim3(RW_WARPS * 32), Shape::bytes(a.K), s, a);
}

// (Instances of their own for what few models need: in the one kernel their code, fetched at every launch, cost a short chat of the
// 350M shape 1.2 % for more than 2048 columns, 0.25 % for other than three taps.)
template <int WR, int EPI, int R, bool NORM, int ROOM>
static int rows_launch(const RowsArgs& a, cudaStream_t s) {
    if constexpr (NORM) if (a.K > 2048) return rows_launch_as<WR, EPI, R, NORM, ROOM, true>(a, s);
    return rows_launch_as<WR, EPI, R, NORM, ROOM, false>(a, s);
}

template <int R, bool NORM, int BIG, int SMALL>
static int rows_run_r(const RowsArgs& a, int epi, cudaStream_t s) {
    // tiles of 8 rows where the busiest SM then has fewer rows of W (3072 rows: 24 against 32; 1024 rows: 8 against 16)
    const int sms = rw_n_sm();
    const auto busiest = [&](int rows) { return ((a.N + rows - 1) / rows + sms - 1) / sms * rows; };
    const bool narrow = busiest(8) < busiest(16);
#define RW_PICK(EPI, ROOM) return narrow ? rows_launch<8, EPI, R, NORM, ROOM>(a, s) : rows_launch<16, EPI, R, NORM, ROOM>(a, s)
    switch (epi) {
        case EPI_STORE: RW_PICK(EPI_STORE, BIG);
        case EPI_STORE_F32: RW_PICK(EPI_STORE_F32, BIG);
        case EPI_ACCUM_F32:
            if constexpr (!NORM) RW_PICK(EPI_ACCUM_F32, SMALL);
            return KP_ERR_BAD_ARG;
        case EPI_ACT: RW_PICK(EPI_ACT, BIG);
        case EPI_SWIGLU: return rows_launch<16, EPI_SWIGLU, R, NORM, BIG>(a, s);
        case EPI_CONV_STEP:
            return a.conv_k == 3 ? rows_launch<24, EPI_CONV_STEP, R, NORM, BIG>(a, s) : rows_launch<24, EPI_CONV_ANY, R, NORM, BIG>(a, s);
        default: return KP_ERR_BAD_ARG;
    }
#undef RW_PICK
}

// Two CTAs an SM or one (see the top).  With more than four rows A weighs as much as half of W, and two CTAs pay up to a residual of
// 1024 columns only: a step through eight layers, us, two | one, of five requests 1024 columns 177 | 186, 1536 225 | 218, 2048
// 283 | 275, 2560 427 | 416; of eight 176 | 185, 227 | 220, 287 | 277, 437 | 427.
template <bool NORM>
static int rows_run(const RowsArgs& a, int epi, cudaStream_t s) {
    if (a.M == 1) return rows_run_r<1, NORM, RW_BIG, RW_SMALL>(a, epi, s);
    if (a.M <= 4) return rows_run_r<4, NORM, RW_BIG, RW_SMALL>(a, epi, s);
    const int residual = epi == EPI_ACCUM_F32 ? a.N : a.K;
    return residual <= 1024 ? rows_run_r<8, NORM, RW_BIG, RW_SMALL>(a, epi, s) : rows_run_r<8, NORM, RW_ALONE, RW_ALONE>(a, epi, s);
}

static int rows_check(const RowsArgs& a) {
    if (a.M > 8 || a.K < 512 || (a.K % 512) || (a.lda & 7) || (a.ldw & 7) || ((uintptr_t)a.A & 15) || ((uintptr_t)a.W & 15))
        return KP_ERR_UNSUPPORTED;
    if (a.gamma && (a.K > RW_NORM_MAX_K || (a.ldx & 3) || ((uintptr_t)a.X & 15) || ((uintptr_t)a.gamma & 15))) return KP_ERR_UNSUPPORTED;
    return 0;
}

extern "C" {

// epi and glu as in gemm_stream.cu
static int rows_args(RowsArgs& a, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N, int K, int& epi,
                     float limit, float alpha, float shift) {
    a.W = (const bf16*)W; a.ldw = ldw; a.bias = bias; a.C = C; a.ldc = ldc;
    a.M = M; a.N = N; a.K = K;
    a.act = KP_EPI_ACT(epi);
    epi = KP_EPI_KIND(epi);
    if (a.act != KP_ACT_SILU && a.act != KP_ACT_RELU && a.act != KP_ACT_GELU_TANH && !(a.act == KP_ACT_GLU_CLAMPED && epi == EPI_SWIGLU) &&
        !(a.act == KP_ACT_RELU_SQ && epi == EPI_ACT)) return KP_ERR_UNSUPPORTED;
    a.glu_limit = limit; a.glu_alpha = alpha; a.glu_shift = shift;
    if (epi == EPI_CONV_STEP) return KP_ERR_BAD_ARG;
    if (epi == EPI_SWIGLU) {
        if (N & 1) return KP_ERR_BAD_ARG;
        a.ff = N / 2;
    }
    return rows_check(a);
}

int kp_gemm_rows(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N, int K,
                 int epi, float limit, float alpha, float shift, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    RowsArgs a = {};
    a.A = (const bf16*)A; a.lda = lda;
    const int st = rows_args(a, W, ldw, bias, C, ldc, M, N, K, epi, limit, alpha, shift);
    return st ? st : rows_run<false>(a, epi, (cudaStream_t)stream);
}

// The product with A = the RMS norm of the float32 rows X (weight gamma), the bits of kp_rmsnorm_rows and kp_gemm_rows: see the top.
// Not with an accumulated output.
int kp_gemm_rows_normed(const float* X, int ldx, const float* gamma, float eps, const void* W, int ldw, const float* bias, void* C,
                        int ldc, int M, int N, int K, int epi, float limit, float alpha, float shift, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    RowsArgs a = {};
    a.X = X; a.ldx = ldx; a.gamma = gamma; a.eps = eps;
    if (!gamma) return KP_ERR_BAD_ARG;
    const int st = rows_args(a, W, ldw, bias, C, ldc, M, N, K, epi, limit, alpha, shift);
    return st ? st : rows_run<true>(a, epi, (cudaStream_t)stream);
}

static int conv_step_args(RowsArgs& a, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N, int K, const float* conv_w,
                          const float* conv_bias, float* conv_state, const int* seg_pos, const int* seg_slot, int conv_k) {
    a.W = (const bf16*)W; a.ldw = ldw; a.bias = bias; a.C = C; a.ldc = ldc;
    a.M = M; a.N = N; a.K = K; a.ff = N / 3;
    if (N % 3) return KP_ERR_BAD_ARG;
    const int st = rows_check(a);
    if (st) return st;
    if (conv_k < 2 || conv_k > 16 || !conv_w || !conv_state || !seg_pos || !seg_slot) return KP_ERR_UNSUPPORTED;
    a.conv_w = conv_w; a.conv_bias = conv_bias; a.conv_state = conv_state; a.seg_pos = seg_pos; a.seg_slot = seg_slot;
    a.conv_k = conv_k;
    return 0;
}

// The in_proj of the gated short convolution with the conv step of a decode step in its epilogue: W = [B; C; X]
// ([3 d, K]), C = [M, d] bfloat16; conv_w [d][conv_k], conv_bias [d] or null, state [slots][conv_k - 1][d], and
// for each of the M <= 8 rows its position (seg_pos) and state slot (seg_slot).  Rows are one-row segments.
int kp_gemm_rows_conv_step(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N,
                           int K, const float* conv_w, const float* conv_bias, float* conv_state, const int* seg_pos,
                           const int* seg_slot, int conv_k, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    RowsArgs a = {};
    a.A = (const bf16*)A; a.lda = lda;
    const int st = conv_step_args(a, W, ldw, bias, C, ldc, M, N, K, conv_w, conv_bias, conv_state, seg_pos, seg_slot, conv_k);
    return st ? st : rows_run<false>(a, EPI_CONV_STEP, (cudaStream_t)stream);
}

// The same behind an RMS norm of the float32 rows X (see kp_gemm_rows_normed).
int kp_gemm_rows_conv_step_normed(const float* X, int ldx, const float* gamma, float eps, const void* W, int ldw, const float* bias,
                                  void* C, int ldc, int M, int N, int K, const float* conv_w, const float* conv_bias, float* conv_state,
                                  const int* seg_pos, const int* seg_slot, int conv_k, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    RowsArgs a = {};
    a.X = X; a.ldx = ldx; a.gamma = gamma; a.eps = eps;
    if (!gamma) return KP_ERR_BAD_ARG;
    const int st = conv_step_args(a, W, ldw, bias, C, ldc, M, N, K, conv_w, conv_bias, conv_state, seg_pos, seg_slot, conv_k);
    return st ? st : rows_run<true>(a, EPI_CONV_STEP, (cudaStream_t)stream);
}

}  // extern "C"
