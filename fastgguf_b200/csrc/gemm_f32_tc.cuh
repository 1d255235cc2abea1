// float32 contraction on the tensor cores without giving up float32: C[m, n] (+)= sum_k A[m, k] * W[n, k] with float32 operands
// and results, for more rows than the weight-streaming kernel takes (part of gemm_tc.cu's translation unit, whose helpers it uses).
//
// A float32 number is the sum of three bfloat16 numbers: hi = bf16(a), mid = bf16(a - hi), lo = a - hi - mid, 8 bits of mantissa each
// and the differences exact - as long as lo is not below bfloat16's smallest number, 2^-133.  A row of an operand that would lose bits
// so, and one whose largest magnitude is not in [2^-40, 2^50), is therefore first multiplied by the power of two that brings its largest
// magnitude just below 2^50 (at most by 2^63, which carries all that float32 holds), and its sums by the inverse power at the end: a row
// whose largest magnitude is below 2^34 is carried whole, down to float32's smallest number, a row with a larger one down to 2^-183 of it.
// Such rows are rare: a flag in scratch memory says whether the operands have one, and without it no power is looked at.
// A product of two such sums is nine products of bfloat16 numbers, each exact in float32; the six largest
// (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi) are computed, the other three are below 2^-24 of the product.
//
// What is left is the order of additions.  The tensor cores' accumulator is float32, but its sums are cut off, not rounded, and over
// a long reduction the cuts all go one way.  So an accumulator in tensor memory only ever holds ONE K-block of 64: the six products in
// rising order of size, hi hi last (four instructions whose cuts count); then the epilogue warps take it out and add it, correctly rounded, to
// the sums they keep in registers.  The chain of additions of an output is K / 64 long instead of K.
//
//   f32_split_kernel        operand -> three bfloat16 planes in scratch memory
//   gemm_f32_pair_kernel    the persistent pair-of-CTAs kernel of gemm_tc.cu with six planes a stage, two accumulators that
//                           alternate from K-block to K-block, and eight warps that add them up
//   gemm_f32_finish_kernel  adds the parts of a contraction that is split along K (few output tiles), in split order
//
// Distance from float64 (2-norm, normal operands, 600 rows): 1.1e-7 at K = 2,048 and 1.5e-7 at 8,192, where the chain of fused multiply-adds
// has 8.1e-7 and 1.6e-6.  Times with the planes' making, against gemm_tile128_kernel (us): 2,048 rows x 16,384 x 2,048: 566 against
// 3,175 (243 TFLOP/s; a sixth of the bfloat16 burst rate is 270); 2,048 x 2,048 x 8,192: 314 against 1,747; 600 x 2,048 x 8,192: 144
// against 1,249; 24 x 2,048 x 2,048: 28 (the kernels alone) against 205.
//
// Two kinds of outputs are computed by the plain chain of fused multiply-adds over the float32 operands, a warp for a tile of 32 x 32:
// those that come out as no finite number (infinities and NaN among the operands), and those whose rows are so large that the plain
// chain might overflow on its way (K times the product of the rows' largest magnitudes above 2^126) - the planes, scaled, would not.
#pragma once
#include <atomic>

#define F32_EPI_WARPS 8
#define F32_THREADS (64 + 32 * F32_EPI_WARPS)
#define F32_STAGING 4096                   // per epilogue warp: a 32 x 32 float32 tile

struct F32Args {
    float *out;                            // [M, ldc], or the parts [splits][M][N]
    const float *A, *W;                    // the float32 operands, for outputs that the plain chain computes
    const int *a_shift, *w_shift;          // exponents of the powers of two that the operands' rows were multiplied by, times 2^23
    int least_shift;                       // an output whose two exponents (times 2^23) sum up to less belongs to the plain chain
    unsigned long long *flag, call;        // *flag == call: a row of this call's operands was multiplied (anything else that memory held says no)
    int M, N, K, ldc, lda, ldw;
    int splits, kb_per_split;
    int a_rows, w_rows;                    // rows between the planes of the operands
    int accumulate, vec_ok;
};

__device__ __forceinline__ bool f32_finite(float v) { return fabsf(v) <= 3.402823466e38f; }
// The bits of the power of two that brings a sum back to scale: 2^-(a_shift + w_shift), whose exponent is at most 126; a sum whose shifts are
// so small that the power is no number belongs to the plain chain (f32_too_large).
__device__ __forceinline__ uint32_t f32_back(int a_shift, int w_shift) { return 0x3f800000u - (uint32_t)a_shift - (uint32_t)w_shift; }
__device__ __forceinline__ bool f32_too_large(int a_shift, int w_shift, int least_shift) { return (a_shift >> 23) + (w_shift >> 23) < (least_shift >> 23); }
// zero where all four are finite numbers (and `sum` was), NaN where one is not
__device__ __forceinline__ float f32_check4(float4 t, float sum) { return fmaf(t.x, 0.f, fmaf(t.y, 0.f, fmaf(t.z, 0.f, fmaf(t.w, 0.f, sum)))); }

// 32 x 32 outputs by the plain chain into a warp's tile T (row r, columns swizzled as the epilogue has them).  16 k of 32 rows of both
// operands at a time lie in T, the next ones are on their way meanwhile; a lane adds up 4 x 8 outputs, each in rising k.  With
// 2,048 rows x 16,384 x 2,048 of NaN the contraction takes 5.9 ms (3.2 on the FMA-unit tiles; a lane an output 92), with one such row 2.1 (4.0).
__device__ __forceinline__ void f32_plain_tile(float *T, const F32Args &a, int m0, int n0) {
    const int lane = threadIdx.x & 31, rg = lane >> 2, cg = lane & 3;          // a lane fetches four numbers of rows rg, rg + 8, ..
    const float *pa[4], *pw[4];
    float4 fa[4], fw[4];
    float acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        pa[i] = a.A + (size_t)min(m0 + i * 8 + rg, a.M - 1) * a.lda + cg * 4;
        pw[i] = a.W + (size_t)min(n0 + i * 8 + rg, a.N - 1) * a.ldw + cg * 4;
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
    }
    auto fetch = [&](int k0) {                             // (K % 8 == 0, rows 16-byte aligned)
        const bool in = k0 + cg * 4 < a.K;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            fa[i] = in ? *(const float4 *)(pa[i] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
            fw[i] = in ? *(const float4 *)(pw[i] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    // vector q of row r: at r * 4 + (q ^ (r / 4 % 4)) for A, r / 8 for W, so that the rows read together lie in different banks
    float4 *TA = (float4 *)T, *TW = TA + 128;
    fetch(0);
    for (int k0 = 0; k0 < a.K; k0 += 16) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = i * 8 + rg;
            TA[r * 4 + (cg ^ ((r >> 2) & 3))] = fa[i];
            TW[r * 4 + (cg ^ ((r >> 3) & 3))] = fw[i];
        }
        __syncwarp();
        if (k0 + 16 < a.K) fetch(k0 + 16);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float4 x[4], y[8];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = TA[(rg * 4 + i) * 4 + (q ^ (rg & 3))];
#pragma unroll
            for (int j = 0; j < 8; j++) y[j] = TW[(cg * 8 + j) * 4 + (q ^ cg)];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    float v = acc[i][j];
                    v = fmaf(x[i].x, y[j].x, v);
                    v = fmaf(x[i].y, y[j].y, v);
                    v = fmaf(x[i].z, y[j].z, v);
                    v = fmaf(x[i].w, y[j].w, v);
                    acc[i][j] = v;
                }
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int r = rg * 4 + i, c = cg * 8 + j;
            T[r * 32 + (((c >> 2) ^ (r & 7)) << 2) + (c & 3)] = acc[i][j];
        }
    __syncwarp();
}

// planes[p][row][k], p = 0 (hi), 1 (mid), 2 (lo) of x[row][k] * 2^shift[row].  Bound by memory: 4 bytes in, 6 out.  A row is a block's, KEEP
// times eight numbers a thread, which stay in registers between the row's largest and smallest magnitudes and the planes (beyond 32,768
// numbers the rest of a row comes from the caches again).  16,384 rows of 2,048 49.5 us (6.8 TB/s; 57 us when threads walked all rows in steps), 2,048 rows of 8,192 25 us,
// 300 rows of 28,672 20 us.
template <int KEEP>
__global__ void __launch_bounds__(KEEP == 2 ? 256 : 512)
f32_split_kernel(const float *__restrict__ x, int ld, bf16 *__restrict__ planes, int *__restrict__ shift, unsigned long long *flag,
                 unsigned long long call, int rows, int K) {
    __shared__ float scratch[32];
    const int n8 = K / 8, r = blockIdx.x;
    const size_t plane = (size_t)rows * K;
    const float *src = x + (size_t)r * ld;
    float v[KEEP][8], largest = 0.f;
    uint32_t smallest = 0xffffffffu;                       // twice the bits of the smallest number that is not a bfloat16 number, less one
    auto fetch = [&](float (&u)[8], int i) {
        const float4 lo = *(const float4 *)(src + i * 8), hi = *(const float4 *)(src + i * 8 + 4);
        u[0] = lo.x; u[1] = lo.y; u[2] = lo.z; u[3] = lo.w; u[4] = hi.x; u[5] = hi.y; u[6] = hi.z; u[7] = hi.w;
    };
    auto look = [&](const float (&u)[8]) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            largest = fmaxf(largest, fabsf(u[j]));         // (a NaN leaves it as it is)
            const uint32_t bits = __float_as_uint(u[j]);
            if (bits & 0xffffu) smallest = min(smallest, (bits << 1) - 1u);
        }
    };
#pragma unroll
    for (int q = 0; q < KEEP; q++) {
        const int i = threadIdx.x + q * blockDim.x;
        if (i < n8) fetch(v[q], i);
        else
#pragma unroll
            for (int j = 0; j < 8; j++) v[q][j] = 0.f;
    }
#pragma unroll
    for (int q = 0; q < KEEP; q++) look(v[q]);
    for (int i = threadIdx.x + KEEP * blockDim.x; i < n8; i += blockDim.x) {
        float u[8];
        fetch(u, i);
        look(u);
    }
    const bool tiny = __syncthreads_or(smallest < (17u << 24) - 1u);           // below 2^(17 - 127): bits below 2^-133
    largest = block_max(largest, scratch);
    // the exponent field f says |x| < 2^(f - 126); infinities as the largest finite numbers
    const int field = min(__float_as_int(largest) >> 23, 254), sh = tiny || field > 176 || (field < 87 && largest > 0.f) ? min(176 - field, 63) : 0;
    const float factor = __int_as_float((sh + 127) << 23);
    if (threadIdx.x == 0) {
        shift[r] = sh << 23;
        if (sh) *flag = call;                              // (every writer writes the same)
    }
    if (r == rows - 1)                                     // (tiles read the shifts of all their rows)
        for (int q = rows + threadIdx.x; q < (rows + 255) / 256 * 256; q += blockDim.x) shift[q] = 0;
    auto write = [&](const float (&u)[8], int i) {
        uint32_t w[3][4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float a = u[2 * j] * factor, b = u[2 * j + 1] * factor;
#pragma unroll
            for (int p = 0; p < 3; p++) {
                const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
                w[p][j] = *(const uint32_t *)&t;
                a -= __low2float(t);
                b -= __high2float(t);
            }
        }
#pragma unroll
        for (int p = 0; p < 3; p++) *(uint4 *)(planes + p * plane + (size_t)r * K + i * 8) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
    };
#pragma unroll
    for (int q = 0; q < KEEP; q++) {
        const int i = threadIdx.x + q * blockDim.x;
        if (i < n8) write(v[q], i);
    }
    for (int i = threadIdx.x + KEEP * blockDim.x; i < n8; i += blockDim.x) {
        float u[8];
        fetch(u, i);
        write(u, i);
    }
}

// Stages: three 16 KB planes of token rows and three of half the weight rows: 96 KB at 256 columns, 72 KB at 128; two fit
// beside the staging tiles.  A K-block is 24 instructions of 256 x BN x 16: 3,072 cycles at 256 columns, for 96 KB of operands - less than half
// of what the bfloat16 kernel asks of the L2-to-SM path.
template <int BN>
__global__ void __launch_bounds__(F32_THREADS, 1)
gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmQ, F32Args a, int n_pt, int n_tiles) {
    constexpr int STAGES = 2;
    constexpr int P_BYTES = BM * BK * 2, Q_BYTES = (BN / 2) * BK * 2;      // one plane of this CTA's share
    constexpr int STAGE_BYTES = 3 * (P_BYTES + Q_BYTES);
    constexpr int TMEM_COLS = 2 * BN;
    constexpr int NC = BN / 2;                                             // columns an epilogue warp adds up

    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * STAGES + 4];
    __shared__ uint32_t tmem_base_s;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int rank = (int)(blockIdx.x & 1);            // 0: the pair's leader (issues the MMAs), 1: its peer
    const int pair = (int)(blockIdx.x >> 1), n_pairs = (int)(gridDim.x >> 1);
    const int nkb = (a.K + BK - 1) / BK;
    const int per_split = n_tiles / a.splits;          // the tile index counts the split, slowest
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[STAGES]);
    const uint32_t tfull0 = smem_u32(&bars[2 * STAGES]), tempty0 = smem_u32(&bars[2 * STAGES + 2]);
    const uint32_t smem0 = smem_u32(smem);
    const uint32_t lead_full0 = mapa_u32(full0, 0), lead_tempty0 = mapa_u32(tempty0, 0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int i = 0; i < 2; i++) { mbar_init(tfull0 + 8 * i, 1); mbar_init(tempty0 + 8 * i, 2 * F32_EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                    // the partner's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (both CTAs)
        int s = 0, ph = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int t2 = tile % per_split, kb0 = tile / per_split * a.kb_per_split, kb1 = min(nkb, kb0 + a.kb_per_split);
            const int p0 = (t2 % n_pt) * (2 * BM) + rank * BM, q0 = (t2 / n_pt) * BN + rank * (BN / 2);
            for (int kb = kb0; kb < kb1; kb++) {
                ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1));
                if (!ok) { raise_error(1); break; }
                if (elect_one()) {
                    const uint32_t dst = smem0 + s * STAGE_BYTES, bar = lead_full0 + 8 * s;
                    if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * STAGE_BYTES);     // both CTAs' copies of the stage
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        // (a box that runs past its plane reads the next plane's rows: outputs of rows past M and N are not stored)
                        tma_load_2d_pair(dst + p * P_BYTES, &tmP, kb * BK, p * a.a_rows + p0, bar);
                        tma_load_2d_pair(dst + 3 * P_BYTES + p * Q_BYTES, &tmQ, kb * BK, p * a.w_rows + q0, bar);
                    }
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (the leader only)
        if (rank == 0) {
            const uint32_t idesc = make_idesc(2 * BM, BN);
            const uint64_t pdesc0 = make_smem_desc(smem0), qdesc0 = make_smem_desc(smem0 + 3 * P_BYTES);
            int s = 0, ph = 0, i = 0;                  // i: K-blocks so far, over all tiles
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                const int kb0 = tile / per_split * a.kb_per_split, kb1 = min(nkb, kb0 + a.kb_per_split);
                for (int kb = kb0; kb < kb1; kb++, i++) {
                    const int acc = i & 1;
                    ok = __all_sync(0xffffffffu, mbar_wait(tempty0 + 8 * acc, ((i >> 1) & 1) ^ 1));
                    if (!ok) { raise_error(4); break; }
                    ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, ph));
                    if (!ok) { raise_error(2); break; }
                    tc_fence_after();
                    const uint64_t soff = (uint64_t)(s * (STAGE_BYTES >> 4));
                    const uint64_t pdesc = pdesc0 + soff, qdesc = qdesc0 + soff;
                    if (elect_one()) {
                        // planes of the two factors, the smallest products first
                        constexpr int PA[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
                        for (int pr = 0; pr < 6; pr++)
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; k++) {
                                const uint64_t koff = (uint64_t)((k * UMMA_K * 2) >> 4);
                                tc_mma_bf16_pair(tmem_base + acc * BN, pdesc + (uint64_t)((PA[pr] * P_BYTES) >> 4) + koff,
                                                 qdesc + (uint64_t)((PB[pr] * Q_BYTES) >> 4) + koff, idesc, (pr | k) != 0);
                            }
                        tc_commit_pair(empty0 + 8 * s);              // frees the stage in both CTAs
                        tc_commit_pair(tfull0 + 8 * acc);            // the K-block's sums are complete
                    }
                    __syncwarp();
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
    } else {
        // ------------------------------------------------------------ sums and epilogue (warps 2.., both CTAs): this CTA's 128 rows
        const int lg = warp & 3, half = (warp - 2) >> 2;
        float *T = (float *)(smem + STAGES * STAGE_BYTES) + (warp - 2) * (F32_STAGING / 4);
        const bool scaled = *a.flag == a.call;
        int i = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int t2 = tile % per_split, z = tile / per_split, kb0 = z * a.kb_per_split, kb1 = min(nkb, kb0 + a.kb_per_split);
            const int m_base = (t2 % n_pt) * (2 * BM) + rank * BM + lg * 32, n_base = (t2 / n_pt) * BN + half * NC;
            float sum[NC];
#pragma unroll
            for (int j = 0; j < NC; j++) sum[j] = 0.f;
            for (int kb = kb0; kb < kb1; kb++, i++) {
                const int acc = i & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, (i >> 1) & 1));
                if (!ok) { raise_error(3); break; }
                tc_fence_after();
                const uint32_t trow = tmem_base + ((uint32_t)(lg * 32) << 16) + acc * BN + half * NC;
#pragma unroll
                for (int c = 0; c < NC / 16; c++) {                // 16 at a time: 128 sums and the kernel's 168 registers a thread
                    float v[16];
                    tc_ld16(trow + c * 16, v);
#pragma unroll
                    for (int j = 0; j < 16; j++) sum[c * 16 + j] += v[j];
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(lead_tempty0 + 8 * acc);
            }
            if (!ok) break;
            // 32 columns at a time through a tile in shared memory, so that a warp stores whole 128-byte lines; parts stay scaled
            const bool part = a.splits > 1;
            float *out = part ? a.out + (size_t)z * a.M * a.N : a.out;
            const int ldc = part ? a.N : a.ldc, ch = lane & 7;
            uint32_t plain[NC / 32], any_plain = 0;                // outputs of this lane's row that the plain chain has to give
#pragma unroll
            for (int c = 0; c < NC / 32; c++) {
                plain[c] = 0;
                float check = 0.f;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float4 t = make_float4(sum[c * 32 + 4 * q], sum[c * 32 + 4 * q + 1], sum[c * 32 + 4 * q + 2], sum[c * 32 + 4 * q + 3]);
                    check = f32_check4(t, check);
                    *(float4 *)(T + lane * 32 + ((q ^ (lane & 7)) << 2)) = t;
                }
                const bool some = !part && (scaled || __any_sync(0xffffffffu, check != 0.f));
                if (some && m_base + lane < a.M) {
                    const int row_shift = scaled ? a.a_shift[m_base + lane] : 0;
#pragma unroll 1
                    for (int j = 0; j < 32 && n_base + c * 32 + j < a.N; j++) {
                        float &v = T[lane * 32 + (((j >> 2) ^ (lane & 7)) << 2) + (j & 3)];
                        const int col_shift = scaled ? a.w_shift[n_base + c * 32 + j] : 0;
                        if (!f32_finite(v) || f32_too_large(row_shift, col_shift, a.least_shift)) plain[c] |= 1u << j;
                        v *= __uint_as_float(f32_back(row_shift, col_shift));
                    }
                }
                any_plain |= some;
                __syncwarp();
                const int n = n_base + c * 32 + ch * 4;
#pragma unroll 2
                for (int pass = 0; pass < 8; pass++) {
                    const int row = pass * 4 + (lane >> 3), m = m_base + row;
                    const uint32_t later = some ? (__shfl_sync(0xffffffffu, plain[c], row) >> (4 * ch)) & 15 : 0;
                    if (m >= a.M || n >= a.N) continue;
                    float4 t = *(const float4 *)(T + row * 32 + ((ch ^ (row & 7)) << 2));
                    float *dst = out + (size_t)m * ldc + n;
                    if (a.vec_ok && n + 3 < a.N && !later) {
                        if (a.accumulate && !part) {
                            const float4 r = __ldcg((const float4 *)dst);
                            t.x += r.x; t.y += r.y; t.z += r.z; t.w += r.w;
                        }
                        *(float4 *)dst = t;
                    } else {
                        const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (n + j < a.N && !(later >> j & 1)) dst[j] = tv[j] + (a.accumulate && !part ? dst[j] : 0.f);
                    }
                }
                __syncwarp();
            }
            if (!any_plain) continue;
#pragma unroll 1
            for (int c = 0; c < NC / 32; c++) {                    // (here, where the sums are no longer needed, it costs the kernel no registers)
                uint32_t bits = plain[0];
#pragma unroll
                for (int i = 1; i < NC / 32; i++) bits = c == i ? plain[i] : bits;
                if (!__any_sync(0xffffffffu, bits != 0)) continue;
                f32_plain_tile(T, a, m_base, n_base + c * 32);
                const int n = n_base + c * 32 + ch * 4;
                for (int pass = 0; pass < 8; pass++) {
                    const int row = pass * 4 + (lane >> 3), m = m_base + row;
                    const uint32_t mine = (__shfl_sync(0xffffffffu, bits, row) >> (4 * ch)) & 15;
                    for (int j = 0; j < 4; j++)
                        if ((mine >> j & 1) && m < a.M && n + j < a.N) {
                            float *dst = out + (size_t)m * ldc + n + j;
                            *dst = T[row * 32 + ((ch ^ (row & 7)) << 2) + j] + (a.accumulate ? *dst : 0.f);
                        }
                }
                __syncwarp();
            }
        }
    }
    // see gemm_tc_prefill_pair_kernel: neither CTA leaves while the other may still touch its memory or its barriers
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// out[m, n] (+)= the sum of the parts [splits][M][N], in split order.  A block takes 32 x 32 outputs, a thread four columns of a row
// (N % 4 == 0 where splits are taken).
__global__ void __launch_bounds__(256, 4)
gemm_f32_finish_kernel(F32Args a, const float *__restrict__ parts) {
    __shared__ float4 TA[32 * 4], TW[32 * 4];
    const int row = threadIdx.x >> 3, ch = threadIdx.x & 7, m0 = blockIdx.y * 32, n0 = blockIdx.x * 32, m = m0 + row, n = n0 + ch * 4;
    const bool in = m < a.M && n < a.N;
    float *dst = a.out + (size_t)m * a.ldc + n;
    float res[4] = {0.f, 0.f, 0.f, 0.f};
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t plain = 0;
    if (in) {
        if (a.accumulate) {
#pragma unroll
            for (int j = 0; j < 4; j++) res[j] = dst[j];
        }
        const float *p = parts + (size_t)m * a.N + n;
#pragma unroll 4
        for (int z = 0; z < a.splits; z++) {
            const float4 v = __ldcs((const float4 *)(p + (size_t)z * a.M * a.N));
            t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
        }
        const bool scaled = *a.flag == a.call;
        const int sa = scaled ? a.a_shift[m] : 0;
        const int4 w = scaled ? *(const int4 *)(a.w_shift + n) : make_int4(0, 0, 0, 0);
        auto back = [&](float &v, int sw, uint32_t bit) {
            if (!f32_finite(v) || f32_too_large(sa, sw, a.least_shift)) plain |= bit;
            v *= __uint_as_float(f32_back(sa, sw));
        };
        back(t.x, w.x, 1); back(t.y, w.y, 2); back(t.z, w.z, 4); back(t.w, w.w, 8);
    }
    if (__syncthreads_or(plain != 0)) {                     // the plain chain, every thread its own four
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const bool w_side = threadIdx.x >= 128;
        const int fr = (threadIdx.x & 127) >> 2, fq = threadIdx.x & 3;
        const float *src = (w_side ? a.W + (size_t)min(n0 + fr, a.N - 1) * a.ldw : a.A + (size_t)min(m0 + fr, a.M - 1) * a.lda) + fq * 4;
        float4 *into = (w_side ? TW : TA) + fr * 4 + (fq ^ ((fr >> (w_side ? 2 : 0)) & 3));
        for (int k0 = 0; k0 < a.K; k0 += 16) {
            const float4 v = k0 + fq * 4 < a.K ? *(const float4 *)(src + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
            __syncthreads();
            *into = v;
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float4 x = TA[row * 4 + (q ^ (row & 3))];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 y = TW[(ch * 4 + j) * 4 + (q ^ (ch & 3))];
                    acc[j] = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, acc[j]))));
                }
            }
        }
        t = make_float4(plain & 1 ? acc[0] : t.x, plain & 2 ? acc[1] : t.y, plain & 4 ? acc[2] : t.z, plain & 8 ? acc[3] : t.w);
    }
    if (!in) return;
    dst[0] = t.x + res[0]; dst[1] = t.y + res[1]; dst[2] = t.z + res[2]; dst[3] = t.w + res[3];
}

// ---------------------------------------------------------------------------- host side
// Bytes of planes of one operand at a time: scratch memory stays bounded.  Half of it, a quarter or an eighth do where memory is short:
// the sums are the same, an operand's rows go through in more portions.
#define F32_PLANE_LIMIT ((size_t)256 << 20)
#define F32_LEAST_LIMIT (F32_PLANE_LIMIT / 8)

struct F32Plan { int M, N, K, bn, splits, kb_per_split, a_rows, w_rows; size_t a_bytes, w_bytes, part_bytes, shift_bytes, bytes; };

// The rows of the operands whose planes are made at a time, where `limit` bytes of planes of an operand are allowed.
static int f32_rows_at_a_time(int rows, int K, size_t limit) {
    const size_t most = limit / ((size_t)K * 6) / 256 * 256;
    return (size_t)rows <= most ? rows : (int)(most < 256 ? 256 : most);
}
static void f32_portions(F32Plan &p, size_t limit) {
    auto up = [](size_t b) { return (b + 1023) / 1024 * 1024; };
    p.a_rows = f32_rows_at_a_time(p.M, p.K, limit); p.w_rows = f32_rows_at_a_time(p.N, p.K, limit);
    p.a_bytes = up((size_t)p.a_rows * p.K * 6); p.w_bytes = up((size_t)p.w_rows * p.K * 6);
    p.part_bytes = p.splits > 1 ? up((size_t)p.splits * p.a_rows * p.w_rows * 4) : 0;
    p.shift_bytes = up((size_t)p.a_rows * 4) + up((size_t)p.w_rows * 4) + 1024;
    p.bytes = p.a_bytes + p.w_bytes + p.part_bytes + p.shift_bytes;
}

// How the contraction is cut: tile width and splits along K.  The times are those of a K-block (microseconds), of the start and end of a
// tile, and of the pass that adds the parts.  Both are chosen for the full limit, so that a smaller one changes no order of additions.
static F32Plan f32_plan(int M, int N, int K) {
    F32Plan best{};
    best.M = M; best.N = N; best.K = K;
    const int nkb = (K + BK - 1) / BK, pairs = sm_count() / 2;
    const int am = f32_rows_at_a_time(M, K, F32_PLANE_LIMIT), wn = f32_rows_at_a_time(N, K, F32_PLANE_LIMIT);
    double best_us = 1e30;
    for (int bn = 128; bn <= 256; bn += 128)
        for (int s = 1; s <= 16; s++) {
            const int per = (nkb + s - 1) / s;
            if (s > 1 && (per < 4 || (s - 1) * per >= nkb || N % 4)) continue;
            const long long tiles = (long long)((am + 255) / 256) * ((wn + bn - 1) / bn) * s;
            const double rounds = (double)((tiles + pairs - 1) / pairs);
            const double us = rounds * (per * (bn == 256 ? 1.75 : 0.95) + 4.0) + (s > 1 ? 4.0 + (s + 2.0) * am * wn * 4.0 / 4e6 : 0.0);
            if (us < best_us) { best_us = us; best.bn = bn; best.splits = s; best.kb_per_split = per; }
        }
    f32_portions(best, F32_PLANE_LIMIT);
    return best;
}

// Scratch memory fg_gemm_f32_tc takes at most, and the least it needs; 0: sizes it does not take.  Rows up to 16 belong to the weight-streaming kernel.  Short
// reductions and narrow outputs (K < 512, N < 256) stay with the plain kernels: one or two rounds of their tiles take about
// what the three launches here do; so do small matrices (a megabyte) at up to 64 rows, which the weight-streaming kernel takes.  From 17 rows on the planes won at every size measured (K 2,048 and 8,192, N 2,048 to 16,384, 24 to
// 2,048 rows: 2.7 to 13 times).
static bool f32_takes(int M, int N, int K) {
    return !(M <= 16 || N < 256 || K < 512 || K % 8 || (M <= 64 && (long long)N * K <= 1 << 18));
}
extern "C" long long fg_gemm_f32_tc_workspace_bytes(int M, int N, int K) { return f32_takes(M, N, K) ? (long long)f32_plan(M, N, K).bytes : 0; }
extern "C" long long fg_gemm_f32_tc_least_bytes(int M, int N, int K) {
    if (!f32_takes(M, N, K)) return 0;
    F32Plan p = f32_plan(M, N, K);
    f32_portions(p, F32_LEAST_LIMIT);
    return (long long)p.bytes;
}

template <int BN>
static int launch_f32_pair(const CUtensorMap &tmP, const CUtensorMap &tmQ, const F32Args &a, cudaStream_t stream) {
    constexpr int smem = 2 * 3 * (BM + BN / 2) * BK * 2 + 1024 + F32_EPI_WARPS * F32_STAGING;
    static FgPerDevice configured;
    if (fg_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_pair_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
    }
    const int n_pt = (a.M + 2 * BM - 1) / (2 * BM), n_tiles = n_pt * ((a.N + BN - 1) / BN) * a.splits, pairs = sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (n_tiles < pairs ? n_tiles : pairs), 1, 1); cfg.blockDim = dim3(F32_THREADS);
    cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, gemm_f32_pair_kernel<BN>, tmP, tmQ, a, n_pt, n_tiles);
}

static int launch_f32_split(const float *x, int ld, bf16 *planes, int *shift, unsigned long long *flag, unsigned long long call, int rows, int K,
                            cudaStream_t stream) {
    if (K <= 4096)
        return fg_launch_in_order(f32_split_kernel<2>, dim3(rows), dim3((K / 16 + 31) / 32 * 32), 0, stream, x, ld, planes, shift, flag, call, rows, K);
    const int threads = K >= 32768 ? 512 : (K / 64 + 31) / 32 * 32;
    return fg_launch_in_order(f32_split_kernel<8>, dim3(rows), dim3(threads), 0, stream, x, ld, planes, shift, flag, call, rows, K);
}

// C[m, n] (+)= sum_k A[m, k] W[n, k], everything float32.  Needs 256-byte aligned scratch memory, from
// fg_gemm_f32_tc_least_bytes to fg_gemm_f32_tc_workspace_bytes of it; FG_ERR_BAD_SIZE for what it does not take (the plain kernels do).  Kernels are launched in plain stream order.
extern "C" int fg_gemm_f32_tc(const float *A, int lda, const float *W, int ldw, float *C, int ldc, int accumulate, int M, int N, int K,
                              void *ws, long long ws_bytes, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!f32_takes(M, N, K) || ws == nullptr || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15) || ((uintptr_t)ws & 255))
        return FG_ERR_BAD_SIZE;
    F32Plan p = f32_plan(M, N, K);
    for (size_t limit = F32_PLANE_LIMIT / 2; (long long)p.bytes > ws_bytes && limit >= F32_LEAST_LIMIT; limit /= 2) f32_portions(p, limit);
    if ((long long)p.bytes > ws_bytes) return FG_ERR_BAD_SIZE;
    bf16 *ap = (bf16 *)ws, *wp = (bf16 *)((char *)ws + p.a_bytes);
    float *parts = (float *)((char *)ws + p.a_bytes + p.w_bytes);
    int *a_shift = (int *)((char *)ws + p.a_bytes + p.w_bytes + p.part_bytes), *w_shift = a_shift + ((size_t)p.a_rows * 4 + 1023) / 1024 * 256;
    unsigned long long *flag = (unsigned long long *)(w_shift + ((size_t)p.w_rows * 4 + 1023) / 1024 * 256);
    static std::atomic<unsigned long long> calls{0x5eed0000f32a11ull};
    const unsigned long long call = calls.fetch_add(1);    // (a recorded call keeps its number: its flag may stay up, which costs time, no bits)
    // |a| < 2^(50 - shift): K products of less than 2^(100 - a_shift - w_shift) stay below 2^126
    int least_shift = -26;
    while ((1LL << (least_shift + 26)) < K) least_shift++;
    least_shift *= 1 << 23;
    for (int m0 = 0; m0 < M; m0 += p.a_rows) {
        const int mr = M - m0 < p.a_rows ? M - m0 : p.a_rows;
        int e = launch_f32_split(A + (size_t)m0 * lda, lda, ap, a_shift, flag, call, mr, K, stream);
        if (e) return e;
        for (int n0 = 0; n0 < N; n0 += p.w_rows) {
            const int nr = N - n0 < p.w_rows ? N - n0 : p.w_rows;
            if (n0 > 0 || m0 == 0 || p.w_rows < N) {                        // (the planes of W are kept where all of them fit)
                e = launch_f32_split(W + (size_t)n0 * ldw, ldw, wp, w_shift, flag, call, nr, K, stream);
                if (e) return e;
            }
            CUtensorMap tmP, tmQ;
            e = make_map(&tmP, ap, 3 * mr, K, K, BM);
            if (e) return e;
            e = make_map(&tmQ, wp, 3 * nr, K, K, p.bn / 2);
            if (e) return e;
            float *out = C + (size_t)m0 * ldc + n0;
            const bool split = p.splits > 1;
            F32Args a{split ? parts : out, A + (size_t)m0 * lda, W + (size_t)n0 * ldw, a_shift, w_shift, least_shift, flag, call, mr, nr, K, ldc, lda, ldw, p.splits, p.kb_per_split, mr, nr,
                      accumulate, split ? nr % 4 == 0 : ((uintptr_t)out % 16 == 0 && ldc % 4 == 0)};
            e = p.bn == 256 ? launch_f32_pair<256>(tmP, tmQ, a, stream) : launch_f32_pair<128>(tmP, tmQ, a, stream);
            if (e) return e;
            if (split) {
                a.out = out;
                e = fg_launch_in_order(gemm_f32_finish_kernel, dim3((nr + 31) / 32, (mr + 31) / 32), dim3(256), 0, stream, a, (const float *)parts);
                if (e) return e;
            }
        }
    }
    return 0;
}
