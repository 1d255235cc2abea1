// float32 contraction of few rows (a decode step, up to 16 rows): the weights are read once, so memory bounds it (part of gemm_tc.cu's
// translation unit, whose helpers it uses).  C[m, n] (+)= sum_k A[m, k] * W[n, k] on the FMA units.
//
// The sums are those of gemv_rows_kernel (gemm_generic.cu): a warp owns weight rows, a lane sums its four of every 128 k in
// rising order, the lanes are added in a fixed tree; the order depends on N and K, not on the token rows.  What differs is how
// the operands arrive.  There a warp asks for 4 KB, waits, computes, and stops with its block every 1,024 k while the activations are
// fetched again: 2.6 TB/s on 16,384 x 2,048 at 8 rows.  Here one warp of a CTA feeds a ring in shared memory with tensor copies, a box
// of weight rows x 128 k and the activations' box beside it, always as far ahead as the ring is deep and across tile boundaries,
// and the first boxes of weights - all of them, for a small projection - before the wait on the preceding kernel.
//   tile height  the weight rows are dealt evenly: ceil(N / (CTAs * rounds)) rows a tile, at most 28, so that every SM reads the
//                same number of bytes
//   two CTAs an SM, seven warps of sums each: with one, every warp's read of the activations from shared memory stood in
//                line with its multiplications (gate/up at 8 rows 31.8 us, with two 25.5; down 27.4, with two 19.3)
// 8 rows of Llama 1B (us, against gemm_generic.cu): gate/up 25.1 (5.3 TB/s) : 49.2, down 18.7 : 25.6, head 171 to 189 (5.6 to 6.1 TB/s) : 312; 16
// rows, where the multiplications bound it: 51 : 79, 33 : 49, 370 to 394 : 510; one row: 20.7 (6.5 TB/s) : 28.3, 16.3 : 16.6, 149 (7.0 TB/s) : 162.
#pragma once

#define FST_WARPS 7                        // warps that compute; one more feeds the ring
#define FST_THREADS (32 * (FST_WARPS + 1))
#define FST_KC 128                         // k a stage: 512 bytes of a row
#define FST_MAX_STAGES 16
#define FST_RW 4                           // weight rows a warp owns at most
#define FST_RING (108 * 1024)              // bytes of shared memory: two CTAs fit an SM

// Adds 32 values over the 32 lanes, all at once: lane l gets the sum of v[l].  At every step a lane hands over the half of the
// values it will not own, so 31 shuffles do the work of 160; the pairs added are those of an xor tree over 16, 8, 4, 2, 1.
__device__ __forceinline__ float fst_sum32(float (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < o; j++) {
            const float mine = up ? v[j + o] : v[j], theirs = up ? v[j] : v[j + o];
            v[j] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
        }
    }
    return v[0];
}

template <int MB>                          // token rows (rows past M are zeros of the copy)
__global__ void __launch_bounds__(FST_THREADS, 2)
gemm_f32_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, float *__restrict__ out, int ldc,
                       int accumulate, int M, int N, int K, int tile_rows, int n_tiles, int stages, int row_groups, int k_groups) {
    constexpr int RW = FST_RW, GROUPS = (RW * MB + 31) / 32;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t bars[2 * FST_MAX_STAGES];
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int w_bytes = tile_rows * FST_KC * 4, stage_bytes = w_bytes + MB * FST_KC * 4;
    const int nk = (K + FST_KC - 1) / FST_KC;
    const int my_tiles = (n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, total = my_tiles * nk;
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[FST_MAX_STAGES]), smem0 = smem_u32(smem);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, row_groups); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();
    if (warp == FST_WARPS) {
        const uint64_t stream_once = l2_evict_first_policy();
        const int pre = min(stages, total);
        auto tile_of = [&](int it) { return ((int)blockIdx.x + it / nk * (int)gridDim.x) * tile_rows; };
        if (elect_one()) {
            for (int it = 0; it < pre; it++) {
                mbar_expect_tx(full0 + 8 * it, stage_bytes);
                tma_load_2d_hint(smem0 + it * stage_bytes, &tmW, it % nk * FST_KC, tile_of(it), full0 + 8 * it, stream_once);
            }
        }
        __syncwarp();
        pdl_wait();
        if (elect_one())
            for (int it = 0; it < pre; it++) tma_load_2d(smem0 + it * stage_bytes + w_bytes, &tmX, it % nk * FST_KC, 0, full0 + 8 * it);
        __syncwarp();
        int s = 0, ph = 1, issued = pre;
        for (int it = pre; it < total; it++) {
            if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1))) { raise_error(1); break; }
            if (elect_one()) {
                mbar_expect_tx(full0 + 8 * s, stage_bytes);
                tma_load_2d_hint(smem0 + s * stage_bytes, &tmW, it % nk * FST_KC, tile_of(it), full0 + 8 * s, stream_once);
                tma_load_2d(smem0 + s * stage_bytes + w_bytes, &tmX, it % nk * FST_KC, 0, full0 + 8 * s);
            }
            __syncwarp();
            issued++;
            if (++s == stages) { s = 0; ph ^= 1; }
        }
        for (int it = max(0, issued - stages); it < issued; it++)      // copies in flight land before the CTA exits
            mbar_wait(full0 + 8 * (it % stages), (it / stages) & 1);
        return;
    }
    // Warp (rg, kg) takes rows rg, rg + row_groups, ... of the tile and every k_groups-th box of it.  A tall tile has all warps on
    // different rows; a low one (7 rows a CTA of a 2,048-row projection) would have every warp read the activations for one
    // row, so there the warps share rows and deal out the boxes, and their sums are added in warp order.
    pdl_wait();                            // (`out` may be the residual stream)
    const int rg = warp % row_groups, kg = warp / row_groups;
    const bool busy = kg < k_groups;
    float *part = (float *)(smem + stages * stage_bytes);                  // [k_groups][row_groups][32 * GROUPS]
    int s = 0, ph = 0;
    for (int t = 0; t < my_tiles; t++) {
        const int n0 = ((int)blockIdx.x + t * (int)gridDim.x) * tile_rows;
        const int rows = min(tile_rows, N - n0), nr = (rows - rg + row_groups - 1) / row_groups;
        float acc[RW][MB];
#pragma unroll
        for (int i = 0; i < RW; i++)
#pragma unroll
            for (int m = 0; m < MB; m++) acc[i][m] = 0.f;
        int turn = 0;
        for (int kc = 0; kc < nk; kc++) {
            if (busy && turn == kg) {
                if (!__all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, ph))) { raise_error(2); break; }
                const float4 *ws = (const float4 *)(smem + s * stage_bytes) + rg * (FST_KC / 4) + lane;
                const float4 *xs = (const float4 *)(smem + s * stage_bytes + w_bytes) + lane;
                float4 x[MB];
#pragma unroll
                for (int m = 0; m < MB; m++) x[m] = xs[m * (FST_KC / 4)];
#pragma unroll
                for (int i = 0; i < RW; i++) {
                    if (i < nr) {
                        const float4 w = ws[i * row_groups * (FST_KC / 4)];
#pragma unroll
                        for (int m = 0; m < MB; m++) {
                            float v = acc[i][m];
                            v = fmaf(x[m].x, w.x, v);
                            v = fmaf(x[m].y, w.y, v);
                            v = fmaf(x[m].z, w.z, v);
                            v = fmaf(x[m].w, w.w, v);
                            acc[i][m] = v;
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty0 + 8 * s) : "memory");
            }
            if (++turn == k_groups) turn = 0;
            if (++s == stages) { s = 0; ph ^= 1; }
        }
#pragma unroll
        for (int g = 0; g < GROUPS; g++) {
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = g * 32 + j < RW * MB ? acc[(g * 32 + j) / MB < RW ? (g * 32 + j) / MB : 0][(g * 32 + j) % MB] : 0.f;
            const float sum = fst_sum32(v, lane);
            if (k_groups > 1) {
                if (busy) part[((kg * row_groups + rg) * GROUPS + g) * 32 + lane] = sum;
                continue;
            }
            const int e = g * 32 + lane, i = e / MB, m = e % MB;
            if (busy && i < nr && i < RW && m < M) {
                float *dst = out + (size_t)m * ldc + n0 + rg + i * row_groups;
                *dst = accumulate ? sum + *dst : sum;
            }
        }
        if (k_groups > 1) {
            asm volatile("bar.sync 1, %0;" ::"n"(32 * FST_WARPS) : "memory");
            for (int e = threadIdx.x; e < row_groups * GROUPS * 32; e += 32 * FST_WARPS) {
                const int r = e / (GROUPS * 32), i = e % (GROUPS * 32) / MB, m = e % (GROUPS * 32) % MB, row = r + i * row_groups;
                if (i >= RW || row >= rows || m >= M) continue;
                float sum = 0.f;
                for (int g = 0; g < k_groups; g++) sum += part[g * row_groups * GROUPS * 32 + e];      // warp order
                float *dst = out + (size_t)m * ldc + n0 + row;
                *dst = accumulate ? sum + *dst : sum;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * FST_WARPS) : "memory");
        }
    }
}

// How the weight rows and the ring are cut.  With boxes dealt out over k_groups (low tiles, one tile a CTA) the ring's depth is a
// multiple of k_groups, so that a stage always belongs to the same warps.  Otherwise a warp whose box lands early could come to a stage
// for its second filling while the first, another warp's, is still under way, and the parity it waits for would be that of
// the phase before: the wait would return at once.
struct StreamPlan { int tile_rows, n_tiles, row_groups, k_groups, stages, part_bytes; };
static StreamPlan stream_plan(int MB, int N) {
    StreamPlan p{};
    const int ctas = 2 * sm_count(), most = FST_WARPS * FST_RW, rounds = (N + ctas * most - 1) / (ctas * most);
    p.tile_rows = (N + ctas * rounds - 1) / (ctas * rounds);
    p.n_tiles = (N + p.tile_rows - 1) / p.tile_rows;
    p.row_groups = (p.tile_rows + FST_RW - 1) / FST_RW;
    p.k_groups = p.n_tiles <= ctas ? FST_WARPS / p.row_groups : 1;
    p.part_bytes = p.k_groups > 1 ? FST_WARPS * ((FST_RW * MB + 31) / 32) * 128 : 0;
    p.stages = (FST_RING - p.part_bytes) / ((p.tile_rows + MB) * FST_KC * 4);
    if (p.stages > FST_MAX_STAGES) p.stages = FST_MAX_STAGES;
    p.stages -= p.stages % p.k_groups;
    return p;
}
// for the tests: {tile_rows, n_tiles, row_groups, k_groups, stages, bytes of shared memory}
extern "C" int fg_gemm_f32_stream_plan(int M, int N, int *out) {
    const int MB = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : M <= 8 ? 8 : 16;
    const StreamPlan p = stream_plan(MB, N);
    out[0] = p.tile_rows; out[1] = p.n_tiles; out[2] = p.row_groups; out[3] = p.k_groups; out[4] = p.stages;
    out[5] = p.stages * (p.tile_rows + MB) * FST_KC * 4 + p.part_bytes;
    return 0;
}

template <int MB>
static int launch_f32_stream(const float *A, int lda, const float *W, int ldw, float *C, int ldc, int accumulate, int M, int N, int K, cudaStream_t stream) {
    const StreamPlan p = stream_plan(MB, N);
    const int ctas = 2 * sm_count(), tile_rows = p.tile_rows;
    CUtensorMap tmW, tmX;
    int e = make_map_f32(&tmW, W, N, K, ldw, tile_rows);
    if (e) return e;
    e = make_map_f32(&tmX, A, M, K, lda, MB);
    if (e) return e;
    static FgPerDevice configured;
    if (fg_needs_setup(configured)) {
        cudaError_t ce = cudaFuncSetAttribute(gemm_f32_stream_kernel<MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, FST_RING + 128);
        if (ce != cudaSuccess) return (int)ce;
    }
    return fg_launch(gemm_f32_stream_kernel<MB>, dim3(p.n_tiles < ctas ? p.n_tiles : ctas), dim3(FST_THREADS),
                     (size_t)p.stages * (tile_rows + MB) * FST_KC * 4 + p.part_bytes + 128, stream, tmW, tmX, C, ldc, accumulate, M, N, K, tile_rows,
                     p.n_tiles, p.stages, p.row_groups, p.k_groups);
}

// Up to 16 rows, everything float32.  FG_ERR_BAD_SIZE for what it does not take (gemm_generic.cu's kernels do): rows that 16-byte copies
// cannot walk, and matrices so small (N or K below 512) that a ring has nothing to run ahead for.
extern "C" int fg_gemm_f32_stream(const float *A, int lda, const float *W, int ldw, float *C, int ldc, int accumulate, int M, int N, int K,
                                  cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 16 || N < 512 || K < 512 || K % 4 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15)) return FG_ERR_BAD_SIZE;
#define FST_RUN(MB) launch_f32_stream<MB>(A, lda, W, ldw, C, ldc, accumulate, M, N, K, stream)
    if (M <= 1) return FST_RUN(1);
    if (M <= 2) return FST_RUN(2);
    if (M <= 4) return FST_RUN(4);
    if (M <= 8) return FST_RUN(8);
    return FST_RUN(16);
#undef FST_RUN
}
