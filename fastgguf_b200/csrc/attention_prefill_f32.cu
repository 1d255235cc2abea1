// Prefill attention in float32 over the paged cache, head sizes 64 and 128: every sequence of the step brings new tokens whose
// keys and values are already in the cache.  The tiled form of attention_generic.cu for steps with enough rows to share keys;
// products, sums and exponentials are the same float32 operations (fused multiply-adds, expf), no tensor cores.
//
// Reference role: attn_rows for a prompt chunk (fastgguf.c:5022-5039).
//
// The any-size kernel gives every (row, head) a block of its own, which reads all its keys again: 2,048 rows x 32 heads read
// 64 GB of keys and values a layer through L2, 5.6 ms a layer of Llama 1B (float32, 2,048 tokens) against 0.25 ms of arithmetic
// at the FMA units' rate.  Here a CTA owns 128 rows = TQ consecutive tokens x the query heads of one KV head, and walks the
// pages (64 keys) its rows may see, so a key is read once a CTA:
//   S = Q K^T       4 x 8 (head size 64) or 4 x 4 scores a thread, operands in shared memory as vectors of four
//   online softmax  a row's scores lie in 8 (16) neighbouring lanes
//   O = O c + P V   4 x 8 outputs a thread; a page's 64 products are summed from zero and then added to the scaled output, so
//                   that an output's chain of additions is 64 + pages long instead of one per key
// K and V of a page have one buffer each, filled by cp.async: K of the next page arrives under the softmax and P V, V under
// Q K^T.  Two CTAs an SM at head size 64 (101 KB of shared memory, 256 threads), one at 128 (169 KB, 512 threads).
// One layer of Llama 1B, 2,048 tokens: 5,583 -> 723 us (24 TFLOP/s).  Eight rows a thread read shared memory less often but leave
// two warps a scheduler: 772 us.
// A row's keys are visited in ascending page order, so its result does not depend on the other rows of a CTA.
//
// A CTA walks its pages alone, 10.4 us a page at head size 64 and 16 at 128, whatever it has of rows; the any-size kernel spreads the
// (row, head) pairs over the GPU, 83 ns and 165 ns for 1,000 keys of a pair.  So a sequence with few new tokens is the any-size
// kernel's, however long its past is (us, this kernel : any-size, 32 heads of 64): 1 token behind 4,000 keys 664 : 78, 16 tokens 665 :
// 204, 64 tokens 676 : 709, 128 tokens 693 : 1,398; no past, 64 tokens 20 : 22, 128 tokens 30 : 49.  24 heads of 128: 32 tokens behind 4,000
// keys 1,012 : 595, 64 tokens 1,029 : 1,075.
#include "common.cuh"

#define PAGE 64
#define ROWS 128

__device__ __forceinline__ void f32_cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void f32_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void f32_cp_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Whether the any-size kernel is the faster one for a sequence alone: its work, tokens x heads x the keys a token sees on average, against
// the keys that a tile's walk passes, by the times above.
__host__ __device__ __forceinline__ bool f32_few_rows(int tokens, int past, int heads, int hd, int window) {
    const long long keys = window ? (long long)min(past, window > 0 ? window : -window) : past;
    return (long long)tokens * heads * (2 * keys + tokens) < (hd == 64 ? 2048LL : 1536LL) * 2 * (keys + tokens);
}

template <int HD> struct PrefillF32 {
    static constexpr int RPT = 4, TX = HD / 8, THREADS = ROWS / RPT * TX, NK = PAGE / TX;       // rows a thread, lanes a row, threads, keys a thread
    static constexpr int LDQ = ROWS + 4, LDK = HD + 4;
    // Q^T [HD][LDQ], P [PAGE][LDQ], K [PAGE][LDK], V [PAGE][HD]
    static constexpr int SMEM = (HD * LDQ + PAGE * LDQ + PAGE * LDK + PAGE * HD) * 4;
};

template <int HD>
__global__ void __launch_bounds__(PrefillF32<HD>::THREADS, HD == 64 ? 2 : 1)
attn_prefill_f32_kernel(const float *__restrict__ q, int ldq, float *__restrict__ out, int ldo, const int *__restrict__ cu_rows,
                        const int *__restrict__ seq_start, const int *__restrict__ block_table, int table_width,
                        const float *__restrict__ k_pool, const float *__restrict__ v_pool, int KV, int G, float scale, int window, int skip_few) {
    using C = PrefillF32<HD>;
    constexpr int RPT = C::RPT, TX = C::TX, NT = C::THREADS, NK = C::NK, LDQ = C::LDQ, LDK = C::LDK;
    extern __shared__ __align__(16) float fsm[];
    float *Qs = fsm, *Ps = Qs + HD * LDQ, *Ks = Ps + PAGE * LDQ, *Vs = Ks + PAGE * LDK;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int Gc = G < 16 ? G : 16, TQ = ROWS / Gc, chunks = (G + Gc - 1) / Gc;
    const int kvh = blockIdx.y / chunks, g0 = (blockIdx.y % chunks) * Gc, b = blockIdx.z;
    const int row0 = cu_rows[b], n_tok = cu_rows[b + 1] - row0, start = seq_start[b];
    const int q0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * TQ;          // late tiles see the most keys: they start first
    if (q0 >= n_tok || (skip_few && f32_few_rows(n_tok, start, KV * G, HD, window))) return;
    const int tq = min(TQ, n_tok - q0);
    const int *bt = block_table + (size_t)b * table_width;
    const size_t H_row = (size_t)kvh * G + g0;                           // the first query head of this CTA

    // row r of the tile is token q0 + r / Gc and head g0 + r % Gc; a thread's rows are ty * 4 + i
    int hi[RPT], lo[RPT];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        const int r = ty * RPT + i, t = r / Gc;
        const bool valid = t < tq && g0 + r % Gc < G;
        hi[i] = valid ? start + q0 + t : -1;
        lo[i] = valid ? first_visible_key(hi[i], window) : 0;
    }
    const int tile_hi = start + q0 + tq - 1, tile_lo = first_visible_key(start + q0, window);
    const int page_begin = tile_lo / PAGE, page_end = tile_hi / PAGE + 1;
    // every row of the tile sees all keys of the pages in [whole_begin, whole_end)
    const int whole_begin = (first_visible_key(tile_hi, window) + PAGE - 1) / PAGE, whole_end = (start + q0 + 1) / PAGE;

    auto load = [&](float *dst, const float *pool, int page, int ld) {
        const float *src = pool + ((size_t)bt[page] * KV + kvh) * PAGE * HD;
#pragma unroll 4
        for (int e = tid; e < PAGE * (HD / 4); e += NT) {
            const int r = e / (HD / 4), c = e % (HD / 4) * 4;
            f32_cp_async16(dst + r * ld + c, src + (size_t)r * HD + c);
        }
    };
    load(Ks, k_pool, page_begin, LDK);
    f32_cp_commit();
    load(Vs, v_pool, page_begin, HD);
    f32_cp_commit();
    for (int e = tid; e < ROWS * (HD / 4); e += NT) {                     // Q, transposed; lanes side by side along the rows
        const int r = e % ROWS, c = e / ROWS * 4, t = r / Gc, g = g0 + r % Gc;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < tq && g < G) v = *(const float4 *)(q + (size_t)(row0 + q0 + t) * ldq + ((size_t)kvh * G + g) * HD + c);
        Qs[c * LDQ + r] = v.x; Qs[(c + 1) * LDQ + r] = v.y; Qs[(c + 2) * LDQ + r] = v.z; Qs[(c + 3) * LDQ + r] = v.w;
    }

    float acc[RPT][8], m_run[RPT], l_run[RPT];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        m_run[i] = -INFINITY; l_run[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
    }
    for (int page = page_begin; page < page_end; page++) {
        f32_cp_wait1();
        __syncthreads();                                                  // K of this page (and, the first time, Q) is here
        float s[RPT][NK];
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < NK; j++) s[i][j] = 0.f;
#pragma unroll 2
        for (int d = 0; d < HD; d += 4) {
            float4 k4[NK];
#pragma unroll
            for (int j = 0; j < NK; j++) k4[j] = *(const float4 *)(Ks + (tx + TX * j) * LDK + d);
#pragma unroll
            for (int dd = 0; dd < 4; dd++) {
                const float4 a0 = *(const float4 *)(Qs + (d + dd) * LDQ + ty * 4);
                const float a[4] = {a0.x, a0.y, a0.z, a0.w};
#pragma unroll
                for (int j = 0; j < NK; j++) {
                    const float kk = dd == 0 ? k4[j].x : dd == 1 ? k4[j].y : dd == 2 ? k4[j].z : k4[j].w;
#pragma unroll
                    for (int i = 0; i < RPT; i++) s[i][j] = fmaf(a[i], kk, s[i][j]);
                }
            }
        }
        __syncthreads();                                                  // K is free
        if (page + 1 < page_end) load(Ks, k_pool, page + 1, LDK);
        f32_cp_commit();
        const bool whole = page >= whole_begin && page < whole_end;
        const int p0 = page * PAGE + tx;                                  // this thread's keys: p0 + TX * j
        float corr[RPT];
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < NK; j++) {
                const int p = p0 + TX * j;
                const bool see = whole || (p <= hi[i] && p >= lo[i]);
                s[i][j] *= scale;
                if (see) mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = TX / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m_run[i], mx);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < NK; j++) {
                const int p = p0 + TX * j;
                const bool see = whole || (p <= hi[i] && p >= lo[i]);
                s[i][j] = see ? expf(s[i][j] - m_new) : 0.f;              // a hidden key has no weight, whatever its score is
                sum += s[i][j];
            }
#pragma unroll
            for (int o = TX / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            // a row that has seen no key yet keeps its zeros (its maximum is still -inf, and exp(-inf + inf) is no number; visible
            // scores of -inf made the sum NaN above, as they do in the any-size kernel)
            const bool none = m_new == -INFINITY && sum == 0.f;
            corr[i] = none ? 1.f : expf(m_run[i] - m_new);
            l_run[i] = l_run[i] * corr[i] + sum;
            m_run[i] = m_new;
        }
#pragma unroll
        for (int j = 0; j < NK; j++) {
            float *dst = Ps + (tx + TX * j) * LDQ + ty * 4;
            *(float4 *)dst = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
        }
        f32_cp_wait1();
        __syncthreads();                                                  // P is written, V of this page is here
        // zero times a value that is no finite number is not zero: where the page holds such a value and some row does not see
        // all of the page, hidden keys are left out one by one
        bool guarded = false;
        if (!whole) {
            bool bad = false;
            for (int e = tid; e < PAGE * HD; e += NT) bad |= !(fabsf(Vs[e]) <= 3.402823466e38f);
            guarded = __syncthreads_or(bad);
        }
        float pv[RPT][8];
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) pv[i][j] = 0.f;
        if (!guarded) {
#pragma unroll 4
            for (int k = 0; k < PAGE; k++) {
                const float4 a0 = *(const float4 *)(Ps + k * LDQ + ty * 4);
                const float4 v0 = *(const float4 *)(Vs + k * HD + tx * 4), v1 = *(const float4 *)(Vs + k * HD + tx * 4 + HD / 2);
                const float a[4] = {a0.x, a0.y, a0.z, a0.w}, v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
                for (int i = 0; i < RPT; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) pv[i][j] = fmaf(a[i], v[j], pv[i][j]);
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < PAGE; k++) {
                const int p = page * PAGE + k;
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    if (p > hi[i] || p < lo[i]) continue;
                    const float a = Ps[k * LDQ + ty * 4 + i];
#pragma unroll
                    for (int j = 0; j < 8; j++) pv[i][j] = fmaf(a, Vs[k * HD + tx * 4 + (j & 3) + (j >> 2) * (HD / 2)], pv[i][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = fmaf(acc[i][j], corr[i], pv[i][j]);
        __syncthreads();                                                  // V and P are free
        if (page + 1 < page_end) load(Vs, v_pool, page + 1, HD);
        f32_cp_commit();
    }
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        if (hi[i] < 0) continue;
        const int r = ty * 4 + i;
        float *dst = out + (size_t)(row0 + q0 + r / Gc) * ldo + (H_row + r % Gc) * HD + tx * 4;
        const float inv = l_run[i] > 0.f ? 1.0f / l_run[i] : 0.f;
        *(float4 *)dst = make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
        *(float4 *)(dst + HD / 2) = make_float4(acc[i][4] * inv, acc[i][5] * inv, acc[i][6] * inv, acc[i][7] * inv);
    }
}

template <int HD>
static int launch_prefill_f32(const float *q, int ldq, float *out, int ldo, const int *cu_rows, const int *seq_start,
                              const int *block_table, int table_width, const float *k_pool, const float *v_pool, int n_seq,
                              int max_new, int H, int KV, float scale, int window, int skip_few, cudaStream_t stream) {
    static FgPerDevice configured;
    if (fg_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(attn_prefill_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, PrefillF32<HD>::SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    const int G = H / KV, Gc = G < 16 ? G : 16, TQ = ROWS / Gc;
    dim3 grid((max_new + TQ - 1) / TQ, KV * ((G + Gc - 1) / Gc), n_seq);
    if (grid.y > 65535) return FG_ERR_BAD_SIZE;
    return fg_launch_in_order(attn_prefill_f32_kernel<HD>, grid, dim3(PrefillF32<HD>::THREADS), (size_t)PrefillF32<HD>::SMEM, stream, q, ldq,
                              out, ldo, cu_rows, seq_start, block_table, table_width, k_pool, v_pool, KV, G, scale, window, skip_few);
}

// q: [rows, ldq] float32 rows of all sequences one after another (cu_rows[b] = first row of sequence b, seq_start[b] = its length
// before the step); pools [pages, KV, 64, hd] float32; out [rows, ldo] float32.  max_new: most rows any sequence brings.
// skip_few: sequences that fg_attention_f32_few_rows names are left out (the any-size kernel has them).
// Refuses (FG_ERR_BAD_SIZE) other head sizes and pages and rows that are not 16-byte aligned; the any-size kernel takes those.
extern "C" int fg_attention_prefill_f32_ext(const void *q, int ldq, void *out, int ldo, const int *cu_rows, const int *seq_start,
                                            const int *block_table, int table_width, const void *k_pool, const void *v_pool, int n_seq,
                                            int max_new, int H, int KV, int hd, int page_size, float scale, int window, int skip_few,
                                            cudaStream_t stream) {
    if (n_seq <= 0 || max_new <= 0) return 0;
    if (page_size != PAGE || KV <= 0 || H % KV || n_seq > 65535 || ldq % 4 || ldo % 4 ||
        (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15))
        return FG_ERR_BAD_SIZE;
#define PF32_RUN(HD) launch_prefill_f32<HD>((const float *)q, ldq, (float *)out, ldo, cu_rows, seq_start, block_table, table_width, \
                                            (const float *)k_pool, (const float *)v_pool, n_seq, max_new, H, KV, scale, window, skip_few, stream)
    if (hd == 64) return PF32_RUN(64);
    if (hd == 128) return PF32_RUN(128);
#undef PF32_RUN
    return FG_ERR_BAD_SIZE;
}

extern "C" int fg_attention_prefill_f32(const void *q, int ldq, void *out, int ldo, const int *cu_rows, const int *seq_start,
                                        const int *block_table, int table_width, const void *k_pool, const void *v_pool, int n_seq,
                                        int max_new, int H, int KV, int hd, int page_size, float scale, int window, cudaStream_t stream) {
    return fg_attention_prefill_f32_ext(q, ldq, out, ldo, cu_rows, seq_start, block_table, table_width, k_pool, v_pool, n_seq, max_new, H, KV, hd,
                                        page_size, scale, window, 0, stream);
}

extern "C" int fg_attention_f32_few_rows(int tokens, int past, int heads, int hd, int window) { return f32_few_rows(tokens, past, heads, hd, window); }

// Pages of 64 keys that the longest tile of a sequence walks (*walk), and the times of both kernels in such walks: of the any-size kernel
// (*any_size) and of all the sequence's tiles on a GPU of n_sm SMs (*tiles).
extern "C" int fg_attention_f32_cost(int tokens, int past, int H, int KV, int hd, int window, int n_sm, double *any_size, double *tiles, double *walk) {
    const double keys = window ? min(past, window > 0 ? window : -window) : past, seen = keys + 0.5 * tokens;
    const int G = H / KV, Gc = G < 16 ? G : 16, TQ = ROWS / Gc;
    const double ctas = (double)((tokens + TQ - 1) / TQ) * KV * ((G + Gc - 1) / Gc);
    *walk = (keys + tokens) / PAGE + 1.0;
    *any_size = (double)tokens * H * seen / PAGE / (hd == 64 ? 2048.0 : 1536.0);
    *tiles = ctas * (seen / PAGE + 1.0) / (hd == 64 ? 2 * n_sm : n_sm);
    return 0;
}
