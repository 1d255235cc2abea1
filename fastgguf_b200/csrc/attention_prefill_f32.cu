// Prefill attention in float32 over the paged cache on the tensor cores (tcgen05), head sizes 64 and 128: every sequence of the
// step brings new tokens whose keys and values are already in the cache.  The tiled form of attention_generic.cu for steps with
// enough rows to share keys.
//
// Reference role: attn_rows for a prompt chunk (fastgguf.c:5022-5039).
//
// A float32 number is the sum of three bfloat16 numbers (hi, mid, lo: eight bits of mantissa each, the differences exact).  A product of two
// such sums is nine products of bfloat16 numbers, each exact in float32; the six largest are computed, the other three are below
// 2^-24 of the product.  The accumulator in tensor memory is float32 but cuts its sums instead of rounding them, so it only ever holds
// sums of 64 terms (a page's scores over 64 dimensions, a page's 64 weighted values), the small products first; the sums over dimensions
// and pages are added, correctly rounded, in registers.  Softmax statistics and exponentials (expf) are float32 as before.
//
// Grid (query tile x kv head x head chunk, sequence), the tiles with the most keys first.  A CTA owns 128 rows = TQ consecutive
// tokens x Gc query heads of one KV head and walks the pages (64 keys) that its rows may see.
// A row's 64 scores of a page lie in two threads (warps w and w + 4), 32 keys and half of the output's columns each.  The same eight warps
// split the float32 pages into planes in shared memory (a page is read once a CTA: K of page j + 1 while the scores of page j wait in
// registers, V of page j after its maximum is known), and the probabilities into planes in tensor memory.  Whichever warp is the last to
// have its part ready issues S = Q K^T (planes of both in shared memory) or P V (P from tensor memory, V the MN-major operand); no warp is
// kept for that, which leaves 128 registers a thread.  S of page j + 1 runs under the softmax of page j, P V of page j under the
// start of page j + 1.
// Two CTAs an SM at head size 64 (100 KB of shared memory, 256 columns of tensor memory), one at 128 (193 KB, 512).
//
// What bounds it: some 44 instructions of the ordinary units a score (expf, the splits of P, K and V; ncu: an instruction issued in 61 % of the
// cycles, four warps a scheduler), beside 48 MMAs of 128 x 64 x 16 a page (46 cycles each and not 32, the floor of one so narrow: 30 % of the time).
// One layer of Llama 1B, 2,048 tokens: 709 us on the FMA units (four scores a thread from shared memory), 169 here (102 TFLOP/s); 8,192
// tokens 7,649 -> 2,088; 24 heads of 128, 2,048 tokens 1,004 -> 269; 64 tokens 31 -> 23.  Distance from float64 (2-norm, 2,048
// tokens): 1.7e-7 (FMA tiles 2.7e-7), with scores three times as large 3.4e-7 (7.5e-7); heads of 128 and twice as large 3.5e-7 (8.2e-7).
//
// The planes carry all of a float32 number as long as no bits lie below 2^-133 and nothing overflows on the way.  Queries and keys of 2^50
// and more, values of 2^60 and more or (not zero and) below 2^-100, infinities and NaN are therefore left to the plain chain of fused
// multiply-adds: a CTA that meets one (at a position that some row of its tile sees) walks its pages again on the FMA units (f32_plain_walk) for
// the rows that see it.
// Scores need no more than an absolute error, so small queries and keys need no such care, and probabilities are multiplied by
// 2^30, which the division by their sum takes back.
// A row's keys are visited in ascending page order, so its result does not depend on the other rows of a CTA.
//
// A CTA walks its pages alone, 3.45 us a page at head size 64 and 5.0 at 128, whatever it has of rows; the any-size kernel spreads the
// (row, head) pairs over the GPU, 83 ns and 165 ns for 1,000 keys of a pair.  So a sequence with few new tokens is the any-size
// kernel's, however long its past is (us, launches behind one another, this kernel : any-size, 32 heads of 64): 2 tokens behind 2,000 keys 117 : 40,
// 8 behind 500 33 : 24, 64 behind 4,000 230 : 702; no past, 17 tokens 9.3 : 6.3, 33 tokens 10.1 : 11.2, 64 tokens 10.1 : 20.6, 512 tokens 35 : 418.  24
// heads of 128: 17 tokens 11.8 : 9.4, 33 tokens 13.4 : 14.7, 64 behind 4,000 keys 320 : 1,073.
#include "common.cuh"
#include <atomic>

#define PAGE 64
#define ROWS 128
#define F32_THREADS 256                        // threads of a CTA
#define FG_ERR_PIPELINE 10003
#define WAIT_LIMIT_CYCLES 2000000000ll
#define WAIT_SHORT_CYCLES 1000000ll

__device__ int g_f32_attn_error = 0;
// how long a wait may last, in SM cycles; a variable so that a test can shorten it (fg_attention_prefill_f32_test_hook)
__device__ long long g_f32_attn_wait_limit = WAIT_LIMIT_CYCLES;
static int g_f32_test_skip = 0;
static std::atomic<bool> g_f32_attn_launched{false};

extern "C" int fg_attention_prefill_f32_test_hook(long long wait_limit_cycles, int skip_scores) {
    long long v = wait_limit_cycles > 0 ? wait_limit_cycles : WAIT_LIMIT_CYCLES;
    g_f32_test_skip = skip_scores ? 1 : 0;
    return (int)cudaMemcpyToSymbol(g_f32_attn_wait_limit, &v, sizeof v);
}

// 0, or the code of the first bounded wait that ran out (clears it).  Nothing is read from the device before the first launch.
extern "C" int fg_attention_prefill_f32_error(void) {
    if (!g_f32_attn_launched.load(std::memory_order_relaxed)) return 0;
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_f32_attn_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_f32_attn_error, &zero, sizeof(int));
    return v;
}

struct F32Attn {
    const float *q; int ldq;
    float *out; int ldo;
    const int *cu_rows, *seq_start, *block_table; int table_width;
    const float *k_pool, *v_pool;
    int KV, G;
    float scale;
    int window;
};

// Whether the any-size kernel is the faster one for a sequence alone: its work, tokens x heads x the keys a token sees on average, against
// the keys that a tile's walk passes.  pairs: (row, head) pairs whose page the any-size kernel takes in the time of a tile's walk of a page.
__host__ __device__ __forceinline__ bool f32_few_rows(int tokens, int past, int heads, int window, int pairs) {
    const long long keys = window ? (long long)min(past, window > 0 ? window : -window) : past;
    return (long long)tokens * heads * (2 * keys + tokens) < (long long)pairs * 2 * (keys + tokens);
}
// 5.3 ns (10.6 at head size 128) a pair's page against 3.45 us (5.0) a tile's
static int f32_pairs(int hd) { return hd == 64 ? 650 : 470; }

// ------------------------------------------------------------------------------------------ the plain chain
__device__ __forceinline__ void f32_cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void f32_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void f32_cp_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

template <int HD> struct PlainF32 {
    static constexpr int TX = HD / 8, RPT = ROWS * TX / F32_THREADS, NK = PAGE / TX;            // lanes a row, rows a thread, keys a thread
    static constexpr int LDQ = ROWS + 4, LDK = HD + 4;
    // Q^T [HD][LDQ], P [PAGE][LDQ], K [PAGE][LDK], V [PAGE][HD]
    static constexpr int SMEM = (HD * LDQ + PAGE * LDQ + PAGE * LDK + PAGE * HD) * 4;
};

// Twice the bits of 2^50, 2^60 and 2^-100: queries and keys from the first on, values from the second on or (zero apart) below the third are
// outside what the planes carry.  (Twice the bits of a number: its sign is gone, a NaN is larger than all.)
#define F32_LARGE_QK ((127u + 50u) << 24)
#define F32_LARGE_V ((127u + 60u) << 24)
#define F32_SMALL_V ((127u - 100u) << 24)

// The tile again with fused multiply-adds alone: a page's products are summed from zero and then added to the scaled output.
// Infinities and NaN reach exactly the rows that see them.  Stored are the rows that see a number outside the planes' range, in their query
// or in a key or value at a position they see; the others keep what the tensor cores gave, so that no row depends on what it cannot see.
template <int HD>
__device__ __noinline__ void f32_plain_walk(const F32Attn &a, float *fsm, int b, int kvh, int g0, int Gc, int q0, int tq, int row0, int start) {
    using C = PlainF32<HD>;
    constexpr int RPT = C::RPT, TX = C::TX, NT = F32_THREADS, NK = C::NK, LDQ = C::LDQ, LDK = C::LDK;
    float *Qs = fsm, *Ps = Qs + HD * LDQ, *Ks = Ps + PAGE * LDQ, *Vs = Ks + PAGE * LDK;
    __shared__ unsigned long long outside_s[2];                          // a bit a key of the page, pages in turn
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    if (tid < 2) outside_s[tid] = 0;
    const int *bt = a.block_table + (size_t)b * a.table_width;
    const size_t H_row = (size_t)kvh * a.G + g0;                         // the first query head of this CTA

    // row r of the tile is token q0 + r / Gc and head g0 + r % Gc; a thread's rows are ty * RPT + i
    int hi[RPT], lo[RPT];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        const int r = ty * RPT + i, t = r / Gc;
        const bool valid = t < tq && g0 + r % Gc < a.G;
        hi[i] = valid ? start + q0 + t : -1;
        lo[i] = valid ? first_visible_key(hi[i], a.window) : 0;
    }
    const int tile_hi = start + q0 + tq - 1, tile_lo = first_visible_key(start + q0, a.window);
    const int page_begin = tile_lo / PAGE, page_end = tile_hi / PAGE + 1;
    // every row of the tile sees all keys of the pages in [whole_begin, whole_end)
    const int whole_begin = (first_visible_key(tile_hi, a.window) + PAGE - 1) / PAGE, whole_end = (start + q0 + 1) / PAGE;

    auto load = [&](float *dst, const float *pool, int page, int ld) {
        const float *src = pool + ((size_t)bt[page] * a.KV + kvh) * PAGE * HD;
#pragma unroll 4
        for (int e = tid; e < PAGE * (HD / 4); e += NT) {
            const int r = e / (HD / 4), c = e % (HD / 4) * 4;
            f32_cp_async16(dst + r * ld + c, src + (size_t)r * HD + c);
        }
    };
    load(Ks, a.k_pool, page_begin, LDK);
    f32_cp_commit();
    load(Vs, a.v_pool, page_begin, HD);
    f32_cp_commit();
    for (int e = tid; e < ROWS * (HD / 4); e += NT) {                     // Q, transposed; lanes side by side along the rows
        const int r = e % ROWS, c = e / ROWS * 4, t = r / Gc, g = g0 + r % Gc;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < tq && g < a.G) v = *(const float4 *)(a.q + (size_t)(row0 + q0 + t) * a.ldq + ((size_t)kvh * a.G + g) * HD + c);
        Qs[c * LDQ + r] = v.x; Qs[(c + 1) * LDQ + r] = v.y; Qs[(c + 2) * LDQ + r] = v.z; Qs[(c + 3) * LDQ + r] = v.w;
    }

    // notes the page's keys that have a number outside the range
    auto look = [&](const float *x, int ld, uint32_t large, uint32_t small, unsigned long long *bits) {
        for (int e = tid; e < PAGE * HD; e += NT) {
            const uint32_t u = __float_as_uint(x[e / HD * ld + e % HD]) << 1;
            if (u >= large || u - 1u < small) atomicOr(bits, 1ull << (e / HD));
        }
    };
    uint32_t stored = 0;                                                  // rows i (bits) that are stored
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
        if (tid == 0) outside_s[(page + 1) & 1] = 0;
        look(Ks, LDK, F32_LARGE_QK, 0u, &outside_s[page & 1]);
        float s[RPT][NK];
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < NK; j++) s[i][j] = 0.f;
#pragma unroll 1
        for (int d = 0; d < HD; d++) {
            float k[NK], x[RPT];
#pragma unroll
            for (int j = 0; j < NK; j++) k[j] = Ks[(tx + TX * j) * LDK + d];
#pragma unroll
            for (int i = 0; i < RPT; i++) x[i] = Qs[d * LDQ + ty * RPT + i];
#pragma unroll
            for (int j = 0; j < NK; j++)
#pragma unroll
                for (int i = 0; i < RPT; i++) s[i][j] = fmaf(x[i], k[j], s[i][j]);
        }
        __syncthreads();                                                  // K is free
        if (page + 1 < page_end) load(Ks, a.k_pool, page + 1, LDK);
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
                s[i][j] *= a.scale;
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
        for (int j = 0; j < NK; j++)
#pragma unroll
            for (int i = 0; i < RPT; i++) Ps[(tx + TX * j) * LDQ + ty * RPT + i] = s[i][j];
        f32_cp_wait1();
        __syncthreads();                                                  // P is written, V of this page is here
        look(Vs, HD, F32_LARGE_V, F32_SMALL_V - 1u, &outside_s[page & 1]);
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
#pragma unroll 1
        for (int k = 0; k < PAGE; k++) {
            const int p = page * PAGE + k;
            const float4 v0 = *(const float4 *)(Vs + k * HD + tx * 4), v1 = *(const float4 *)(Vs + k * HD + tx * 4 + HD / 2);
            const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
            for (int i = 0; i < RPT; i++) {
                if (guarded && (p > hi[i] || p < lo[i])) continue;
                const float x = Ps[k * LDQ + ty * RPT + i];
#pragma unroll
                for (int j = 0; j < 8; j++) pv[i][j] = fmaf(x, v[j], pv[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = fmaf(acc[i][j], corr[i], pv[i][j]);
        __syncthreads();                                                  // V and P are free
        const unsigned long long outside = outside_s[page & 1];
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            const int first = max(lo[i] - page * PAGE, 0), last = min(hi[i] - page * PAGE, PAGE - 1);       // the keys that the row sees
            if (first <= last && (outside >> first << first << (PAGE - 1 - last)) != 0) stored |= 1u << i;
        }
        if (page + 1 < page_end) load(Vs, a.v_pool, page + 1, HD);
        f32_cp_commit();
    }
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        if (hi[i] < 0) continue;
        const int r = ty * RPT + i;
        for (int d = 0; d < HD; d++)
            if (__float_as_uint(Qs[d * LDQ + r]) << 1 >= F32_LARGE_QK) stored |= 1u << i;
        if (!(stored >> i & 1)) continue;
        float *dst = a.out + (size_t)(row0 + q0 + r / Gc) * a.ldo + (H_row + r % Gc) * HD + tx * 4;
        const float inv = l_run[i] > 0.f ? 1.0f / l_run[i] : 0.f;
        *(float4 *)dst = make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
        *(float4 *)(dst + HD / 2) = make_float4(acc[i][4] * inv, acc[i][5] * inv, acc[i][6] * inv, acc[i][7] * inv);
    }
}

// ------------------------------------------------------------------------------------------ tensor cores
__device__ __forceinline__ uint32_t f32_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void f32_mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool f32_mbar_wait(uint32_t bar, uint32_t parity) {
    long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        const long long waited = clock64() - t0;
        if (waited > WAIT_SHORT_CYCLES) {
            // once a wait has run out somewhere, every later wait gives up after a short time
            if (*(volatile int *)&g_f32_attn_error != 0) return false;
            if (waited > *(volatile long long *)&g_f32_attn_wait_limit) return false;
        }
    }
}
__device__ __forceinline__ void f32_raise_error(int role) { atomicCAS(&g_f32_attn_error, 0, (FG_ERR_PIPELINE << 8) | role); }
__device__ __forceinline__ void f32_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void f32_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void f32_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void f32_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D (tensor memory) (+)= A B with A in shared memory, and with A in tensor memory (a lane a row, two neighbouring k a column)
__device__ __forceinline__ void f32_mma_ss(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void f32_mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void f32_tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ void f32_tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ void f32_tmem_st8(uint32_t taddr, const uint32_t (&w)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
// K-major operand tile (rows of 128 B, 8-row groups 1024 B apart), 128-byte swizzle
__device__ __forceinline__ uint64_t f32_desc_k_major(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// MN-major operand tile: rows of 128 B hold 64 consecutive N elements of one k, groups of 8 k are 1024 B apart, blocks of 64 N elements
// `mn_block_bytes` apart
__device__ __forceinline__ uint64_t f32_desc_mn_major(uint32_t saddr, uint32_t mn_block_bytes) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)((mn_block_bytes >> 4) & 0x3FFF) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// bf16 x bf16 -> f32, M x N; b_mn_major: B's rows are k (keys)
__device__ __forceinline__ uint32_t f32_idesc(int M, int N, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// two numbers as a pair of bfloat16, and what is left of them
__device__ __forceinline__ uint32_t f32_split_off(float &a, float &b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    a -= __low2float(t);
    b -= __high2float(t);
    return *(const uint32_t *)&t;
}
// twice the bits of the largest magnitude of eight numbers (a NaN is larger than all), and of the smallest that is not zero, less one
__device__ __forceinline__ void f32_extent(const float4 &x, const float4 &y, uint32_t &largest, uint32_t &smallest) {
    const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t u = __float_as_uint(v[i]) << 1;
        largest = max(largest, u);
        smallest = min(smallest, u - 1u);
    }
}
// eight neighbouring numbers of a row -> 16 bytes of each plane at dst, dst + plane, dst + 2 plane (shared memory)
__device__ __forceinline__ void f32_store_planes(const float4 &x, const float4 &y, uint32_t dst, uint32_t plane) {
    float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
    for (int p = 0; p < 3; p++) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = f32_split_off(v[2 * j], v[2 * j + 1]);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + p * plane), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
    }
}

template <int HD> struct F32Tc {
    static constexpr int CH = HD / 64;                                                // 64-wide chunks of a head
    static constexpr int UNITS = PAGE * HD / 8 / F32_THREADS;                         // runs of eight numbers of a page that a thread splits
    static constexpr int Q_PLANE = ROWS * HD * 2, KV_PLANE = PAGE * HD * 2;
    static constexpr uint32_t P_COL = 64 * CH, O_COL = P_COL + 96, TMEM_COLS = HD == 64 ? 256 : 512;   // score tiles, planes of P, P V of a page
    static constexpr int PLANES = 3 * (Q_PLANE + 2 * KV_PLANE);
    static constexpr int SMEM = 1024 + (PLANES > PlainF32<HD>::SMEM ? PLANES : PlainF32<HD>::SMEM);
    static_assert(O_COL + HD <= TMEM_COLS, "the accumulator fits behind the planes of P");
};
#define F32_P_SCALE 1073741824.0f            // 2^30: what probabilities are multiplied by, for their planes to hold the smallest ones

template <int HD>
__global__ void __launch_bounds__(F32_THREADS, HD == 64 ? 2 : 1) attn_prefill_f32_kernel(const F32Attn a, int skip_few, int test_skip) {
    using C = F32Tc<HD>;
    constexpr int CH = C::CH, UNITS = C::UNITS, OC = HD / 2;                          // OC: output columns of a thread
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ float x_max[2][2][ROWS], x_sum[2][ROWS];
    __shared__ uint32_t tmem_base_s, arrived[2];
    __shared__ int special_s;

    const int G = a.G, KV = a.KV, Gc = G < 16 ? G : 16, TQ = ROWS / Gc, chunks = (G + Gc - 1) / Gc;
    const int per_tile = KV * chunks, tile = blockIdx.x / per_tile, y = blockIdx.x % per_tile;
    const int kvh = y / chunks, g0 = (y % chunks) * Gc, b = blockIdx.z;
    const int row0 = a.cu_rows[b], n_tok = a.cu_rows[b + 1] - row0, start = a.seq_start[b];
    const int q0 = ((int)gridDim.x / per_tile - 1 - tile) * TQ;          // late tiles see the most keys: they start first
    if (q0 >= n_tok || (skip_few && f32_few_rows(n_tok, start, KV * G, a.window, skip_few))) return;
    const int tq = min(TQ, n_tok - q0);
    const int *bt = a.block_table + (size_t)b * a.table_width;
    const int tile_hi = start + q0 + tq - 1, tile_lo = first_visible_key(start + q0, a.window);
    const int p_begin = tile_lo / PAGE, n_iter = tile_hi / PAGE + 1 - p_begin;
    // every row of the tile sees all keys of the pages in [whole_begin, whole_end)
    const int whole_begin = (first_visible_key(tile_hi, a.window) + PAGE - 1) / PAGE, whole_end = (start + q0 + 1) / PAGE;

    const int warp = warp_index(), lane = threadIdx.x & 31, tid = threadIdx.x;
    const uint32_t qs = f32_smem_u32(smem), ks = qs + 3 * C::Q_PLANE, vs = ks + 3 * C::KV_PLANE;
    const uint32_t s_full = f32_smem_u32(&bars[0]), pv_full = s_full + 8;
    if (tid == 0) {
        f32_mbar_init(s_full, 1); f32_mbar_init(pv_full, 1);
        special_s = 0; arrived[0] = arrived[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(f32_smem_u32(&tmem_base_s)), "r"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    f32_fence_before();
    __syncthreads();
    f32_fence_after();
    const uint32_t tmem = tmem_base_s;

    // the last of the eight warps to arrive at a place issues what all of them have prepared (a count an MMA group, eight a page)
    auto last_of = [&](int which) {
        uint32_t n = 0;
        __syncwarp();
        if (lane == 0) asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(n) : "r"(f32_smem_u32(&arrived[which])) : "memory");
        return (__shfl_sync(0xffffffffu, n, 0) & 7) == 7;
    };
    constexpr int PA[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};              // planes of the two factors, the smallest products first
    auto issue_s = [&](int j) {
        if (!last_of(0)) return;
        f32_fence_after();
        if (!(test_skip && j == 0) && elect_one()) {                 // (a test may ask for the first scores to stay away)
            const uint32_t idesc = f32_idesc(ROWS, PAGE, 0);
#pragma unroll
            for (int c = 0; c < CH; c++)
#pragma unroll
                for (int pr = 0; pr < 6; pr++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        f32_mma_ss(tmem + c * 64, f32_desc_k_major(qs + PA[pr] * C::Q_PLANE + c * (ROWS * 128) + k * 32),
                                   f32_desc_k_major(ks + PB[pr] * C::KV_PLANE + c * (PAGE * 128) + k * 32), idesc, (pr | k) != 0);
            f32_commit(s_full);
        }
        __syncwarp();
    };
    auto issue_pv = [&]() {
        if (!last_of(1)) return;
        f32_fence_after();
        if (elect_one()) {
            const uint32_t idesc = f32_idesc(ROWS, HD, 1);
#pragma unroll
            for (int pr = 0; pr < 6; pr++)
#pragma unroll
                for (int k = 0; k < 4; k++)                          // 16 keys = eight columns of P, two 8-key groups of V
                    f32_mma_ts(tmem + C::O_COL, tmem + C::P_COL + PA[pr] * 32 + k * 8,
                               f32_desc_mn_major(vs + PB[pr] * C::KV_PLANE + k * 2048, PAGE * 128), idesc, (pr | k) != 0);
            f32_commit(pv_full);
        }
        __syncwarp();
    };

    {
        // ------------------------------------------------------------ splits and softmax
        const int half = warp >> 2, lg = warp & 3, r = lg * 32 + lane;
        const int t_row = r / Gc, g_row = g0 + r % Gc;
        const bool valid = t_row < tq && g_row < G;
        const int hi = valid ? start + q0 + t_row : -1, lo = valid ? first_visible_key(hi, a.window) : 0;
        const uint32_t trow = tmem + ((uint32_t)(lg * 32) << 16);
        uint32_t largest = 0, smallest = 0xffffffffu, unused = 0xffffffffu;
        bool ok = true;
        // a run of eight numbers of row `row` of a tile of `rows` rows, in 128-byte rows with a 128-byte swizzle
        auto place = [](int row, int c8, int rows) { return (uint32_t)((c8 >> 3) * (rows * 128) + row * 128 + (((c8 & 7) ^ (row & 7)) << 4)); };
        // Q: all 128 rows (rows without a token or head are zero)
#pragma unroll
        for (int i = 0; i < ROWS * HD / 8 / F32_THREADS; i++) {
            const int u = tid + i * F32_THREADS, row = u / (HD / 8), c8 = u % (HD / 8), t = row / Gc, g = g0 + row % Gc;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (t < tq && g < G) {
                const float *src = a.q + (size_t)(row0 + q0 + t) * a.ldq + ((size_t)kvh * G + g) * HD + c8 * 8;
                x = *(const float4 *)src;
                y = *(const float4 *)(src + 4);
            }
            f32_extent(x, y, largest, unused);
            f32_store_planes(x, y, qs + place(row, c8, ROWS), C::Q_PLANE);
        }
        // a page's keys or values: UNITS runs of eight numbers a thread, those that no row of the tile sees as zeros
        float4 buf[2 * UNITS];
        auto fetch = [&](const float *pool, int page) {
            const float *src = pool + ((size_t)bt[page] * KV + kvh) * PAGE * HD;
#pragma unroll
            for (int i = 0; i < UNITS; i++) {
                const int u = tid + i * F32_THREADS, p = page * PAGE + u / (HD / 8);
                buf[2 * i] = buf[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p >= tile_lo && p <= tile_hi) {
                    buf[2 * i] = *(const float4 *)(src + u * 8);
                    buf[2 * i + 1] = *(const float4 *)(src + u * 8 + 4);
                }
            }
        };
        auto store = [&](uint32_t dst) {
#pragma unroll
            for (int i = 0; i < UNITS; i++) {
                const int u = tid + i * F32_THREADS;
                f32_store_planes(buf[2 * i], buf[2 * i + 1], dst + place(u / (HD / 8), u % (HD / 8), PAGE), C::KV_PLANE);
            }
        };
        auto store_k = [&]() {
#pragma unroll
            for (int i = 0; i < UNITS; i++) f32_extent(buf[2 * i], buf[2 * i + 1], largest, unused);
            store(ks);
            f32_fence_async();
        };
        fetch(a.k_pool, p_begin);
        store_k();
        issue_s(0);
        if (n_iter > 1) fetch(a.k_pool, p_begin + 1);

        float acc[OC], m_run = -INFINITY, l_run = 0.f, corr = 1.f;
#pragma unroll
        for (int i = 0; i < OC; i++) acc[i] = 0.f;
        uint32_t v_largest = 0;
        // P V of the page before: acc = acc * corr + pv
        auto gather = [&]() {
            f32_fence_after();
#pragma unroll
            for (int c = 0; c < OC; c += 16) {
                float pv[16];
                f32_tmem_ld16(trow + C::O_COL + half * OC + c, pv);
#pragma unroll
                for (int i = 0; i < 16; i++) acc[c + i] = fmaf(acc[c + i], corr, pv[i]);
            }
        };
        for (int j = 0; j < n_iter; j++) {
            const int page = p_begin + j;
            // (a wait that ran out is not repeated, and the loop goes on: the other warp of these rows meets this one at a barrier)
            if (ok && !f32_mbar_wait(s_full, j & 1)) { f32_raise_error(3); ok = false; }
            f32_fence_after();
            float s[32];
            __syncwarp();
            f32_tmem_ld32(trow + half * 32, s);
            if (CH == 2) {
#pragma unroll
                for (int c = 0; c < 32; c += 16) {
                    float s2[16];
                    f32_tmem_ld16(trow + 64 + half * 32 + c, s2);
#pragma unroll
                    for (int i = 0; i < 16; i++) s[c + i] += s2[i];
                }
            }
            f32_fence_before();
            if (j + 1 < n_iter) {                                    // S of this page is complete and read: K and the score tile are free
                store_k();
                issue_s(j + 1);
            }
            fetch(a.v_pool, page);
            const bool whole = page >= whole_begin && page < whole_end;
            const int p0 = page * PAGE + half * 32;
            float mx = -INFINITY;
            if (whole) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    s[i] *= a.scale;
                    mx = fmaxf(mx, s[i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    s[i] = p0 + i <= hi && p0 + i >= lo ? s[i] * a.scale : -INFINITY;
                    mx = fmaxf(mx, s[i]);
                }
            }
            x_max[j & 1][half][r] = mx;
            asm volatile("barrier.cta.sync %0, 64;" ::"r"(1 + lg) : "memory");         // the two warps of these rows
            const float m_new = fmaxf(m_run, fmaxf(mx, x_max[j & 1][half ^ 1][r]));
            // a row that has seen no key yet keeps its zeros (exp(-inf + inf) is no number)
            const float base = m_new == -INFINITY ? 0.f : m_new;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 32; i++) {
                s[i] = expf(s[i] - base) * F32_P_SCALE;              // (hidden keys: exp(-inf) = 0)
                sum += s[i];
            }
            if (j > 0) {
                if (ok && !f32_mbar_wait(pv_full, (j - 1) & 1)) { f32_raise_error(4); ok = false; }
                __syncwarp();
                gather();
            }
            corr = expf(m_run - base);
            if (m_new == -INFINITY) corr = 1.f;
            l_run = l_run * corr + sum;
            m_run = m_new;
            // V of this page and P, as planes
#pragma unroll
            for (int i = 0; i < UNITS; i++) f32_extent(buf[2 * i], buf[2 * i + 1], v_largest, smallest);
            if (v_largest >= F32_LARGE_V)                            // (for rows that do not see them: zero times them has to be zero)
#pragma unroll
                for (int i = 0; i < 2 * UNITS; i++) {
                    float4 &x = buf[i];
                    auto in = [](float v) { return __float_as_uint(v) << 1 >= F32_LARGE_V ? 0.f : v; };
                    x = make_float4(in(x.x), in(x.y), in(x.z), in(x.w));
                }
            store(vs);
            f32_fence_async();
            if (j + 2 < n_iter) fetch(a.k_pool, page + 2);
#pragma unroll
            for (int c = 0; c < 32; c += 16)
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) w[i] = f32_split_off(s[c + 2 * i], s[c + 2 * i + 1]);
                    f32_tmem_st8(trow + C::P_COL + p * 32 + half * 16 + c / 2, w);
                }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            f32_fence_before();
            issue_pv();
        }
        if (!f32_mbar_wait(pv_full, (n_iter - 1) & 1) && ok) f32_raise_error(4);       // (in any case: nothing is in flight when tensor memory is freed)
        __syncwarp();
        gather();
        f32_fence_before();
        x_sum[half][r] = l_run;
        if (largest >= F32_LARGE_QK || v_largest >= F32_LARGE_V || smallest < F32_SMALL_V - 1u) special_s = 1;      // (every writer writes the same)
        asm volatile("barrier.cta.sync %0, 64;" ::"r"(1 + lg) : "memory");
        const float l = l_run + x_sum[half ^ 1][r];
        if (valid) {
            float *dst = a.out + (size_t)(row0 + q0 + t_row) * a.ldo + ((size_t)kvh * G + g_row) * HD + half * OC;
            const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
            for (int i = 0; i < OC; i += 4) *(float4 *)(dst + i) = make_float4(acc[i] * inv, acc[i + 1] * inv, acc[i + 2] * inv, acc[i + 3] * inv);
        }
    }
    __syncthreads();
    f32_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
    if (special_s) f32_plain_walk<HD>(a, (float *)smem, b, kvh, g0, Gc, q0, tq, row0, start);
}

template <int HD>
static int launch_prefill_f32(const float *q, int ldq, float *out, int ldo, const int *cu_rows, const int *seq_start,
                              const int *block_table, int table_width, const float *k_pool, const float *v_pool, int n_seq,
                              int max_new, int H, int KV, float scale, int window, int skip_few, cudaStream_t stream) {
    static FgPerDevice configured;
    if (fg_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(attn_prefill_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Tc<HD>::SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    const int G = H / KV, Gc = G < 16 ? G : 16, TQ = ROWS / Gc;
    const long long blocks = (long long)KV * ((G + Gc - 1) / Gc) * ((max_new + TQ - 1) / TQ);
    if (blocks > 0x7fffffff) return FG_ERR_BAD_SIZE;
    dim3 grid((unsigned)blocks, 1, n_seq);
    F32Attn a = {q, ldq, out, ldo, cu_rows, seq_start, block_table, table_width, k_pool, v_pool, KV, G, scale, window};
    g_f32_attn_launched.store(true, std::memory_order_relaxed);
    // in plain stream order: a tensor-memory kernel does not start beside another one (see common.cuh)
    return fg_launch_in_order(attn_prefill_f32_kernel<HD>, grid, dim3(F32_THREADS), (size_t)F32Tc<HD>::SMEM, stream, a, skip_few, g_f32_test_skip);
}

// q: [rows, ldq] float32 rows of all sequences one after another (cu_rows[b] = first row of sequence b, seq_start[b] = its length
// before the step); pools [pages, KV, 64, hd] float32; out [rows, ldo] float32.  max_new: most rows any sequence brings.
// skip_few > 0: sequences that f32_few_rows names with pairs = skip_few are left out (the any-size kernel has them).
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
                                            (const float *)k_pool, (const float *)v_pool, n_seq, max_new, H, KV, scale, window, \
                                            skip_few, stream)
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

// skip_few for fg_attention_prefill_f32_ext by the times of both kernels, and whether it leaves a sequence out
extern "C" int fg_attention_f32_skip_few(int hd) { return f32_pairs(hd); }
extern "C" int fg_attention_f32_left_out(int tokens, int past, int heads, int hd, int window) { return f32_few_rows(tokens, past, heads, window, f32_pairs(hd)); }

// Pages of 64 keys that the longest tile of a sequence walks (*walk), and the times of both kernels in such walks: of the any-size kernel
// (*any_size) and of all the sequence's tiles on a GPU of n_sm SMs (*tiles).
extern "C" int fg_attention_f32_cost(int tokens, int past, int H, int KV, int hd, int window, int n_sm, double *any_size, double *tiles, double *walk) {
    const double keys = window ? min(past, window > 0 ? window : -window) : past, seen = keys + 0.5 * tokens;
    const int G = H / KV, Gc = G < 16 ? G : 16, TQ = ROWS / Gc;
    const double ctas = (double)((tokens + TQ - 1) / TQ) * KV * ((G + Gc - 1) / Gc);
    *walk = (keys + tokens) / PAGE + 1.0;
    *any_size = (double)tokens * H * (seen / PAGE + 1.0) / f32_pairs(hd);           // (a pair's block takes a page's time beside its pages')
    *tiles = ctas * (seen / PAGE + 1.0) / ((hd == 64 ? 1.23 : 0.86) * n_sm);        // (2,048 tokens: an SM walks a page in 2.8 us, 5.8 at 128)
    return 0;
}
