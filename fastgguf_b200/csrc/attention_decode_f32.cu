// Decode attention in float32 over the paged cache, one new token a sequence: rotation of q and of the new k, cache append of k and v, and
// attention in ONE kernel, as attention_decode.cu has it in bfloat16.  Head sizes 16, 32, 64 and 128, pages of 64 keys.
//
// Reference role: attn_rows for one token (fastgguf.c:4769-4786), rope (fastgguf.c:3273-3326).
//
// What a row gives depends on its own sequence alone: the units (a half page, 32 keys; head sizes 16 and 32: a page) that the token sees are
// cut into R runs, R the smallest power of two that leaves none longer than one unit, 64 at most; a run is walked from its first unit on, and
// the runs' (maximum, sum, output) meet in a binary tree, neighbours first.  Which warp of which CTA walks a run, and where two results meet, is
// free, and follows the step's shape.
//
// Grid (split, chunk of NH query heads, kv head, sequence, in one dimension), the splits of a (sequence, kv head, chunk) a cluster.  A warp has a row of
// neighbouring runs, with a K and a V buffer of its own (cp.async; the next K is asked for when the scores are done, the next V behind P V) and a
// stack of results that wait for their neighbour.  The cache holds only older tokens - the new one comes in registers from the projection's
// row -, so the first loads start before the wait on the kernel in front (see common.cuh for why that is allowed: positions, the page
// table and this entry's pool are written by no kernel that may still run).
//   scores   a lane has one key (small heads: two; their rows in shared memory, padded) and NH query heads (broadcast)
//   P V      a lane has HD / 32 of the output's columns (HD 16: one, of half the keys), a unit's products are summed in chains of 16
// Products and sums are float32 fused multiply-adds, exponentials expf; sums change their base by powers of two.
//
// Bound by memory where there are many long sequences (64 of 1,000 keys, a query head a key head: 153 us, 6.8 TB/s), else by latency: a unit's
// load, scores, softmax and P V one behind the other, then the merge (3.7 us with one unit a warp and no cluster).  Times a layer behind one another (us): rotation and the any-size kernel :
// this kernel when a page was walked by one of six warps in every CTA of 217 KB, with four rows whatever the group has : as it is.
//   32 heads of 64 on 8 key heads   1 x 2,000 keys 56 : 8.5 : 8.1   1 x 16,000 401 : 33.5 : 25   8 x 1,000 59 : 15 : 12.5   64 x 200 58 : 30 : 19   256 x 20 76 : 90 : 25
//   32 heads of 64 on 32            1 x 2,000 62 : 14.5 : 11        64 x 1,000 242 : 246 : 153   256 x 20 91 : 335 : 53
//   32 heads of 128 on 8            8 x 1,000 65 : 28 : 22          64 x 1,000 395 : 176 : 131
//   4 heads of 16 on 2              8 x 40 5.7 : 5.4 : 4.5          256 x 300 25 : 8.8 : 7.9
//   16 heads of 32 on 4             8 x 40 6.9 : 5.3 : 5.3          8 x 1,000 34 : 6.6 : 7.3
// Distance from float64, against the any-size kernel's (2-norm, 1.00 there): 0.98 to 0.90 at head sizes 64 and 128, 0.96 to 0.73 at 16 and 32.
#include "common.cuh"

#define PAGE 64
#define RUNS 64                                // runs of a sequence at most
#define CHAIN 16                               // weighted values that are added one to the other

__device__ __forceinline__ void df_cp16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void df_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void df_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// N neighbouring numbers, N * 4 bytes aligned
template <int N> __device__ __forceinline__ void df_load(const float *src, float (&v)[N]) {
    if (N == 4) { const float4 x = *(const float4 *)src; v[0] = x.x; v[1 % N] = x.y; v[2 % N] = x.z; v[3 % N] = x.w; }
    else if (N == 2) { const float2 x = *(const float2 *)src; v[0] = x.x; v[1 % N] = x.y; }
    else v[0] = src[0];
}
template <int N> __device__ __forceinline__ void df_store(float *dst, const float (&v)[N]) {
    if (N == 4) *(float4 *)dst = make_float4(v[0], v[1 % N], v[2 % N], v[3 % N]);
    else if (N == 2) *(float2 *)dst = make_float2(v[0], v[1 % N]);
    else dst[0] = v[0];
}

struct DecodeF32 {
    const float *qkv; int ldq;                 // rows of (q heads | k heads | v heads), not rotated
    float *out; int ldo;
    const int *positions, *block_table; int table_width;
    float *k_pool, *v_pool;                    // [pages, KV, 64, HD]
    const float *cos_t, *sin_t;                // [positions, HD / 2]
    int H, KV, G;
    float scale;
    int window;
};

// Weights are exp(score - base), the base a multiple of ln 2 just above the largest score so far, subtracted in two parts (Cody and Waite).  What
// was summed under one base then goes over to another by a power of two, exactly: with factors exp(old maximum - new maximum) every sum
// would carry the rounding of each factor it met.  Maxima of 2^20 and more, where such multiples get coarse, and infinite ones are bases
// themselves.
#define LN2_HI 0.693147180559945309f                                           /* as a float, */
#define LN2_LO ((float)(0.693147180559945309 - (double)LN2_HI))                /* and what that leaves */
__device__ __forceinline__ bool df_small(float m) { return fabsf(m) < 1048576.f; }
__device__ __forceinline__ float df_multiple(float m) { return df_small(m) ? ceilf(__fmul_rn(m, 1.44269504f)) : 0.f; }       // (1 / ln 2)
__device__ __forceinline__ float df_rest(float m) { return df_small(m) || m == -INFINITY ? 0.f : m; }
__device__ __forceinline__ float df_less(float x, float k) { return fmaf(-k, LN2_LO, fmaf(-k, LN2_HI, x)); }       // x - k ln 2
// from the base of maximum `old` to that of `now` (not below it).  A sum whose maximum is -inf holds nothing but zeros, or a NaN that stays.
__device__ __forceinline__ float df_factor(float old, float now) {
    const float ko = df_multiple(old), kn = df_multiple(now), d = ko - kn;
    float f = old == -INFINITY || d < -126.f ? 0.f : __uint_as_float((uint32_t)(127 + (int)d) << 23);
    if (old > -INFINITY && !(df_small(old) && df_small(now))) f = old == now ? 1.f : expf(df_less(df_less(__fsub_rn(df_rest(old), df_rest(now)), kn), -ko));
    return f;
}
// (roundings named one by one here and below: which products go into a multiply-add must not change from one instance of the kernel to the next)
__device__ __forceinline__ void df_rotate(float x, float z, float c, float s, float &a, float &b) {
    a = fmaf(x, c, -__fmul_rn(z, s));
    b = fmaf(x, s, __fmul_rn(z, c));
}
// the largest of a warp's numbers, NaN left out: one integer reduction in place of five exchanges
__device__ __forceinline__ float df_warp_max(float x) {
    int i = __float_as_int(x == x ? x : -INFINITY);
    i = __reduce_max_sync(0xffffffffu, i ^ ((i >> 31) & 0x7fffffff));
    return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}
// a warp's sums of N numbers each, number lane * N / 32's in a lane
template <int N> __device__ __forceinline__ float df_warp_sums(const float (&x)[N], int lane) {
    float y = x[0];
    const bool high = lane & 16, odd = lane & 8;
    if (N == 4) {
        const float a = (high ? x[2 % N] : x[0]) + __shfl_xor_sync(0xffffffffu, high ? x[0] : x[2 % N], 16);
        const float b = (high ? x[3 % N] : x[1 % N]) + __shfl_xor_sync(0xffffffffu, high ? x[1 % N] : x[3 % N], 16);
        y = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
    } else {
        y = N == 2 ? (high ? x[1 % N] : x[0]) + __shfl_xor_sync(0xffffffffu, high ? x[0] : x[1 % N], 16) : y + __shfl_xor_sync(0xffffffffu, y, 16);
        y += __shfl_xor_sync(0xffffffffu, y, 8);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y;
}
// The tree over n results of neighbours (a power of two, 8 at most), every `step`-th of which there is.  Its node j (1: the root, 2 j and 2 j + 1
// below it) joins the `half` results from 2 half (j - 2^level) on with the next half.  Lanes 8 g + j of a warp find the factors of head g's node j from
// the maxima alone, m(i) of result i, into f[2 (8 g + j)]; what a node joins is then one multiplication and one multiply-add.
template <typename M> __device__ __forceinline__ void df_node_factors(int n, int step, int lane, int heads, float *f, M m) {
    const int j = lane & 7;
    if (lane < 8 * heads && j > 0 && j < n) {
        const int level = 31 - __clz(j), half = n >> (level + 1), first = 2 * half * (j - (1 << level));
        float ma = -INFINITY, mb = -INFINITY;
        for (int i = 0; i < half; i += step) {
            ma = fmaxf(ma, m(first + i));
            mb = fmaxf(mb, m(first + half + i));
        }
        const float top = fmaxf(ma, mb);
        f[2 * lane] = df_factor(ma, top);
        f[2 * lane + 1] = df_factor(mb, top);
    }
}
template <int N> __device__ __forceinline__ void df_tree(float (&l)[N], float (&o)[N], int n, int step, const float *f) {
#pragma unroll
    for (int s = 1; s < N; s *= 2) {
        if (s < step || s >= n) continue;
#pragma unroll
        for (int i = 0; i + s < N; i += 2 * s) {
            if (i >= n) break;
            const float2 w = *(const float2 *)(f + 2 * ((n + i) / (2 * s)));
            l[i] = fmaf(w.y, l[i + s], __fmul_rn(w.x, l[i]));
            o[i] = fmaf(w.y, o[i + s], __fmul_rn(w.x, o[i]));
        }
    }
}

template <int HD, int NW, int NH> struct DfSizes {
    static constexpr int log2_of(int n) { return n <= 1 ? 0 : 1 + log2_of(n / 2); }
    static constexpr int UNIT = HD >= 64 ? 32 : 64;                             // keys that a warp takes at a time: a half page, small heads: a page
    static constexpr int LDK = HD + 4, K = UNIT * LDK, WARP = K + UNIT * HD;
    static constexpr int Q = NH * HD, P = UNIT * NH > 64 ? UNIT * NH : 64;
    static constexpr int STATE = NH * (HD + 2), DEPTH = log2_of(RUNS / NW);      // a result (maximum, sum, output a head), and how many a warp may have waiting
    static constexpr int SMEM = (NW * (WARP + P + DEPTH * STATE) + Q + (NW + 1) * STATE) * 4;
    static constexpr int CTAS = (HD >= 64 ? 8 : 16) / NW;                       // what registers leave room for on an SM
};

template <int HD, int NW, int NH>
__global__ void __launch_bounds__(NW * 32, DfSizes<HD, NW, NH>::CTAS)
attn_decode_f32_kernel(const DecodeF32 a, int n_splits) {
    using Z = DfSizes<HD, NW, NH>;
    constexpr int UNIT = Z::UNIT, KPL = UNIT / 32, LDK = Z::LDK, DPL = HD >= 32 ? HD / 32 : 1, KGRP = 32 * DPL / HD, CHAINS = UNIT / (CHAIN * KGRP), HALF = HD / 2;
    extern __shared__ __align__(16) float dsm[];
    const int warp = warp_index(), lane = threadIdx.x & 31, tid = threadIdx.x;
    float *Ks = dsm + warp * Z::WARP, *Vs = Ks + Z::K;
    float *qs = dsm + NW * Z::WARP, *ps = qs + Z::Q + warp * Z::P;
    float *held = qs + Z::Q + NW * Z::P + warp * Z::DEPTH * Z::STATE, *parts = qs + Z::Q + NW * (Z::P + Z::DEPTH * Z::STATE), *one = parts + NW * Z::STATE;
    const int chunks = (a.G + NH - 1) / NH;
    const int split = blockIdx.x & (n_splits - 1), y = blockIdx.x >> (31 - __clz(n_splits)), head = y % (a.KV * chunks), b = y / (a.KV * chunks);
    const int kvh = head / chunks, g0 = (head % chunks) * NH;
    const int rows = min(NH, a.G - g0);
    pdl_launch_dependents();
    const int pos = a.positions[b], lo_key = first_visible_key(pos, a.window), first_unit = lo_key / UNIT, last_unit = pos / UNIT;
    const int n_units = last_unit - first_unit + 1, log_r = n_units > RUNS / 2 ? Z::log2_of(RUNS) : 32 - __clz(n_units - 1);
    const int workers = n_splits * NW, worker = split * NW + warp;
    const int log_w = 31 - __clz(workers), step = 1 << max(log_w - log_r, 0);          // every step-th worker has runs
    const int runs = log_r >= log_w ? 1 << (log_r - log_w) : (worker & (step - 1)) == 0, run0 = log_r >= log_w ? worker << (log_r - log_w) : worker >> (log_w - log_r);
    auto unit_of = [&](int r) { return first_unit + (int)((long long)n_units * r >> log_r); };
    const int *bt = a.block_table + (size_t)b * a.table_width;
    auto load = [&](float *dst, int ld, const float *pool, int u) {             // rows in front of the new token
        const float *src = pool + (((size_t)bt[u * UNIT / PAGE] * a.KV + kvh) * PAGE + u * UNIT % PAGE) * HD;
        const int n = min(UNIT, pos - u * UNIT) * (HD / 4);
#pragma unroll 8
        for (int e = lane; e < n; e += 32) df_cp16(dst + e / (HD / 4) * ld + e % (HD / 4) * 4, src + e * 4);
    };
    int u = unit_of(run0);
    const int u_end = unit_of(run0 + runs);
    if (u < u_end) {
        load(Ks, LDK, a.k_pool, u);
        df_commit();
        load(Vs, HD, a.v_pool, u);
        df_commit();
    }
    pdl_wait();                                // q, k and v of the new token come from the kernel in front
    const float *row = a.qkv + (size_t)b * a.ldq, *cs = a.cos_t + (size_t)pos * HALF, *sn = a.sin_t + (size_t)pos * HALF;
    for (int e = tid; e < NH * HALF; e += NW * 32) {
        const int g = e / HALF, j = e % HALF;
        float x = 0.f, z = 0.f;
        if (g < rows) {
            const float *q = row + (size_t)(kvh * a.G + g0 + g) * HD;
            x = q[j]; z = q[j + HALF];
        }
        const float c = cs[j], s = sn[j];
        df_rotate(x, z, c, s, qs[g * HD + j], qs[g * HD + j + HALF]);
    }
    __syncthreads();
    float acc[NH][DPL], m[NH], l[NH];                                          // (l: of this lane's keys)
    const int dl = lane * DPL % HD, kg = lane * DPL / HD, gl = lane * NH / 32;     // this lane's columns of P V, its part of the keys, and the head whose sum it has
    for (int c = 0; c < runs; c++) {
        const int run_end = unit_of(run0 + c + 1);
#pragma unroll
        for (int g = 0; g < NH; g++) {
            m[g] = -INFINITY; l[g] = 0.f;
#pragma unroll
            for (int d = 0; d < DPL; d++) acc[g][d] = 0.f;
        }
        for (; u < run_end; u++) {
            const int key0 = u * UNIT;
            df_wait<1>();                      // K of these keys is here
            __syncwarp();
            if (u == last_unit) {
                // the rotated k of the new token into the tile, and into the cache once a kv head
                const int off = pos % UNIT;
                const float *k = row + (size_t)(a.H + kvh) * HD;
                float *dst = a.k_pool + (((size_t)bt[pos / PAGE] * a.KV + kvh) * PAGE + pos % PAGE) * HD;
                for (int j = lane; j < HALF; j += 32) {
                    float r0, r1;
                    df_rotate(k[j], k[j + HALF], cs[j], sn[j], r0, r1);
                    Ks[off * LDK + j] = r0;
                    Ks[off * LDK + j + HALF] = r1;
                    if (g0 == 0) { dst[j] = r0; dst[j + HALF] = r1; }
                }
                __syncwarp();
            }
            float s[KPL][NH];
#pragma unroll
            for (int x = 0; x < KPL; x++)
#pragma unroll
                for (int g = 0; g < NH; g++) s[x][g] = 0.f;
#pragma unroll 8
            for (int d = 0; d < HD; d += 4) {
                float4 k[KPL];
#pragma unroll
                for (int x = 0; x < KPL; x++) k[x] = *(const float4 *)(Ks + (lane + 32 * x) * LDK + d);
#pragma unroll
                for (int g = 0; g < NH; g++) {
                    const float4 q = *(const float4 *)(qs + g * HD + d);
#pragma unroll
                    for (int x = 0; x < KPL; x++) {
                        s[x][g] = fmaf(q.x, k[x].x, s[x][g]); s[x][g] = fmaf(q.y, k[x].y, s[x][g]);
                        s[x][g] = fmaf(q.z, k[x].z, s[x][g]); s[x][g] = fmaf(q.w, k[x].w, s[x][g]);
                    }
                }
            }
            __syncwarp();
            if (u + 1 < u_end) load(Ks, LDK, a.k_pool, u + 1);
            df_commit();
            bool see[KPL];
#pragma unroll
            for (int x = 0; x < KPL; x++) see[x] = key0 + lane + 32 * x >= lo_key && key0 + lane + 32 * x <= pos;
            float corr[NH], w[KPL][NH];
#pragma unroll
            for (int g = 0; g < NH; g++) {
                float most = -INFINITY;
#pragma unroll
                for (int x = 0; x < KPL; x++) {
                    s[x][g] = __fmul_rn(s[x][g], a.scale);
                    if (see[x]) most = fmaxf(most, s[x][g]);
                }
                // (a NaN score makes its weight NaN; a maximum of -inf stands for base 0, and such keys count for nothing beside others)
                const float m_new = fmaxf(m[g], df_warp_max(most)), k = df_multiple(m_new), rest = df_rest(m_new);
                corr[g] = df_factor(m[g], m_new);
                m[g] = m_new;
#pragma unroll
                for (int x = 0; x < KPL; x++) {
                    w[x][g] = see[x] ? expf(df_less(__fsub_rn(s[x][g], rest), k)) : 0.f;
                    l[g] = x == 0 ? fmaf(l[g], corr[g], w[x][g]) : __fadd_rn(l[g], w[x][g]);
                }
            }
#pragma unroll
            for (int x = 0; x < KPL; x++) df_store<NH>(ps + (lane + 32 * x) * NH, w[x]);
            df_wait<1>();                      // V of these keys is here
            __syncwarp();
            if (u == last_unit) {
                const int off = pos % UNIT;
                const float *v = row + (size_t)(a.H + a.KV + kvh) * HD;
                float *dst = a.v_pool + (((size_t)bt[pos / PAGE] * a.KV + kvh) * PAGE + pos % PAGE) * HD;
                for (int j = lane; j < HD; j += 32) {
                    Vs[off * HD + j] = v[j];
                    if (g0 == 0) dst[j] = v[j];
                }
                __syncwarp();
            }
            float pv[CHAINS][NH][DPL];
#pragma unroll
            for (int i = 0; i < CHAINS; i++)
#pragma unroll
                for (int g = 0; g < NH; g++)
#pragma unroll
                    for (int d = 0; d < DPL; d++) pv[i][g][d] = 0.f;
            auto add = [&](int i, int k) {
                float wg[NH], v[DPL];
                df_load<NH>(ps + k * NH, wg);
                df_load<DPL>(Vs + k * HD + dl, v);
#pragma unroll
                for (int g = 0; g < NH; g++)
#pragma unroll
                    for (int d = 0; d < DPL; d++) pv[i][g][d] = fmaf(wg[g], v[d], pv[i][g][d]);
            };
            // (keys outside what the token sees are left out: zero times what a page happens to hold need not be zero)
            const int k_lo = lo_key - key0, k_hi = pos - key0;
            if (k_lo <= 0 && k_hi >= UNIT - 1) {
#pragma unroll 8
                for (int k = 0; k < CHAIN; k++)
#pragma unroll
                    for (int i = 0; i < CHAINS; i++) add(i, k + (i + kg * CHAINS) * CHAIN);
            } else {
#pragma unroll
                for (int i = 0; i < CHAINS; i++) {
                    const int first = (i + kg * CHAINS) * CHAIN, end = min(first + CHAIN - 1, k_hi);
#pragma unroll 4
                    for (int k = max(first, k_lo); k <= end; k++) add(i, k);
                }
            }
            __syncwarp();
            if (u + 1 < u_end) load(Vs, HD, a.v_pool, u + 1);
            df_commit();
#pragma unroll
            for (int g = 0; g < NH; g++)
#pragma unroll
                for (int d = 0; d < DPL; d++) {
#pragma unroll
                    for (int i = 1; i < CHAINS; i *= 2)
#pragma unroll
                        for (int x = 0; x + i < CHAINS; x += 2 * i) pv[x][g][d] = __fadd_rn(pv[x][g][d], pv[x + i][g][d]);
                    if (KGRP > 1) pv[0][g][d] = __fadd_rn(pv[0][g][d], __shfl_xor_sync(0xffffffffu, pv[0][g][d], HD / DPL));
                    acc[g][d] = fmaf(acc[g][d], corr[g], pv[0][g][d]);
                }
        }
        // The run is done: it joins the results that wait for it, and waits itself for the next one.
        float sum = df_warp_sums<NH>(l, lane);
        int depth = __popc(c);                                                 // results that wait: one for every bit of c
        for (int t = c; t & 1; t >>= 1) {
            const float *left = held + --depth * Z::STATE;
            float fa[NH], fb[NH];
            __syncwarp();
#pragma unroll
            for (int g = 0; g < NH; g++) {
                const float *x = left + g * (HD + 2);
                const float ma = x[0], top = fmaxf(ma, m[g]);
                fa[g] = df_factor(ma, top); fb[g] = df_factor(m[g], top);
                m[g] = top;
#pragma unroll
                for (int d = 0; d < DPL; d++) acc[g][d] = fmaf(fb[g], acc[g][d], __fmul_rn(fa[g], x[2 + dl + d]));
            }
#pragma unroll
            for (int g = 0; g < NH; g++)
                if (g == gl) sum = fmaf(fb[g], sum, __fmul_rn(fa[g], left[g * (HD + 2) + 1]));
        }
        float *dst = c + 1 < runs ? held + depth * Z::STATE : parts + warp * Z::STATE;
        __syncwarp();
        if (lane % (32 / NH) == 0) dst[gl * (HD + 2) + 1] = sum;
#pragma unroll
        for (int g = 0; g < NH; g++) {
            if (lane == 0) dst[g * (HD + 2)] = m[g];
            if (kg == 0)
#pragma unroll
                for (int d = 0; d < DPL; d++) dst[g * (HD + 2) + 2 + dl + d] = acc[g][d];
        }
    }
    df_wait<0>();
    __syncthreads();
    auto store = [&](int g, int d, float M, float L, float O) {
        a.out[(size_t)b * a.ldo + (size_t)(kvh * a.G + g0 + g) * HD + d] = M == -INFINITY ? M - M : O / L;      // no finite score at all: no number
    };
    // the warps' results, where this CTA has any (its first warp's, then); every warp finds the factors for itself, where its weights were
    const int step_cta = max(step / NW, 1);
    if ((split & (step_cta - 1)) == 0) {
        if (step < NW) {
            df_node_factors(NW, step, lane, rows, ps, [&](int i) { return parts[i * Z::STATE + (lane >> 3) * (HD + 2)]; });
            __syncwarp();
        }
        for (int e = tid; e < rows * HD; e += NW * 32) {
            const int g = e / HD, d = e % HD;
            float M = -INFINITY, L[NW], O[NW];
#pragma unroll
            for (int i = 0; i < NW; i++)
                if ((i & (step - 1)) == 0) {
                    const float *x = parts + i * Z::STATE + g * (HD + 2);
                    M = fmaxf(M, x[0]); L[i] = x[1]; O[i] = x[2 + d];
                }
            df_tree<NW>(L, O, NW, step, ps + 16 * g);
            if (n_splits == 1) { store(g, d, M, L[0], O[0]); continue; }
            one[g * (HD + 2) + 2 + d] = O[0];
            if (d == 0) { one[g * (HD + 2)] = M; one[g * (HD + 2) + 1] = L[0]; }
        }
    }
    if (n_splits == 1) return;
    // the CTAs of a cluster leave theirs in shared memory, and each gathers its share of the columns from all of them
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t one_s = (uint32_t)__cvta_generic_to_shared(one);
    auto remote = [&](int rank, int i) {
        uint32_t at;
        float v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(one_s + i * 4), "r"(rank));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
        return v;
    };
    const int share = (rows * HD + n_splits - 1) / n_splits;
    if (warp * 32 < share) {
        float M[8];                            // of head lane / 8
#pragma unroll
        for (int i = 0; i < 8; i++) M[i] = i < n_splits && (i & (step_cta - 1)) == 0 && (lane >> 3) < rows ? remote(i, (lane >> 3) * (HD + 2)) : -INFINITY;
        df_node_factors(n_splits, step_cta, lane, rows, ps, [&](int at) {
            float x = -INFINITY;
#pragma unroll
            for (int i = 0; i < 8; i++) x = i == at ? M[i] : x;
            return x;
        });
        __syncwarp();
    }
    for (int e = split * share + tid; e < min(rows * HD, (split + 1) * share); e += NW * 32) {
        const int g = e / HD, d = e % HD;
        float M = -INFINITY, L[8], O[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            L[i] = O[i] = 0.f;
            if (i < n_splits && (i & (step_cta - 1)) == 0) {
                M = fmaxf(M, remote(i, g * (HD + 2)));
                L[i] = remote(i, g * (HD + 2) + 1); O[i] = remote(i, g * (HD + 2) + 2 + d);
            }
        }
        df_tree<8>(L, O, n_splits, step_cta, ps + 16 * g);
        store(g, d, M, L[0], O[0]);
    }
    // nobody leaves while another still reads its shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int HD, int NW, int NH>
static int launch_decode_f32(const DecodeF32 &a, int B, int n_splits, cudaStream_t stream) {
    using Z = DfSizes<HD, NW, NH>;
    static_assert(Z::SMEM <= 227 * 1024, "a CTA's shared memory");
    static FgPerDevice configured;
    if (fg_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(attn_decode_f32_kernel<HD, NW, NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, Z::SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    const long long blocks = (long long)n_splits * a.KV * ((a.G + NH - 1) / NH) * B;
    if (blocks > 0x7fffffff) return FG_ERR_BAD_SIZE;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks); cfg.blockDim = dim3(NW * 32); cfg.dynamicSmemBytes = Z::SMEM; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (fg_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (n_splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = n_splits; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr; cfg.numAttrs = n;
    return (int)cudaLaunchKernelEx(&cfg, attn_decode_f32_kernel<HD, NW, NH>, a, n_splits);
}

// (sequence, kv head, chunk of n query heads) triples of a step
static long long df_items(int B, int H, int KV, int n) { return (long long)B * KV * ((H / KV + n - 1) / n); }

// Splits of a sequence, by the step's shape: as many CTAs as fill the GPU once.  Clusters of eight fill half of it: sixteen of them do not find room at
// once (8 sequences, 8 heads of 64 on one key head, 160 keys: 11.1 us, in clusters of four 5.7).
extern "C" int fg_attention_decode_f32_splits(int B, int H, int KV, int table_width, int n_sm) {
    if (B <= 0 || KV <= 0 || H <= 0 || H % KV) return 1;
    const long long ctas = df_items(B, H, KV, 4);
    int s = 1;
    while (s < 8 && 2 * s * ctas <= (s == 4 ? n_sm / 2 : n_sm) && 2 * s <= table_width) s *= 2;
    return s;
}

// Warps a CTA, by the number of CTAs: eight have an SM to themselves (head size 64), four share it with another CTA, two with three others.
// Head size 64 (us, eight : four : two warps): 256 CTAs of 300 keys 19.9 : 13.0 : 19.2; 512 of 1,000 64 : 53 : 49, of up to 2,000 73 : 73 : 86; 2,048 of
// 20 70 : 36 : 24.  Small heads, 128 CTAs in clusters of four: 7.3 : 6.3.
static int df_warps(long long items, int n_splits, int hd) {
    const long long ctas = items * n_splits;
    return ctas > 592 ? 2 : ctas > (hd <= 32 ? 64 : 148) || hd == 128 ? 4 : 8;
}

// qkv: [B, ldq] float32 rows straight from the projection; positions[b] is the new token's place; n_splits 1, 2, 4 or 8, warps 2, 4 or 8 (head
// size 128: 2 or 4), 0: by the step's shape.  Neither changes a bit of what comes out.  Refuses (FG_ERR_BAD_SIZE) other head sizes and pages, and
// pools that are not 16-byte aligned; fg_rope_append and the any-size kernel take those.
extern "C" int fg_attention_decode_f32_ext(const void *qkv, int ldq, void *out, int ldo, const int *positions, const int *block_table, int table_width,
                                           void *k_pool, void *v_pool, const float *cos_t, const float *sin_t, int B, int H, int KV, int hd, int page_size,
                                           float scale, int window, int n_splits, int warps, cudaStream_t stream) {
    if (B <= 0) return 0;
    if (page_size != PAGE || KV <= 0 || H <= 0 || H % KV || B > 65535 || (n_splits != 1 && n_splits != 2 && n_splits != 4 && n_splits != 8) ||
        (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15))
        return FG_ERR_BAD_SIZE;
    const DecodeF32 a = {(const float *)qkv, ldq, (float *)out, ldo, positions, block_table, table_width, (float *)k_pool, (float *)v_pool, cos_t, sin_t, H, KV, H / KV,
                         scale, window};
    // (two heads a CTA where four of a small size leave the GPU idle: 8 sequences of 40 keys, 32 heads of 16 on 8, 5.3 us with four, 4.6 with two)
    const int G = H / KV, nh = G < 3 ? G : hd <= 32 && df_items(B, H, KV, 2) <= 128 ? 2 : 4;
    if (warps == 0) warps = df_warps(df_items(B, H, KV, nh), n_splits, hd);
#define DF_HEADS_OF(HD, NW) (nh == 4 ? launch_decode_f32<HD, NW, 4>(a, B, n_splits, stream) : \
                             nh == 2 ? launch_decode_f32<HD, NW, 2>(a, B, n_splits, stream) : launch_decode_f32<HD, NW, 1>(a, B, n_splits, stream))
#define DF_RUN(HD, NW) do { if (hd == HD && warps == NW) return DF_HEADS_OF(HD, NW); } while (0)
    DF_RUN(16, 2); DF_RUN(16, 4); DF_RUN(16, 8);
    DF_RUN(32, 2); DF_RUN(32, 4); DF_RUN(32, 8);
    DF_RUN(64, 2); DF_RUN(64, 4); DF_RUN(64, 8);
    DF_RUN(128, 2); DF_RUN(128, 4);
#undef DF_RUN
#undef DF_HEADS_OF
    return FG_ERR_BAD_SIZE;
}

extern "C" int fg_attention_decode_f32(const void *qkv, int ldq, void *out, int ldo, const int *positions, const int *block_table, int table_width,
                                       void *k_pool, void *v_pool, const float *cos_t, const float *sin_t, int B, int H, int KV, int hd, int page_size,
                                       float scale, int window, int n_splits, cudaStream_t stream) {
    return fg_attention_decode_f32_ext(qkv, ldq, out, ldo, positions, block_table, table_width, k_pool, v_pool, cos_t, sin_t, B, H, KV, hd, page_size, scale,
                                       window, n_splits, 0, stream);
}
