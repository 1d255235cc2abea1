// Decode attention in float32 over the paged cache, one new token a sequence: rotation of q and of the new k, cache append of k and v, and
// attention in ONE kernel, as attention_decode.cu has it in bfloat16.  Head sizes 16, 32, 64 and 128, pages of 64 keys.
//
// Reference role: attn_rows for one token (fastgguf.c:4769-4786), rope (fastgguf.c:3273-3326).
//
// Grid (split x kv head x chunk of four query heads, sequence), the splits of a (sequence, kv head) a cluster.  A sequence's pages are divided
// evenly among the splits, a CTA's warps take its pages in turn, each with a K and a V buffer of its own (cp.async; the next K is asked for when
// the scores are done, the next V behind P V).  Pages hold only older tokens - the new one comes in registers from the projection's row -, so the
// first loads start before the wait on the kernel in front (see common.cuh for why that is allowed: positions, the page table and this
// entry's pool are written by no kernel that may still run).
//   scores   a lane has two keys (their rows in shared memory, padded) and four query heads (broadcast)
//   P V      a lane has HD / 32 of the output's columns (HD 16: half of the keys), a page's products are summed from zero
// Products and sums are float32 fused multiply-adds, exponentials expf; pages are added in ascending order a warp, warps and splits in their order,
// and which page is whose follows from the sequence's length and the step's shape alone.
//
// Bound by latency: the any-size kernel gives a (row, head) a block that starts after the rotation's kernel and reads its keys thread by
// thread.  Inside a step of 8 sequences (Llama 1B sizes, contexts of 17 to 160): 12.0 us, 4.0 us for the rotation and 4.1 for each norm
// before.  This kernel and the norm in registers (elementwise.cu) take the step from 1.54 to 1.39 ms, the tiny model's of the tests from 45 to 41 us.
#include "common.cuh"

#define PAGE 64
#define DF_HEADS 4                             // query heads a CTA takes

__device__ __forceinline__ void df_cp16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void df_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void df_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

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

template <int HD, int NW> struct DfSizes {
    static constexpr int LDK = HD + 4, K_FLOATS = PAGE * LDK, V_FLOATS = PAGE * HD, WARP = K_FLOATS + V_FLOATS;
    static constexpr int Q = DF_HEADS * HD, P = PAGE * DF_HEADS, PARTS = NW * DF_HEADS * (HD + 2), ONE = DF_HEADS * (HD + 2);
    static constexpr int SMEM = (NW * WARP + Q + NW * P + PARTS + ONE) * 4;
};

template <int HD, int NW>
__global__ void __launch_bounds__(NW * 32)
attn_decode_f32_kernel(const DecodeF32 a, int n_splits) {
    using Z = DfSizes<HD, NW>;
    constexpr int LDK = Z::LDK, DPL = HD >= 32 ? HD / 32 : 1, KGRP = 32 * DPL / HD, HALF = HD / 2;
    extern __shared__ __align__(16) float dsm[];
    const int warp = warp_index(), lane = threadIdx.x & 31, tid = threadIdx.x;
    float *Ks = dsm + warp * Z::WARP, *Vs = Ks + Z::K_FLOATS;
    float *qs = dsm + NW * Z::WARP, *ps = qs + Z::Q + warp * Z::P, *parts = qs + Z::Q + NW * Z::P, *one = parts + Z::PARTS;
    const int chunks = (a.G + DF_HEADS - 1) / DF_HEADS;
    const int split = blockIdx.x % n_splits, y = blockIdx.x / n_splits, kvh = y / chunks, g0 = (y % chunks) * DF_HEADS, b = blockIdx.y;
    const int rows = min(DF_HEADS, a.G - g0);
    pdl_launch_dependents();
    const int pos = a.positions[b], lo_key = first_visible_key(pos, a.window), first_page = lo_key / PAGE, last_page = pos / PAGE;
    const int per = (last_page - first_page + n_splits) / n_splits;            // pages a split
    const int p_begin = first_page + split * per, p_end = min(last_page + 1, p_begin + per);
    const int *bt = a.block_table + (size_t)b * a.table_width;
    auto load = [&](float *dst, int ld, const float *pool, int p) {
        const float *src = pool + ((size_t)bt[p] * a.KV + kvh) * PAGE * HD;
#pragma unroll 8
        for (int e = lane; e < PAGE * HD / 4; e += 32) df_cp16(dst + e / (HD / 4) * ld + e % (HD / 4) * 4, src + e * 4);
    };
    int p = p_begin + warp;
    if (p < p_end) {
        load(Ks, LDK, a.k_pool, p);
        df_commit();
        load(Vs, HD, a.v_pool, p);
        df_commit();
    }
    pdl_wait();                                // q, k and v of the new token come from the kernel in front
    const float *row = a.qkv + (size_t)b * a.ldq, *cs = a.cos_t + (size_t)pos * HALF, *sn = a.sin_t + (size_t)pos * HALF;
    for (int e = tid; e < DF_HEADS * HALF; e += NW * 32) {
        const int g = e / HALF, j = e % HALF;
        float x = 0.f, z = 0.f;
        if (g < rows) {
            const float *q = row + (size_t)(kvh * a.G + g0 + g) * HD;
            x = q[j]; z = q[j + HALF];
        }
        const float c = cs[j], s = sn[j];
        qs[g * HD + j] = x * c - z * s;
        qs[g * HD + j + HALF] = x * s + z * c;
    }
    __syncthreads();
    float acc[DF_HEADS][DPL], m[DF_HEADS], l[DF_HEADS];
#pragma unroll
    for (int g = 0; g < DF_HEADS; g++) {
        m[g] = -INFINITY; l[g] = 0.f;
#pragma unroll
        for (int d = 0; d < DPL; d++) acc[g][d] = 0.f;
    }
    const int dl = lane * DPL % HD, kg = lane * DPL / HD;                      // this lane's columns of P V, and its part of the keys
    for (; p < p_end; p += NW) {
        const int pn = p + NW, key0 = p * PAGE;
        df_wait<1>();                          // K of this page is here
        __syncwarp();
        if (p == last_page) {
            // the rotated k of the new token into the tile, and into the cache once a kv head
            const int off = pos % PAGE;
            const float *k = row + (size_t)(a.H + kvh) * HD;
            float *dst = a.k_pool + (((size_t)bt[p] * a.KV + kvh) * PAGE + off) * HD;
            for (int j = lane; j < HALF; j += 32) {
                const float x = k[j], z = k[j + HALF], c = cs[j], s = sn[j], r0 = x * c - z * s, r1 = x * s + z * c;
                Ks[off * LDK + j] = r0;
                Ks[off * LDK + j + HALF] = r1;
                if (g0 == 0) { dst[j] = r0; dst[j + HALF] = r1; }
            }
            __syncwarp();
        }
        float s[DF_HEADS][2];
#pragma unroll
        for (int g = 0; g < DF_HEADS; g++) s[g][0] = s[g][1] = 0.f;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            const float4 k0 = *(const float4 *)(Ks + lane * LDK + d), k1 = *(const float4 *)(Ks + (lane + 32) * LDK + d);
#pragma unroll
            for (int g = 0; g < DF_HEADS; g++) {
                const float4 q = *(const float4 *)(qs + g * HD + d);
                s[g][0] = fmaf(q.x, k0.x, s[g][0]); s[g][0] = fmaf(q.y, k0.y, s[g][0]); s[g][0] = fmaf(q.z, k0.z, s[g][0]); s[g][0] = fmaf(q.w, k0.w, s[g][0]);
                s[g][1] = fmaf(q.x, k1.x, s[g][1]); s[g][1] = fmaf(q.y, k1.y, s[g][1]); s[g][1] = fmaf(q.z, k1.z, s[g][1]); s[g][1] = fmaf(q.w, k1.w, s[g][1]);
            }
        }
        __syncwarp();
        if (pn < p_end) load(Ks, LDK, a.k_pool, pn);
        df_commit();
        const bool see0 = key0 + lane >= lo_key && key0 + lane <= pos, see1 = key0 + lane + 32 >= lo_key && key0 + lane + 32 <= pos;
        float corr[DF_HEADS], w0[DF_HEADS], w1[DF_HEADS];
#pragma unroll
        for (int g = 0; g < DF_HEADS; g++) {
            s[g][0] *= a.scale;
            s[g][1] *= a.scale;
            const float m_new = fmaxf(m[g], warp_max(fmaxf(see0 ? s[g][0] : -INFINITY, see1 ? s[g][1] : -INFINITY)));
            // (a page whose every score is -inf counts for nothing as long as another key has a finite one; a NaN score makes its weight NaN)
            const bool none = m_new == -INFINITY;
            const float base = none ? 0.f : m_new;
            w0[g] = see0 ? expf(s[g][0] - base) : 0.f;
            w1[g] = see1 ? expf(s[g][1] - base) : 0.f;
            corr[g] = none ? 1.f : expf(m[g] - m_new);
            l[g] = l[g] * corr[g] + warp_sum(w0[g] + w1[g]);
            m[g] = m_new;
        }
        *(float4 *)(ps + lane * DF_HEADS) = make_float4(w0[0], w0[1], w0[2], w0[3]);
        *(float4 *)(ps + (lane + 32) * DF_HEADS) = make_float4(w1[0], w1[1], w1[2], w1[3]);
        df_wait<1>();                          // V of this page is here
        __syncwarp();
        if (p == last_page) {
            const int off = pos % PAGE;
            const float *v = row + (size_t)(a.H + a.KV + kvh) * HD;
            float *dst = a.v_pool + (((size_t)bt[p] * a.KV + kvh) * PAGE + off) * HD;
            for (int j = lane; j < HD; j += 32) {
                Vs[off * HD + j] = v[j];
                if (g0 == 0) dst[j] = v[j];
            }
            __syncwarp();
        }
        float pv[DF_HEADS][DPL];
#pragma unroll
        for (int g = 0; g < DF_HEADS; g++)
#pragma unroll
            for (int d = 0; d < DPL; d++) pv[g][d] = 0.f;
        // (keys outside what the token sees are left out: zero times what a page happens to hold need not be zero)
        const int k_lo = max(0, lo_key - key0), k_hi = min(PAGE - 1, pos - key0);
#pragma unroll 4
        for (int k = k_lo + kg; k <= k_hi; k += KGRP) {
            const float4 w = *(const float4 *)(ps + k * DF_HEADS);
            const float wg[DF_HEADS] = {w.x, w.y, w.z, w.w};
            float v[DPL];
#pragma unroll
            for (int d = 0; d < DPL; d++) v[d] = Vs[k * HD + dl + d];
#pragma unroll
            for (int g = 0; g < DF_HEADS; g++)
#pragma unroll
                for (int d = 0; d < DPL; d++) pv[g][d] = fmaf(wg[g], v[d], pv[g][d]);
        }
        __syncwarp();
        if (pn < p_end) load(Vs, HD, a.v_pool, pn);
        df_commit();
#pragma unroll
        for (int g = 0; g < DF_HEADS; g++)
#pragma unroll
            for (int d = 0; d < DPL; d++) {
                if (KGRP > 1) pv[g][d] += __shfl_xor_sync(0xffffffffu, pv[g][d], HD / DPL);
                acc[g][d] = fmaf(acc[g][d], corr[g], pv[g][d]);
            }
    }
    df_wait<0>();
    // (maximum, sum, O) of every warp, then of the CTA
    float *mine = parts + warp * DF_HEADS * (HD + 2);
#pragma unroll
    for (int g = 0; g < DF_HEADS; g++) {
        if (lane == 0) { mine[g * (HD + 2)] = m[g]; mine[g * (HD + 2) + 1] = l[g]; }
        if (kg == 0)
#pragma unroll
            for (int d = 0; d < DPL; d++) mine[g * (HD + 2) + 2 + dl + d] = acc[g][d];
    }
    __syncthreads();
    // (a part whose maximum is -inf has nothing but zeros, or a NaN that reaches the result)
    auto weight = [](float x, float M) { return x == -INFINITY ? 1.f : expf(x - M); };
    auto merge = [&](const float *src, int n, int stride, int g, int d, float &M, float &L, float &O) {
        M = -INFINITY; L = 0.f; O = 0.f;
        for (int i = 0; i < n; i++) M = fmaxf(M, src[i * stride + g * (HD + 2)]);
        for (int i = 0; i < n; i++) {
            const float *x = src + i * stride + g * (HD + 2), f = weight(x[0], M);
            L = fmaf(f, x[1], L);
            O = fmaf(f, x[2 + d], O);
        }
    };
    auto store = [&](int g, int d, float M, float L, float O) {
        a.out[(size_t)b * a.ldo + (size_t)(kvh * a.G + g0 + g) * HD + d] = M == -INFINITY ? M - M : O / L;      // no finite score at all: no number
    };
    if (n_splits == 1) {
        for (int e = tid; e < rows * HD; e += NW * 32) {
            float M, L, O;
            merge(parts, NW, DF_HEADS * (HD + 2), e / HD, e % HD, M, L, O);
            store(e / HD, e % HD, M, L, O);
        }
        return;
    }
    // the CTAs of a cluster leave theirs in shared memory, and each gathers its share of the columns from all of them, in split order
    for (int e = tid; e < rows * HD; e += NW * 32) {
        const int g = e / HD, d = e % HD;
        float M, L, O;
        merge(parts, NW, DF_HEADS * (HD + 2), g, d, M, L, O);
        one[g * (HD + 2) + 2 + d] = O;
        if (d == 0) { one[g * (HD + 2)] = M; one[g * (HD + 2) + 1] = L; }
    }
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
    for (int e = split * share + tid; e < min(rows * HD, (split + 1) * share); e += NW * 32) {
        const int g = e / HD, d = e % HD;
        float x[8], M = -INFINITY, L = 0.f, O = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            x[i] = i < n_splits ? remote(i, g * (HD + 2)) : -INFINITY;
            M = fmaxf(M, x[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (i >= n_splits) break;
            const float f = weight(x[i], M);
            L = fmaf(f, remote(i, g * (HD + 2) + 1), L);
            O = fmaf(f, remote(i, g * (HD + 2) + 2 + d), O);
        }
        store(g, d, M, L, O);
    }
    // nobody leaves while another still reads its shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int HD, int NW>
static int launch_decode_f32(const DecodeF32 &a, int B, int n_splits, cudaStream_t stream) {
    static FgPerDevice configured;
    if (fg_needs_setup(configured)) {
        cudaError_t e = cudaFuncSetAttribute(attn_decode_f32_kernel<HD, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, DfSizes<HD, NW>::SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    const long long blocks = (long long)n_splits * a.KV * ((a.G + DF_HEADS - 1) / DF_HEADS);
    if (blocks > 0x7fffffff) return FG_ERR_BAD_SIZE;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks, B); cfg.blockDim = dim3(NW * 32); cfg.dynamicSmemBytes = DfSizes<HD, NW>::SMEM; cfg.stream = stream;
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
    return (int)cudaLaunchKernelEx(&cfg, attn_decode_f32_kernel<HD, NW>, a, n_splits);
}

// Splits of a sequence's pages, by the step's shape: as many CTAs as fill the GPU once (a CTA at head sizes 64 and 128 has an SM to itself).
extern "C" int fg_attention_decode_f32_splits(int B, int H, int KV, int table_width, int n_sm) {
    if (B <= 0 || KV <= 0 || H <= 0 || H % KV) return 1;
    const long long ctas = (long long)B * KV * ((H / KV + DF_HEADS - 1) / DF_HEADS);
    int s = 1;
    while (s < 8 && 2 * s * ctas <= n_sm && 2 * s <= table_width) s *= 2;
    return s;
}

// qkv: [B, ldq] float32 rows straight from the projection; positions[b] is the new token's place; n_splits 1, 2, 4 or 8.  Refuses (FG_ERR_BAD_SIZE)
// other head sizes and pages, and pools that are not 16-byte aligned; fg_rope_append and the any-size kernel take those.
extern "C" int fg_attention_decode_f32(const void *qkv, int ldq, void *out, int ldo, const int *positions, const int *block_table, int table_width,
                                       void *k_pool, void *v_pool, const float *cos_t, const float *sin_t, int B, int H, int KV, int hd, int page_size,
                                       float scale, int window, int n_splits, cudaStream_t stream) {
    if (B <= 0) return 0;
    if (page_size != PAGE || KV <= 0 || H <= 0 || H % KV || B > 65535 || (n_splits != 1 && n_splits != 2 && n_splits != 4 && n_splits != 8) ||
        (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15))
        return FG_ERR_BAD_SIZE;
    DecodeF32 a = {(const float *)qkv, ldq, (float *)out, ldo, positions, block_table, table_width, (float *)k_pool, (float *)v_pool, cos_t, sin_t, H, KV, H / KV,
                   scale, window};
    if (hd == 16) return launch_decode_f32<16, 4>(a, B, n_splits, stream);
    if (hd == 32) return launch_decode_f32<32, 4>(a, B, n_splits, stream);
    if (hd == 64) return launch_decode_f32<64, 6>(a, B, n_splits, stream);
    if (hd == 128) return launch_decode_f32<128, 3>(a, B, n_splits, stream);
    return FG_ERR_BAD_SIZE;
}
