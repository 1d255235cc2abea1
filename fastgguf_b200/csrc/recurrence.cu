// Recurrent mixers whose state decays by ONE factor per head and token: the state-space form ("duality") and the gated
// delta rule, and what stands between their projections and the recurrence.
//
// Both are one recurrence over a state S [d, dv] per head, with a token's key k and query q (size d), value v (size dv),
// decay a in (0, 1], step b and a skip weight D:
//     S <- a S;   u = b (v - [delta] S^T k);   S <- S + k u^T;   o = S^T q + D v
//   state space:  k = B_t, q = C_t, v = x_t, b = dt_t = softplus(dt + bias), a = exp(-exp(A_log) dt_t), no delta term, D per head
//   delta rule:   k, q unit vectors (q also times d^-1/2), b = sigmoid(.), a = exp(-exp(A_log) softplus(. + bias)), D = 0
// Every column of S (one value channel) runs by itself: S[:, j] only meets v[j].  So a column belongs to R neighbouring
// lanes of a warp, lane r holding rows r, r + R, ... in registers; the two sums over rows are shuffles inside those R
// lanes and nothing else crosses threads.  A block stages TC tokens' k, q, v, a and b in shared memory, walks them without
// a barrier while the next TC are being copied, and goes on.  State, decays, steps and sums are 32-bit in every engine dtype.
// A sequence's state row holds S as [head][row / R][column][row % R], so that a warp reads and writes whole lines.
//
// Around it:
//   fg_conv1d_silu / fg_conv1d_state: the short causal convolution over time per channel (weights [channels, taps], the
//     last column meets the current token), then SiLU; the last taps - 1 inputs of a sequence are part of its state row.
//   fg_decay_gates: a and b of every (token, head) from the projections' raw numbers.
//   fg_unit_heads: x / sqrt(sum(x^2) + eps) * scale per head.
//   fg_gated_group_norm: the gate and the norm behind the recurrence, in either order.
#include "common.cuh"

#define REC_THREADS 256
#define REC_RPL 16                  // rows of a column a lane holds at most
#define REC_KEEP 8                  // numbers of a group that a lane of the norms holds in registers
#define REC_TAPS 8                  // taps of a convolution that the single-token kernel takes
#define REC_TC 16                   // tokens staged at a time (fewer where a head's rows are many)

__device__ __forceinline__ float rec_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float rec_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float rec_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// ------------------------------------------------------------------ convolution
// out[m, c] = silu(bias[c] + sum_j w[c, j] * u(t - taps + 1 + j)), u = the channel's inputs of the row's sequence: rows of
// this step where there are some, else the sequence's state (its last taps - 1 inputs, oldest first; zeros at its start).
template <bool FEW>                                        // few rows: see fg_conv1d_silu
__global__ void __launch_bounds__(256)
conv1d_silu_kernel(const float *__restrict__ in, int ld, const float *__restrict__ w, const float *__restrict__ bias, int taps,
                   const float *__restrict__ state, long long state_stride, const int *__restrict__ row_seq,
                   const int *__restrict__ cu_rows, const int *__restrict__ slots, float *__restrict__ out, int ldo, int C) {
    pdl_launch_dependents_small_step(gridDim.x);
    // the weights of the thread's first channel before the wait: nothing writes them
    const int c_first = blockIdx.y * 256 + threadIdx.x;
    float w_first[4] = {0.f, 0.f, 0.f, 0.f}, b_first = 0.f;
    const bool ahead = FEW && taps <= 4;
    if (ahead && c_first < C) {
        b_first = bias ? bias[c_first] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (j < taps) w_first[j] = w[(size_t)c_first * taps + j];
    }
    pdl_wait();
    const int m = blockIdx.x;
    const int s = row_seq[m], first = cu_rows[s], i = m - first;
    const float *st = state + (size_t)slots[s] * state_stride;
    auto input = [&](int j, int c) {
        const int t = i - (taps - 1) + j;
        return t >= 0 ? in[(size_t)(first + t) * ld + c] : st[(size_t)(taps - 1 + t) * C + c];
    };
    for (int c = c_first; c < C; c += gridDim.y * 256) {
        float acc;
        if (ahead && c == c_first) {
            float u[4];
#pragma unroll
            for (int j = 0; j < 4; j++) u[j] = j < taps ? input(j, c) : 0.f;         // (asked for together)
            acc = b_first;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < taps) acc = fmaf(w_first[j], u[j], acc);
        } else {
            acc = bias ? bias[c] : 0.f;
            for (int j = 0; j < taps; j++) {
                const int t = i - (taps - 1) + j;
                const float u = t >= 0 ? in[(size_t)(first + t) * ld + c] : st[(size_t)(taps - 1 + t) * C + c];
                acc = fmaf(w[(size_t)c * taps + j], u, acc);
            }
        }
        out[(size_t)m * ldo + c] = rec_silu(acc);
    }
}

// the sequences' last taps - 1 inputs to their state rows (a kernel of its own: no row may read a state another has replaced)
__global__ void __launch_bounds__(256)
conv1d_state_kernel(const float *__restrict__ in, int ld, int taps, float *__restrict__ state, long long state_stride,
                    const int *__restrict__ cu_rows, const int *__restrict__ slots, int C) {
    pdl_wait();
    const int s = blockIdx.x, c = blockIdx.y * 256 + threadIdx.x;
    if (c >= C) return;
    const int first = cu_rows[s], n = cu_rows[s + 1] - first;
    if (n <= 0) return;
    float *st = state + (size_t)slots[s] * state_stride;
    for (int u = 0; u < taps - 1; u++) {
        const int t = n - (taps - 1) + u;               // ascending u: an old entry is read before its place is rewritten
        st[(size_t)u * C + c] = t >= 0 ? in[(size_t)(first + t) * ld + c] : st[(size_t)(u + n) * C + c];
    }
}

// One token a sequence: the output and the state's shift by one, in one kernel - a thread owns a channel of a row, and nobody else reads or
// writes that channel's inputs.  Weights, and with AHEAD the state, are fetched before the wait (see decay_step_kernel below).  8 rows of 4,352
// channels, four taps, launches behind one another: 7.3 us as two kernels, 1.4 here; 256 rows 16.8 : 9.7.
template <bool AHEAD>
__global__ void __launch_bounds__(256)
conv1d_step_kernel(const float *__restrict__ in, int ld, const float *__restrict__ w, const float *__restrict__ bias, int taps, float *state,
                   long long state_stride, const int *__restrict__ row_seq, const int *__restrict__ slots, float *__restrict__ out, int ldo, int C) {
    pdl_launch_dependents_small_step(gridDim.x);
    const int m = blockIdx.x, c = blockIdx.y * 256 + threadIdx.x;
    const bool live = c < C;
    float wc[REC_TAPS], u[REC_TAPS], acc = 0.f;
    if (live) {
        acc = bias ? bias[c] : 0.f;
#pragma unroll
        for (int j = 0; j < REC_TAPS; j++) wc[j] = j < taps ? w[(size_t)c * taps + j] : 0.f;
    }
    if (!AHEAD) pdl_wait();
    float *st = state + (size_t)slots[row_seq[m]] * state_stride + c;
#pragma unroll
    for (int j = 0; j < REC_TAPS; j++) u[j] = live && j < taps - 1 ? st[(size_t)j * C] : 0.f;
    if (AHEAD) pdl_wait();
    if (!live) return;
    const float x = in[(size_t)m * ld + c];
#pragma unroll
    for (int j = 0; j < REC_TAPS; j++)
        if (j < taps) acc = fmaf(wc[j], j < taps - 1 ? u[j] : x, acc);
    out[(size_t)m * ldo + c] = rec_silu(acc);
#pragma unroll
    for (int j = 0; j < REC_TAPS - 1; j++)
        if (j < taps - 1) st[(size_t)j * C] = j + 1 < taps - 1 ? u[j + 1] : x;
}

// ------------------------------------------------------------------ decays and steps
// mode 0: b = softplus(a_raw + dt_bias), a = exp(-exp(A_log) b)                    (one raw number a head)
// mode 1: a = exp(-exp(A_log) softplus(a_raw + dt_bias)), b = sigmoid(b_raw)
__device__ __forceinline__ void rec_gates(float a_raw, const float *b_raw, float A_log, float dt_bias, int mode, float &decay, float &step) {
    const float sp = rec_softplus(a_raw + dt_bias);
    decay = expf(-expf(A_log) * sp);
    step = mode == 0 ? sp : rec_sigmoid(*b_raw);
}
__global__ void decay_gates_kernel(const float *__restrict__ a_raw, int lda, const float *__restrict__ b_raw, int ldb,
                                   const float *__restrict__ A_log, const float *__restrict__ dt_bias, int mode,
                                   float *__restrict__ decay, float *__restrict__ step, int M, int H) {
    pdl_launch_dependents_small_step(M);
    pdl_wait();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M * H) return;
    const int m = e / H, h = e % H;
    rec_gates(a_raw[(size_t)m * lda + h], mode ? b_raw + (size_t)m * ldb + h : nullptr, A_log[h], dt_bias[h], mode, decay[e], step[e]);
}

// x[m, h, :] <- x / sqrt(sum(x^2) + eps) * scale (heads from n_scaled on: * 1), a warp a (row, head)
__global__ void __launch_bounds__(256)
unit_heads_kernel(float *__restrict__ x, int ld, int n_heads, int d, float eps, float scale_of, int n_scaled, int M) {
    pdl_launch_dependents_small_step(M);
    pdl_wait();
    const int id = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (id >= M * n_heads) return;
    float *p = x + (size_t)(id / n_heads) * ld + (size_t)(id % n_heads) * d;
    const float scale = id % n_heads < n_scaled ? scale_of : 1.0f;
    float ss = 0.f;
    if (d <= 32 * REC_KEEP) {                               // a head in the warp's registers: its loads are in flight together
        float v[REC_KEEP];
#pragma unroll
        for (int j = 0; j < REC_KEEP; j++) v[j] = lane + 32 * j < d ? p[lane + 32 * j] : 0.f;
#pragma unroll
        for (int j = 0; j < REC_KEEP; j++) ss = fmaf(v[j], v[j], ss);
        const float f = scale / sqrtf(warp_sum(ss) + eps);
#pragma unroll
        for (int j = 0; j < REC_KEEP; j++)
            if (lane + 32 * j < d) p[lane + 32 * j] = v[j] * f;
        return;
    }
    for (int i = lane; i < d; i += 32) ss = fmaf(p[i], p[i], ss);
    ss = warp_sum(ss);
    const float f = scale / sqrtf(ss + eps);
    for (int i = lane; i < d; i += 32) p[i] *= f;
}

// ------------------------------------------------------------------ the recurrence, token by token
__device__ __forceinline__ void rec_copy4(float *dst, const float *src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void rec_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void rec_wait_all_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Shared memory holds TWO sets of TC tokens: while the warps walk one, the copies of the next are in flight (cp.async, four
// bytes each, since a lane's rows r, r + R, ... of k and q are laid side by side: [token][r][row / R], rows padded with zeros
// to `stride` floats, so that a lane reads its rows as 16-byte pieces and the R lanes of a column hit different banks).
// the sum of x over the R neighbouring lanes that share a column (R a power of two)
__device__ __forceinline__ float rec_lanes_sum(float x, int R) {
    if (R > 16) x += __shfl_xor_sync(0xffffffffu, x, 16);
    if (R > 8) x += __shfl_xor_sync(0xffffffffu, x, 8);
    if (R > 4) x += __shfl_xor_sync(0xffffffffu, x, 4);
    if (R > 2) x += __shfl_xor_sync(0xffffffffu, x, 2);
    if (R > 1) x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x;
}

// NJ: 16-byte pieces of rows a lane holds (its rows padded to 4 * NJ; the padding's k and q are zero, so its state stays zero)
template <bool DELTA, int NJ>
__global__ void __launch_bounds__(REC_THREADS, 1)
decay_recurrence_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ k, int ldk, const float *__restrict__ v, int ldv,
                        const float *__restrict__ decay, const float *__restrict__ step, const float *__restrict__ skip,
                        float *__restrict__ out, int ldo, const int *__restrict__ cu_rows, const int *__restrict__ slots,
                        float *__restrict__ state, long long state_stride, int H, int Hq, int d, int dv, int R, int logR, int cols,
                        int TC, int stride) {
    extern __shared__ __align__(16) float sm[];
    pdl_wait();
    const int seq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, NT = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, n_warps = NT >> 5;
    const int row0 = cu_rows[seq], row1 = cu_rows[seq + 1];
    if (row1 <= row0) return;
    const int epl = (d + R - 1) / R;                        // rows a lane holds
    const int c0 = blockIdx.z * cols;                       // this block's first column
    const int cl = tid >> logR, r = tid & (R - 1), c = c0 + cl;
    const bool live = cl < cols && c < dv;
    const int hq = h / (H / Hq);
    const int qk_floats = TC * R * stride, set_floats = (2 * qk_floats + TC * cols + 2 * TC + 3) & ~3;      // one set: q, k, v, decays, steps
    for (int e = tid; e < 2 * set_floats; e += NT) sm[e] = 0.f;       // the padding stays zero for good
    float *Sg = state + (size_t)slots[seq] * state_stride + (size_t)h * epl * dv * R;
    float S[4 * NJ];
#pragma unroll
    for (int e = 0; e < 4 * NJ; e++) S[e] = (live && e < epl) ? Sg[((size_t)e * dv + c) * R + r] : 0.f;
    const float Dh = skip ? skip[h] : 0.f;
    __syncthreads();
    // the copies of the tokens from t0 on into set `b`: a warp a token, its lanes along the rows
    auto fetch = [&](int t0, int b) {
        const int n = min(TC, row1 - t0);
        float *qs = sm + b * set_floats, *ks = qs + qk_floats, *vs = ks + qk_floats, *as = vs + TC * cols, *bs = as + TC;
        for (int t = warp; t < n; t += n_warps) {
            const float *qg = q + (size_t)(t0 + t) * ldq + (size_t)hq * d, *kg = k + (size_t)(t0 + t) * ldk + (size_t)hq * d;
            for (int i = lane; i < d; i += 32) {
                const int at = (t * R + (i & (R - 1))) * stride + (i >> logR);
                rec_copy4(qs + at, qg + i);
                rec_copy4(ks + at, kg + i);
            }
            const float *vg = v + (size_t)(t0 + t) * ldv + (size_t)h * dv + c0;
            for (int j = lane; j < cols; j += 32)
                if (c0 + j < dv) rec_copy4(vs + t * cols + j, vg + j);
        }
        if (tid < n) {
            rec_copy4(as + tid, decay + (size_t)(t0 + tid) * H + h);
            rec_copy4(bs + tid, step + (size_t)(t0 + tid) * H + h);
        }
        rec_commit();
    };
    const bool warp_on = ((tid & ~31) >> logR) < cols;      // a warp without a column sits the walk out (whole warps only: the shuffles name every lane)
    const int tok4 = R * stride / 4;                        // 16-byte pieces between two tokens' rows
    fetch(row0, 0);
    int b = 0;
    for (int t0 = row0; t0 < row1; t0 += TC, b ^= 1) {
        const int n = min(TC, row1 - t0);
        fetch(t0 + TC, b ^ 1);                               // (an empty group behind the last tokens)
        rec_wait_all_but_one();
        __syncthreads();                                    // everybody's copies of this set have landed
        const float *qs = sm + b * set_floats, *ks = qs + qk_floats, *vs = ks + qk_floats, *as = vs + TC * cols, *bs = as + TC;
        if (warp_on) {
            const float4 *kt = (const float4 *)(ks + r * stride), *qt = (const float4 *)(qs + r * stride);
            const float *vt = vs + (cl < cols ? cl : 0);
            float *og = out + (size_t)t0 * ldo + (size_t)h * dv + c;
            // four tokens at a time: the sums over a column's R lanes that give the outputs are not part of the chain from
            // token to token, so the four of them are formed together behind the four updates (their shuffles overlap)
            for (int tb = 0; tb < n; tb += 4) {
                float o_part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (tb + u < n) {
                        const float a = as[tb + u], vj = vt[(tb + u) * cols];
                        float4 k4[NJ];
                        float d0 = 0.f, d1 = 0.f;
#pragma unroll
                        for (int j = 0; j < NJ; j++) {
                            k4[j] = kt[j];
                            S[4 * j] *= a; S[4 * j + 1] *= a; S[4 * j + 2] *= a; S[4 * j + 3] *= a;
                            if (DELTA) {
                                d0 = fmaf(S[4 * j], k4[j].x, d0); d1 = fmaf(S[4 * j + 1], k4[j].y, d1);
                                d0 = fmaf(S[4 * j + 2], k4[j].z, d0); d1 = fmaf(S[4 * j + 3], k4[j].w, d1);
                            }
                        }
                        const float dot = DELTA ? rec_lanes_sum(d0 + d1, R) : 0.f;
                        const float w = bs[tb + u] * (vj - dot);
                        float o0 = 0.f, o1 = 0.f;
#pragma unroll
                        for (int j = 0; j < NJ; j++) {
                            const float4 q4 = qt[j];
                            S[4 * j] = fmaf(k4[j].x, w, S[4 * j]); S[4 * j + 1] = fmaf(k4[j].y, w, S[4 * j + 1]);
                            S[4 * j + 2] = fmaf(k4[j].z, w, S[4 * j + 2]); S[4 * j + 3] = fmaf(k4[j].w, w, S[4 * j + 3]);
                            o0 = fmaf(S[4 * j], q4.x, o0); o1 = fmaf(S[4 * j + 1], q4.y, o1);
                            o0 = fmaf(S[4 * j + 2], q4.z, o0); o1 = fmaf(S[4 * j + 3], q4.w, o1);
                        }
                        o_part[u] = o0 + o1;
                    }
                    kt += tok4; qt += tok4;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) o_part[u] = rec_lanes_sum(o_part[u], R);
                if (r == 0 && live) {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (tb + u < n) og[(size_t)(tb + u) * ldo] = fmaf(Dh, vt[(tb + u) * cols], o_part[u]);
                }
            }
        }
        __syncthreads();                                    // this set is free for the copies of the tokens after the next
    }
    if (live)
#pragma unroll
        for (int e = 0; e < 4 * NJ; e++)
            if (e < epl) Sg[((size_t)e * dv + c) * R + r] = S[e];
}

// The same for one token a sequence (a decode step): nothing to stage, so a lane reads its rows of k and q from the caches, the gates are computed
// where they are used, and the state is in flight before the wait on the kernel in front (AHEAD: state rows are written by this entry's kernels
// alone, once a step, and slots by the copy that opens a step, see common.cuh).  Lanes, rows and order of additions are those of the kernel above.
// Bound by memory: 2 x 1 MB of state a sequence, 2.6 us for 8 and 21 for 64.  Gates and recurrence as two kernels : this one, launches behind one another
// (us): 32 heads of 128 x 64, 8 sequences 12.1 : 4.9, 64 sequences 83 : 34, 1 sequence 4.6 : 2.3; the delta rule at 16 heads of 128 x 128, 8 sequences
// 12.9 : 5.2, 256 sequences 351 : 140.  With conv1d_step_kernel and the norms of q and k in one launch a step with two layers of each went from 712 to 644 us.
#define STEP_THREADS 128
template <bool DELTA, int NJ, bool AHEAD>
__global__ void __launch_bounds__(STEP_THREADS)
decay_step_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ k, int ldk, const float *__restrict__ v, int ldv,
                  const float *__restrict__ a_raw, int lda, const float *__restrict__ b_raw, int ldb, const float *__restrict__ A_log,
                  const float *__restrict__ dt_bias, const float *__restrict__ skip, float *__restrict__ out, int ldo,
                  const int *__restrict__ cu_rows, const int *__restrict__ slots, float *state, long long state_stride, int H, int Hq, int d,
                  int dv, int R, int logR) {
    pdl_launch_dependents_small_step(gridDim.x);
    const int seq = blockIdx.x, h = blockIdx.y, at = blockIdx.z * STEP_THREADS + threadIdx.x;
    const int epl = (d + R - 1) / R, c = at >> logR, r = at & (R - 1), hq = h / (H / Hq);
    const bool live = c < dv;
    if (!AHEAD) pdl_wait();
    float *Sg = state + (size_t)slots[seq] * state_stride + (size_t)h * epl * dv * R + (size_t)c * R + r;
    const size_t next = (size_t)dv * R;
    float S[4 * NJ];
#pragma unroll
    for (int e = 0; e < 4 * NJ; e++) S[e] = live && e < epl ? Sg[e * next] : 0.f;
    const float Dh = skip ? skip[h] : 0.f, al = A_log[h], bias = dt_bias[h];
    if (AHEAD) pdl_wait();
    const int row = cu_rows[seq];
    if (cu_rows[seq + 1] <= row) return;
    const float *kg = k + (size_t)row * ldk + (size_t)hq * d, *qg = q + (size_t)row * ldq + (size_t)hq * d;
    float kk[4 * NJ], qq[4 * NJ];
#pragma unroll
    for (int e = 0; e < 4 * NJ; e++) {
        const int i = (e << logR) + r;
        kk[e] = i < d ? kg[i] : 0.f;
        qq[e] = i < d ? qg[i] : 0.f;
    }
    const float vj = live ? v[(size_t)row * ldv + (size_t)h * dv + c] : 0.f;
    float a, b;
    rec_gates(a_raw[(size_t)row * lda + h], DELTA ? b_raw + (size_t)row * ldb + h : nullptr, al, bias, DELTA, a, b);
    float d0 = 0.f, d1 = 0.f;
#pragma unroll
    for (int e = 0; e < 4 * NJ; e += 2) {
        S[e] *= a; S[e + 1] *= a;
        if (DELTA) { d0 = fmaf(S[e], kk[e], d0); d1 = fmaf(S[e + 1], kk[e + 1], d1); }
    }
    const float w = b * (vj - (DELTA ? rec_lanes_sum(d0 + d1, R) : 0.f));
    float o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int e = 0; e < 4 * NJ; e += 2) {
        S[e] = fmaf(kk[e], w, S[e]); S[e + 1] = fmaf(kk[e + 1], w, S[e + 1]);
        o0 = fmaf(S[e], qq[e], o0); o1 = fmaf(S[e + 1], qq[e + 1], o1);
    }
    const float o = rec_lanes_sum(o0 + o1, R);
    if (!live) return;
    if (r == 0) out[(size_t)row * ldo + (size_t)h * dv + c] = fmaf(Dh, vj, o);
#pragma unroll
    for (int e = 0; e < 4 * NJ; e++)
        if (e < epl) Sg[e * next] = S[e];
}

// ------------------------------------------------------------------ gate and norm behind the recurrence
// gate_first: t = y * silu(g), out = t / rms_group(t) * w[c]                         (groups of `group` neighbouring channels)
// else:       out = y / rms_group(y) * w[c % w_period] * silu(g)
// sigmoid_gate: sigmoid(g) where silu(g) stands
__device__ __forceinline__ float rec_gate(float z, int sigmoid_gate) { return (sigmoid_gate ? 1.0f : z) / (1.0f + expf(-z)); }
template <typename TO, bool FEW>
__global__ void __launch_bounds__(256)
gated_group_norm_kernel(const float *__restrict__ y, int ldy, const float *__restrict__ g, int ldg, const float *__restrict__ w,
                        int w_period, TO *__restrict__ out, int ldo, int C, int group, float eps, int gate_first,
                        int sigmoid_gate) {
    __shared__ float scratch[32];
    pdl_launch_dependents_small_step(gridDim.x);
    pdl_wait();
    const int m = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float *yr = y + (size_t)m * ldy, *gr = g + (size_t)m * ldg;
    TO *orow = out + (size_t)m * ldo;
    const bool whole = w_period >= C, by_group = w_period == group;
    // Few rows: a group that fits the registers of its threads (the block, or a warp for narrow ones) is read once, all of it in
    // flight together.  In a step, where its rows come from memory, 8 rows of 2,048 9.7 -> 6.2 us; the sums are those of the loops below.  Alone,
    // with everything in L2 (registers against loops, us): one group of 2,048 3.4 : 4.6 up to 64 rows, 3.7 : 4.8 at 256, 5.3 : 5.3 at 512, 33 : 34 at
    // 4,925; groups of 128 of 2,048 5.5 : 4.3 up to 96 rows, 9.0 : 4.9 at 512, 60 : 33 at 4,925.  Narrow groups' loops would win alone, but not in
    // a step (Saluzen's decode case 35.09 ms this way, 35.18 with loops for narrow groups).
    const bool wide = group >= 1024;
    const int step = wide ? 256 : 32, lane0 = wide ? (int)threadIdx.x : lane;
    if (FEW && group <= step * REC_KEEP) {
        const int first = wide ? blockIdx.y : blockIdx.y * 8 + warp, stride = wide ? gridDim.y : gridDim.y * 8;
        for (int grp = first; grp * group < C; grp += stride) {
            const int b0 = grp * group;
            float t[REC_KEEP], sg[REC_KEEP], wc[REC_KEEP], ss = 0.f;
#pragma unroll
            for (int j = 0; j < REC_KEEP; j++) {
                const int i = lane0 + step * j, c = b0 + i;
                const bool in = i < group && c < C;
                t[j] = in ? yr[c] : 0.f;
                sg[j] = in ? gr[c] : 0.f;
                wc[j] = in ? w[whole ? c : (by_group ? i : c % w_period)] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < REC_KEEP; j++) {
                sg[j] = rec_gate(sg[j], sigmoid_gate);
                if (gate_first) t[j] *= sg[j];
                ss = fmaf(t[j], t[j], ss);
            }
            const float inv = 1.0f / sqrtf((wide ? block_sum(ss, scratch) : warp_sum(ss)) / (float)group + eps);
#pragma unroll
            for (int j = 0; j < REC_KEEP; j++) {
                const int i = lane0 + step * j, c = b0 + i;
                if (i < group && c < C) orow[c] = from_f32<TO>(gate_first ? t[j] * inv * wc[j] : t[j] * inv * wc[j] * sg[j]);
            }
        }
        return;
    }
    if (group >= 1024) {
        // few wide groups: the whole block takes a group (fixed reduction order: lanes, then warps in order)
        for (int b0 = blockIdx.y * group; b0 < C; b0 += gridDim.y * group) {
            float ss = 0.f;
            for (int i = threadIdx.x; i < group; i += 256) {
                const float t = gate_first ? yr[b0 + i] * rec_gate(gr[b0 + i], sigmoid_gate) : yr[b0 + i];
                ss = fmaf(t, t, ss);
            }
            const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)group + eps);
            for (int i = threadIdx.x; i < group; i += 256) {
                const int c = b0 + i;
                const float sg = rec_gate(gr[c], sigmoid_gate);
                const float wc = w[whole ? c : (by_group ? i : c % w_period)];        // (no division where the weight spans the row or a group)
                orow[c] = from_f32<TO>(gate_first ? yr[c] * sg * inv * wc : yr[c] * inv * wc * sg);
            }
        }
        return;
    }
    for (int grp = blockIdx.y * 8 + warp; grp * group < C; grp += gridDim.y * 8) {
        const int b0 = grp * group;
        float ss = 0.f;
        for (int i = lane; i < group; i += 32) {
            const float t = gate_first ? yr[b0 + i] * rec_gate(gr[b0 + i], sigmoid_gate) : yr[b0 + i];
            ss = fmaf(t, t, ss);
        }
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / (float)group + eps);
        for (int i = lane; i < group; i += 32) {
            const int c = b0 + i;
            const float sg = rec_gate(gr[c], sigmoid_gate);
            const float wc = w[whole ? c : (by_group ? i : c % w_period)];        // (no division where the weight spans the row or a group)
                orow[c] = from_f32<TO>(gate_first ? yr[c] * sg * inv * wc : yr[c] * inv * wc * sg);
        }
    }
}

// ------------------------------------------------------------------ launchers
extern "C" int fg_conv1d_silu(const float *in, int ld, const float *w, const float *bias, int taps, const float *state,
                              long long state_stride, const int *row_seq, const int *cu_rows, const int *slots, float *out, int ldo,
                              int M, int C, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (C <= 0 || taps <= 0 || (taps > 1 && !state)) return FG_ERR_BAD_SIZE;
    // With few rows latency counts: the weights come before the wait on the preceding kernel and a channel's inputs together.  That pays in
    // a step, where the weights come from memory (8 rows of 4,096 channels 10.3 -> 7.3 us); alone, with everything in L2, the plain form is as
    // fast (8 rows 4.1 us against 5.1, 64 rows 4.6 against 5.5) and leaves the other behind as the rows grow (256 rows 8.2 against 10.7, 4,925 rows
    // 128 against 297), so the line lies where a step stops being a decode step.
    return fg_launch(M <= 64 ? conv1d_silu_kernel<true> : conv1d_silu_kernel<false>, dim3(M, (C + 1023) / 1024), dim3(256), 0, stream, in, ld, w, bias,
                     taps, state, state_stride, row_seq, cu_rows, slots, out, ldo, C);
}

extern "C" int fg_conv1d_state(const float *in, int ld, int taps, float *state, long long state_stride, const int *cu_rows,
                               const int *slots, int n_seq, int C, cudaStream_t stream) {
    if (n_seq <= 0 || taps <= 1) return 0;
    if (C <= 0) return FG_ERR_BAD_SIZE;
    return fg_launch(conv1d_state_kernel, dim3(n_seq, (C + 255) / 256), dim3(256), 0, stream, in, ld, taps, state, state_stride, cu_rows,
                              slots, C);
}

extern "C" int fg_decay_gates(const float *a_raw, int lda, const float *b_raw, int ldb, const float *A_log, const float *dt_bias,
                              int mode, float *decay, float *step, int M, int H, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (H <= 0 || (mode != 0 && mode != 1) || (mode == 1 && !b_raw)) return FG_ERR_BAD_SIZE;
    return fg_launch(decay_gates_kernel, dim3((M * H + 255) / 256), dim3(256), 0, stream, a_raw, lda, b_raw, ldb, A_log, dt_bias, mode,
                              decay, step, M, H);
}

// heads of two neighbouring projections in one launch: the first n_scaled take the scale
extern "C" int fg_unit_heads_pair(float *x, int ld, int n_heads, int d, float eps, float scale, int n_scaled, int M, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (n_heads <= 0 || d <= 0) return FG_ERR_BAD_SIZE;
    return fg_launch(unit_heads_kernel, dim3((M * n_heads + 7) / 8), dim3(256), 0, stream, x, ld, n_heads, d, eps, scale, n_scaled, M);
}
extern "C" int fg_unit_heads(float *x, int ld, int n_heads, int d, float eps, float scale, int M, cudaStream_t stream) {
    return fg_unit_heads_pair(x, ld, n_heads, d, eps, scale, n_heads, M, stream);
}

// lanes that share a column of the state: the smallest power of two that leaves a lane at most REC_RPL rows
extern "C" int fg_decay_recurrence_lanes(int d) {
    int R = 1;
    while (R < 32 && (d + R - 1) / R > REC_RPL) R *= 2;
    return (d + R - 1) / R > REC_RPL ? 0 : R;
}
// floats of a sequence's state: [H][rows a lane][dv][R]
extern "C" long long fg_decay_recurrence_state_floats(int H, int d, int dv) {
    const int R = fg_decay_recurrence_lanes(d);
    return R ? (long long)H * ((d + R - 1) / R) * dv * R : -1;
}

extern "C" int fg_decay_recurrence(const float *q, int ldq, const float *k, int ldk, const float *v, int ldv, const float *decay,
                                   const float *step, const float *skip, float *out, int ldo, const int *cu_rows, const int *slots,
                                   float *state, long long state_stride, int n_seq, int H, int Hq, int d, int dv, int delta,
                                   cudaStream_t stream) {
    if (n_seq <= 0) return 0;
    const int R = fg_decay_recurrence_lanes(d);
    if (!R || H <= 0 || Hq <= 0 || H % Hq || dv <= 0 || H > 65535) return FG_ERR_BAD_SIZE;
    // Blocks of 256 threads where there are many (sequence, head) pairs; fewer threads a block - down to two warps - where the
    // blocks would not fill the GPU otherwise: a token's work in a warp is a chain of dependent instructions, and warps that
    // share a scheduler lengthen every token's turn.
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    int threads = REC_THREADS;
    while (threads > 64 && (long long)n_seq * H * ((dv + threads / R - 1) / (threads / R)) < 2LL * n_sm && threads / 2 >= R) threads /= 2;
    const int per_block = threads / R, cols = per_block < dv ? per_block : dv, tiles = (dv + cols - 1) / cols;
    int logR = 0;
    while ((1 << logR) < R) logR++;
    const int epl = (d + R - 1) / R, stride = (epl + 3) / 4 * 4 + 4;
    // two sets of TC tokens in shared memory; fewer tokens a set where a head is large
    int TC = REC_TC;
    auto bytes = [&](int tc) { return (size_t)2 * ((2 * tc * R * stride + tc * cols + 2 * tc + 3) & ~3) * sizeof(float); };
    while (TC > 2 && bytes(TC) > 96 * 1024) TC /= 2;
    const size_t smem = bytes(TC);
    if (smem > 96 * 1024) return FG_ERR_BAD_SIZE;
    dim3 grid(n_seq, H, tiles);
    const int NJ = (epl + 3) / 4;
#define REC_LAUNCH(DELTA, NJ_)                                                                                                            \
    do {                                                                                                                                  \
        static FgPerDevice setup;                                                                                                         \
        if (fg_needs_setup(setup)) cudaFuncSetAttribute(decay_recurrence_kernel<DELTA, NJ_>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024); \
        return fg_launch(decay_recurrence_kernel<DELTA, NJ_>, grid, dim3(threads), smem, stream, q, ldq, k, ldk, v, ldv, decay, step, skip, out, \
                                  ldo, cu_rows, slots, state, state_stride, H, Hq, d, dv, R, logR, cols, TC, stride);                      \
    } while (0)
    if (delta) {
        if (NJ == 1) REC_LAUNCH(true, 1);
        if (NJ == 2) REC_LAUNCH(true, 2);
        if (NJ == 3) REC_LAUNCH(true, 3);
        REC_LAUNCH(true, 4);
    }
    if (NJ == 1) REC_LAUNCH(false, 1);
    if (NJ == 2) REC_LAUNCH(false, 2);
    if (NJ == 3) REC_LAUNCH(false, 3);
    REC_LAUNCH(false, 4);
#undef REC_LAUNCH
}

// One token a sequence, gates included (raw numbers as for fg_decay_gates, mode 0 without the delta term, 1 with it).  early: the state is
// fetched before the wait on the kernel in front, which must not have written it (see decay_step_kernel).
extern "C" int fg_decay_recurrence_step(const float *q, int ldq, const float *k, int ldk, const float *v, int ldv, const float *a_raw, int lda,
                                        const float *b_raw, int ldb, const float *A_log, const float *dt_bias, const float *skip, float *out, int ldo,
                                        const int *cu_rows, const int *slots, float *state, long long state_stride, int n_seq, int H, int Hq, int d,
                                        int dv, int delta, int early, cudaStream_t stream) {
    if (n_seq <= 0) return 0;
    const int R = fg_decay_recurrence_lanes(d);
    if (!R || H <= 0 || Hq <= 0 || H % Hq || dv <= 0 || H > 65535 || (delta && !b_raw)) return FG_ERR_BAD_SIZE;
    int logR = 0;
    while ((1 << logR) < R) logR++;
    const long long tiles = ((long long)dv * R + STEP_THREADS - 1) / STEP_THREADS;
    if (tiles > 65535) return FG_ERR_BAD_SIZE;
    const dim3 grid(n_seq, H, (unsigned)tiles);
    const int NJ = ((d + R - 1) / R + 3) / 4;
#define STEP_RUN(DELTA, NJ_, AHEAD) fg_launch(decay_step_kernel<DELTA, NJ_, AHEAD>, grid, dim3(STEP_THREADS), 0, stream, q, ldq, k, ldk, v, ldv, a_raw, lda, b_raw, \
                                              ldb, A_log, dt_bias, skip, out, ldo, cu_rows, slots, state, state_stride, H, Hq, d, dv, R, logR)
#define STEP_NJ(NJ_) do { \
        if (delta) return early ? STEP_RUN(true, NJ_, true) : STEP_RUN(true, NJ_, false); \
        return early ? STEP_RUN(false, NJ_, true) : STEP_RUN(false, NJ_, false); } while (0)
    if (NJ == 1) STEP_NJ(1);
    if (NJ == 2) STEP_NJ(2);
    if (NJ == 3) STEP_NJ(3);
    STEP_NJ(4);
#undef STEP_NJ
#undef STEP_RUN
}

// One token a sequence: fg_conv1d_silu and fg_conv1d_state in one (early: as above).  FG_ERR_BAD_SIZE beyond eight taps.
extern "C" int fg_conv1d_step(const float *in, int ld, const float *w, const float *bias, int taps, float *state, long long state_stride,
                              const int *row_seq, const int *slots, float *out, int ldo, int M, int C, int early, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (C <= 0 || taps <= 0 || taps > REC_TAPS || (taps > 1 && !state)) return FG_ERR_BAD_SIZE;
    return fg_launch(early ? conv1d_step_kernel<true> : conv1d_step_kernel<false>, dim3(M, (C + 255) / 256), dim3(256), 0, stream, in, ld, w, bias, taps, state,
                     state_stride, row_seq, slots, out, ldo, C);
}

extern "C" int fg_gated_group_norm(const float *y, int ldy, const float *g, int ldg, const float *w, int w_period, void *out,
                                   int out_dtype, int ldo, int M, int C, int group, float eps, int gate_first, int sigmoid_gate,
                                   cudaStream_t stream) {
    if (M <= 0) return 0;
    if (C <= 0 || group <= 0 || C % group || w_period <= 0) return FG_ERR_BAD_SIZE;
    const int groups = C / group;
    dim3 grid(M, group >= 1024 ? (groups < 4 ? groups : 4) : groups >= 64 ? 4 : 1);
#define GGN_RUN(TO, FEW) fg_launch(gated_group_norm_kernel<TO, FEW>, grid, dim3(256), 0, stream, y, ldy, g, ldg, w, w_period, (TO *)out, ldo, C, group, \
                                   eps, gate_first, sigmoid_gate)
    if (out_dtype == FG_F32) return M <= 64 ? GGN_RUN(float, true) : GGN_RUN(float, false);
    if (out_dtype == FG_BF16) return M <= 64 ? GGN_RUN(bf16, true) : GGN_RUN(bf16, false);
#undef GGN_RUN
    return FG_ERR_BAD_DTYPE;
}
