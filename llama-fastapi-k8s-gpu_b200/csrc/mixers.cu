// Token mixers and norms of the layer-list models, over a ragged step (layered.h): post-sum layer norm with RMS-normed
// branches, sliding-window attention with a kept prefix over the paged cache (query/key norm, partial interleaved
// rotary with blended frequencies, values = un-normalised keys), selective scan (causal depthwise convolution +
// diagonal state recurrence), and the mLSTM matrix memory. Softmax, norms, gates, decays and all recurrent state are
// 32-bit; only the cache pages may be bf16. Every recurrence walks a segment's tokens in order from the state its
// slot holds, so a sequence cut into portions gives the same numbers as the whole.
#include "kernels.h"
#include "layered.h"
#include "softmax_tc.h"
#include "ptx.cuh"
#include "quant_blocks.cuh"

#include <stdlib.h>

#include <algorithm>

namespace b2 {

__device__ __forceinline__ float block_sum(float v, float* red) {      // all threads get the sum; red: >= 33 floats
    v = warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nw ? red[lane] : 0.f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

__device__ __forceinline__ void cp_async_4(float* smem_dst, const float* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float log_sigmoid_f(float z) { return -softplus_f(-z); }

// z / (1 + exp(-z)) without a branch, so that it can run between other work
__device__ __forceinline__ float silu_inline(float z) { return over_one_plus_exp(z, -z); }

// ---------------------------------------------------------------- embedding, gather
// Entries i .. i + N - 1 of token t's row (N: 1, or 4 from a multiple of 4 in rows on 16-byte boundaries): the table's, times the scale, plus its pair's, plus
// its position's turns
template <int N>
__device__ __forceinline__ void embed_at(const EmbedDev& d, int W, int t, int i, float (&v)[N]) {
    auto read = [&](const void* table, int type, size_t row, float (&to)[N]) {
        if constexpr (N == 4) {
            if (type == T_BF16) {
                const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(table) + row * W + i);
                const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&u.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
                to[0] = __low2float(lo); to[1] = __high2float(lo); to[2] = __low2float(hi); to[3] = __high2float(hi);
            } else {
                const float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(table) + row * W + i);
                to[0] = f.x; to[1] = f.y; to[2] = f.z; to[3] = f.w;
            }
        } else to[0] = type == T_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(table)[row * W + i]) : reinterpret_cast<const float*>(table)[row * W + i];
    };
    const int cur = d.tok[t];
    read(d.table, d.w_type, (size_t)cur, v);
#pragma unroll
    for (int k = 0; k < N; k++) v[k] *= d.scale;
    if (d.bg.table) {
        const int prev = d.tok_prev[t];
        float w[N];
        read(d.bg.table, d.bg.w_type, prev < 0 ? d.bg.buckets : (size_t)(((long long)prev * d.bg.mul_prev + (long long)cur * d.bg.mul_cur) % d.bg.buckets), w);
#pragma unroll
        for (int k = 0; k < N; k++) v[k] += w[k];
    }
    if (d.turns) {                               // whole turns are dropped in double precision, so far positions lose nothing
        const double pos = (double)d.tok_pos[t];
#pragma unroll
        for (int k = 0; k < N; k += 2) {
            const double a = pos * d.turns[(i + k) >> 1];
            const float half_turns = (float)(2.0 * (a - rint(a)));
            if constexpr (N == 1) v[0] += i & 1 ? cospif(half_turns) : sinpif(half_turns);
            else { v[k] += sinpif(half_turns); v[k + 1] += cospif(half_turns); }
        }
    }
}
static bool embed_wide(const EmbedDev& d, int W) {
    return W % 4 == 0 && ((reinterpret_cast<uintptr_t>(d.table) | reinterpret_cast<uintptr_t>(d.bg.table)) & 15) == 0;
}
// N entries a thread, 256 threads a CTA. (2048 rows of 4096: one entry of two bytes a thread 20 us, 11 here. 2048 rows of 2048 with turns: both functions of a turn
// in every warp 19 us; as part of the first norms below, embedding, experts' tables and norms take 25 us instead of 43, a chat's 7 instead of 10.)
template <int N>
__global__ void __launch_bounds__(256) embed_ragged_kernel(const EmbedDev d, int W, float* __restrict__ x, EmbedCopies c) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x, i = (blockIdx.y * 256 + threadIdx.x) * N;
    if (i >= W) return;
    float v[N];
    embed_at(d, W, t, i, v);
    auto put = [&](float* to) {
        if constexpr (N == 4) *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
        else *to = v[0];
    };
    put(x + (size_t)t * W + i);
    for (int k = 0; k < 2; k++) if (c.copy[k]) put(c.copy[k] + (size_t)t * c.ld_copy + i);
}
cudaError_t embed_ragged_launch(const EmbedDev& d, int W, int T, float* x, const EmbedCopies& c, cudaStream_t s) {
    if (d.bg.table && !d.tok_prev) return cudaErrorInvalidValue;
    const uintptr_t out = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(c.copy[0]) | reinterpret_cast<uintptr_t>(c.copy[1]);
    if (embed_wide(d, W) && c.ld_copy % 4 == 0 && (out & 15) == 0) return launch_chain(embed_ragged_kernel<4>, dim3(T, (W + 1023) / 1024), dim3(256), 0, s, d, W, x, c);
    return launch_chain(embed_ragged_kernel<1>, dim3(T, (W + 255) / 256), dim3(256), 0, s, d, W, x, c);
}

__global__ void gather_rows_kernel(const float* __restrict__ x, int W, const int* __restrict__ rows, float* __restrict__ y) {
    griddep_launch();
    griddep_wait();
    const float* src = x + (size_t)rows[blockIdx.x] * W;
    for (int i = threadIdx.x; i < W; i += blockDim.x) y[(size_t)blockIdx.x * W + i] = src[i];
}
cudaError_t gather_rows_launch(const float* x, int W, const int* rows, int n, float* y, cudaStream_t s) {
    return launch_chain(gather_rows_kernel, dim3(n), dim3(128), 0, s, x, W, rows, y);
}

__device__ __forceinline__ void store_bf16x4(__nv_bfloat16* to, const float4& v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// ---------------------------------------------------------------- norms
// one CTA per token; the row lives in shared memory between the passes (mean, then squared deviations)
__global__ void __launch_bounds__(256) postsum_norm_kernel(float* __restrict__ x, const float* __restrict__ a, const float* __restrict__ wa,
                                                           const float* __restrict__ b, const float* __restrict__ wb,
                                                           const float* __restrict__ w, float alpha, float eps, int W) {
    griddep_launch();
    griddep_wait();
    extern __shared__ float row[];
    __shared__ float red[33];
    const size_t base = (size_t)blockIdx.x * W;
    float ra = 1.f, rb = 1.f;
    if (b) {
        float sa = 0.f, sb = 0.f;
        for (int i = threadIdx.x; i < W; i += blockDim.x) { const float u = a[base + i], v = b[base + i]; sa += u * u; sb += v * v; }
        sa = block_sum(sa, red); sb = block_sum(sb, red);
        ra = 1.f / sqrtf(sa / (float)W + eps); rb = 1.f / sqrtf(sb / (float)W + eps);
    }
    float sum = 0.f;
    for (int i = threadIdx.x; i < W; i += blockDim.x) {
        float yv = b ? 0.5f * (a[base + i] * ra * wa[i] + b[base + i] * rb * wb[i]) : (a ? a[base + i] : 0.f);
        const float v = alpha * x[base + i] + yv;
        row[i] = v;
        sum += v;
    }
    const float mean = block_sum(sum, red) / (float)W;
    float sq = 0.f;
    for (int i = threadIdx.x; i < W; i += blockDim.x) { const float dlt = row[i] - mean; sq += dlt * dlt; }
    const float rstd = 1.f / sqrtf(block_sum(sq, red) / (float)W + eps);
    for (int i = threadIdx.x; i < W; i += blockDim.x) x[base + i] = (row[i] - mean) * rstd * w[i];
}
// The same for rows of at most 4096 entries on 16-byte boundaries: a thread keeps its entries (NV times four) in registers, all of them read at
// once. Bound by memory: 134 MB for 2048 rows of 4096 with two branches, 52 us with
// the row in shared memory and single reads, 39 here; with one branch 34 and 25.
template <int NV>
__global__ void __launch_bounds__(256) postsum_norm_vec_kernel(PostsumArgs p, int W) {
    griddep_launch();
    griddep_wait();
    __shared__ float red[33];
    const size_t base = (size_t)blockIdx.x * W;
    auto get = [&](const float* from, int k) {
        const int i = (k * 256 + threadIdx.x) * 4;
        return i < W ? *reinterpret_cast<const float4*>(from + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 v[NV], a[NV], b[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k] = get(p.x + base, k);
        a[k] = p.a ? get(p.a + base, k) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.b) b[k] = get(p.b + base, k);
    }
    auto square = [](const float4& u) { return u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w; };
    if (p.b) {
        float sa = 0.f, sb = 0.f;
#pragma unroll
        for (int k = 0; k < NV; k++) { sa += square(a[k]); sb += square(b[k]); }
        sa = block_sum(sa, red); sb = block_sum(sb, red);
        const float ra = 0.5f / sqrtf(sa / (float)W + p.eps), rb = 0.5f / sqrtf(sb / (float)W + p.eps);
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const float4 wa = get(p.wa, k), wb = get(p.wb, k);
            a[k].x = a[k].x * ra * wa.x + b[k].x * rb * wb.x; a[k].y = a[k].y * ra * wa.y + b[k].y * rb * wb.y;
            a[k].z = a[k].z * ra * wa.z + b[k].z * rb * wb.z; a[k].w = a[k].w * ra * wa.w + b[k].w * rb * wb.w;
        }
    }
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k].x = fmaf(p.alpha, v[k].x, a[k].x); v[k].y = fmaf(p.alpha, v[k].y, a[k].y);
        v[k].z = fmaf(p.alpha, v[k].z, a[k].z); v[k].w = fmaf(p.alpha, v[k].w, a[k].w);
        sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
    }
    const float mean = block_sum(sum, red) / (float)W;
    float sq = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k].x -= mean; v[k].y -= mean; v[k].z -= mean; v[k].w -= mean;
        if ((k * 256 + threadIdx.x) * 4 < W) sq += square(v[k]);
    }
    const float rstd = 1.f / sqrtf(block_sum(sq, red) / (float)W + p.eps);
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const int i = (k * 256 + threadIdx.x) * 4;
        if (i >= W) break;
        const float4 w = get(p.w, k), y = make_float4(v[k].x * rstd * w.x, v[k].y * rstd * w.y, v[k].z * rstd * w.z, v[k].w * rstd * w.w);
        *reinterpret_cast<float4*>(p.x + base + i) = y;
        if (p.x_rounded) store_bf16x4(p.x_rounded + base + i, y);
    }
}
bool postsum_leaves_rounded(const PostsumArgs& p, int W) {
    const float* const all[] = {p.x, p.a, p.wa, p.b, p.wb, p.w};
    uintptr_t at = 0;
    for (const float* q : all) at |= reinterpret_cast<uintptr_t>(q);
    return W % 4 == 0 && W <= 4096 && (at & 15) == 0;
}
cudaError_t postsum_norm_launch(const PostsumArgs& p, int W, int T, cudaStream_t s) {
    if (postsum_leaves_rounded(p, W)) {
        if (W <= 1024) return launch_chain(postsum_norm_vec_kernel<1>, dim3(T), dim3(256), 0, s, p, W);
        if (W <= 2048) return launch_chain(postsum_norm_vec_kernel<2>, dim3(T), dim3(256), 0, s, p, W);
        return launch_chain(postsum_norm_vec_kernel<4>, dim3(T), dim3(256), 0, s, p, W);
    }
    if (p.x_rounded) return cudaErrorInvalidValue;
    return launch_chain(postsum_norm_kernel, dim3(T), dim3(256), (size_t)W * 4, s, p.x, p.a, p.wa, p.b, p.wb, p.w, p.alpha, p.eps, W);
}

// pre-norm blocks: the pending branch output joins the 32-bit residual stream, and the next sublayer's input is made in the same pass
__global__ void __launch_bounds__(256) resid_rms_norm_kernel(float* __restrict__ x, const float* __restrict__ add, float mult,
                                                             const float* __restrict__ w, float w_offset, float out_scale, float eps, int W,
                                                             float* __restrict__ y) {
    griddep_launch();
    griddep_wait();
    extern __shared__ float row[];
    __shared__ float red[33];
    const size_t base = (size_t)blockIdx.x * W;
    float ss = 0.f;
    for (int i = threadIdx.x; i < W; i += blockDim.x) {
        float v = x[base + i];
        if (add) { v = fmaf(mult, add[base + i], v); x[base + i] = v; }
        row[i] = v;
        ss = fmaf(v, v, ss);
    }
    if (!y) return;
    const float rinv = 1.f / sqrtf(block_sum(ss, red) / (float)W + eps);
    for (int i = threadIdx.x; i < W; i += blockDim.x) y[base + i] = row[i] * rinv * (w_offset + w[i]) * out_scale;
}
cudaError_t resid_rms_norm_launch(float* x, const float* add, float mult, const float* w, float w_offset, float out_scale,
                                  float eps, int W, int T, float* y, cudaStream_t s) {
    return launch_chain(resid_rms_norm_kernel, dim3(T), dim3(256), (size_t)W * 4, s, x, add, mult, w, w_offset, out_scale, eps, W, y);
}

// Norm of rows rows[0], rows[1], .. of x. A thread keeps its entries of rows up to 256 LN_U in registers, read at once; longer rows are
// read again for each pass.
constexpr int LN_U = 16;
__global__ void __launch_bounds__(256) layer_norm_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ w,
                                                         const float* __restrict__ b, float eps, int W, float* __restrict__ y) {
    griddep_launch();
    griddep_wait();
    __shared__ float red[33];
    const float* from = x + (size_t)rows[blockIdx.x] * W;
    float* to = y + (size_t)blockIdx.x * W;
    float sum = 0.f, sq = 0.f;
    if (W <= 256 * LN_U) {
        float v[LN_U], wv[LN_U], bv[LN_U];
#pragma unroll
        for (int u = 0; u < LN_U; u++) {
            const int i = threadIdx.x + 256 * u;
            const bool in = i < W;
            v[u] = in ? from[i] : 0.f; wv[u] = in ? w[i] : 0.f; bv[u] = in && b ? b[i] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < LN_U; u++) if (threadIdx.x + 256 * u < W) sum += v[u];
        const float mean = block_sum(sum, red) / (float)W;
#pragma unroll
        for (int u = 0; u < LN_U; u++) if (threadIdx.x + 256 * u < W) { const float dlt = v[u] - mean; sq += dlt * dlt; }
        const float rstd = 1.f / sqrtf(block_sum(sq, red) / (float)W + eps);
#pragma unroll
        for (int u = 0; u < LN_U; u++) if (threadIdx.x + 256 * u < W) to[threadIdx.x + 256 * u] = fmaf((v[u] - mean) * rstd, wv[u], bv[u]);
        return;
    }
    for (int i = threadIdx.x; i < W; i += blockDim.x) sum += from[i];
    const float mean = block_sum(sum, red) / (float)W;
    for (int i = threadIdx.x; i < W; i += blockDim.x) { const float dlt = from[i] - mean; sq += dlt * dlt; }
    const float rstd = 1.f / sqrtf(block_sum(sq, red) / (float)W + eps);
    for (int i = threadIdx.x; i < W; i += blockDim.x) to[i] = fmaf((from[i] - mean) * rstd, w[i], b ? b[i] : 0.f);
}
cudaError_t layer_norm_rows_launch(const float* x, const int* rows, const float* w, const float* b, float eps, int W, int n, float* y, cudaStream_t s) {
    return launch_chain(layer_norm_kernel, dim3(n), dim3(256), 0, s, x, rows, w, b, eps, W, y);
}

// parallel blocks: both sublayers' outputs (a mixture's expert rows are summed here) join the 32-bit stream, and both norms of
// the next layer are made from one mean and one variance; the row lives in shared memory between the passes. Bound by latency: the
// entries of a thread are read JOIN_U at a time (the stores between them would otherwise keep every read behind the last one), with an
// expert row's number looked up once per batch. 32 rows of 2048 with two experts each: 12.1 -> 7.0 us.
constexpr int JOIN_U = 4;
struct ParallelJoinDev { ParallelJoinArgs a; MoeJoinArgs j; EmbedDev e; int moe; };
// EMBED: the stream starts here, from the embedding. That reads nothing of a kernel before it (the step's description is a copy ahead of all kernels), so the
// tables of the step's experts may still be made; it ends after them, since what comes next waits for this kernel alone.
template <int NT, bool EMBED>
__global__ void __launch_bounds__(NT) parallel_join_kernel(const __grid_constant__ ParallelJoinDev p, int W) {
    griddep_launch();
    if constexpr (!EMBED) griddep_wait();
    extern __shared__ float row[];
    __shared__ float red[33];
    const ParallelJoinArgs& a = p.a;
    const MoeJoinArgs& j = p.j;
    const int t = blockIdx.x;
    const size_t base = (size_t)t * W;
    const bool adds = a.a || a.b || p.moe;
    float sum = 0.f;
    for (int i0 = threadIdx.x; i0 < W; i0 += NT * JOIN_U) {
        float v[JOIN_U], y[JOIN_U], z[JOIN_U];
#pragma unroll
        for (int u = 0; u < JOIN_U; u++) {
            const int i = i0 + u * NT;
            const bool in = i < W;
            if constexpr (EMBED) { float e[1] = {0.f}; if (in) embed_at(p.e, W, t, i, e); v[u] = e[0]; }
            else v[u] = in ? a.x[base + i] : 0.f;
            y[u] = in && a.a ? a.a[base + i] : 0.f;
            z[u] = in && a.b ? a.b[base + i] : 0.f;
        }
        if (a.b)
#pragma unroll
            for (int u = 0; u < JOIN_U; u++) y[u] += z[u];
        if (p.moe) {
            float acc[JOIN_U] = {};
            for (int c = 0; c < j.top; c++) {
                const int q = t * j.top + c;
                const float wt = j.weight ? j.weight[q] : 1.f;
                const float* from = j.sel[q] < j.n_experts ? j.rows + (size_t)(j.pos ? j.pos[q] : q) * W : j.h + base;
#pragma unroll
                for (int u = 0; u < JOIN_U; u++) z[u] = i0 + u * NT < W ? from[i0 + u * NT] : 0.f;
#pragma unroll
                for (int u = 0; u < JOIN_U; u++) acc[u] = fmaf(wt, z[u], acc[u]);
            }
#pragma unroll
            for (int u = 0; u < JOIN_U; u++) y[u] += acc[u];
        }
#pragma unroll
        for (int u = 0; u < JOIN_U; u++) {
            const int i = i0 + u * NT;
            if (i >= W) continue;
            if (adds) v[u] += y[u];
            if (adds || EMBED) a.x[base + i] = v[u];
            if (a.x_copy) a.x_copy[(size_t)t * a.ld_copy + i] = v[u];
            row[i] = v[u];
            sum += v[u];
        }
    }
    if (!a.w1 && !a.w2) {
        if constexpr (EMBED) griddep_wait();
        return;
    }
    const float mean = block_sum(sum, red) / (float)W;
    float sq = 0.f;
    for (int i = threadIdx.x; i < W; i += NT) { const float dlt = row[i] - mean; sq = fmaf(dlt, dlt, sq); }
    const float rstd = 1.f / sqrtf(block_sum(sq, red) / (float)W + a.eps);
    for (int i0 = threadIdx.x; i0 < W; i0 += NT * JOIN_U) {
        float w1[JOIN_U], b1[JOIN_U], w2[JOIN_U], b2[JOIN_U];
#pragma unroll
        for (int u = 0; u < JOIN_U; u++) {
            const int i = i0 + u * NT;
            const bool in = i < W;
            w1[u] = in && a.w1 ? a.w1[i] : 0.f; b1[u] = in && a.w1 && a.b1 ? a.b1[i] : 0.f;
            w2[u] = in && a.w2 ? a.w2[i] : 0.f; b2[u] = in && a.w2 && a.b2 ? a.b2[i] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < JOIN_U; k++) {
            const int i = i0 + k * NT;
            if (i >= W) continue;
            const float u = (row[i] - mean) * rstd;
            if (a.w1) {
                const float v = fmaf(u, w1[k], b1[k]);
                if (a.y1) a.y1[base + i] = v;
                if (a.y1_bf16) a.y1_bf16[base + i] = __float2bfloat16(v);
            }
            if (a.w2) {
                const float v = fmaf(u, w2[k], b2[k]);
                if (a.y2) a.y2[base + i] = v;
                if (a.y2_bf16) a.y2_bf16[base + i] = __float2bfloat16(v);
            }
        }
    }
    if constexpr (EMBED) griddep_wait();
}
// The same for rows of at most 4096 entries on 16-byte boundaries: a thread keeps its entries (NV times four) in registers. Bound by memory:
// 2048 rows of 2048 with two experts' rows each, both norms' outputs among 100 MB: 46 us with single reads and the row in shared memory, 34 here
// (from the launch, which is ahead of the product before it: prompts 748 -> 732 and 1593 -> 1558). Wider rows than 4096 would not fit the registers.
template <int NV, bool EMBED>
__global__ void __launch_bounds__(256) parallel_join_vec_kernel(const __grid_constant__ ParallelJoinDev p, int W) {
    griddep_launch();
    if constexpr (!EMBED) griddep_wait();
    __shared__ float red[33];
    const ParallelJoinArgs& a = p.a;
    const MoeJoinArgs& j = p.j;
    const int t = blockIdx.x;
    const size_t base = (size_t)t * W;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto at = [&](int k) { return (k * 256 + (int)threadIdx.x) * 4; };
    auto get = [&](const float* from, int k) { return from && at(k) < W ? *reinterpret_cast<const float4*>(from + at(k)) : zero; };
    auto put = [&](float* to, int k, const float4& v) { *reinterpret_cast<float4*>(to + at(k)) = v; };
    float4 v[NV], y[NV], z[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        if constexpr (EMBED) {
            float e[4] = {0.f, 0.f, 0.f, 0.f};
            if (at(k) < W) embed_at(p.e, W, t, at(k), e);
            v[k] = make_float4(e[0], e[1], e[2], e[3]);
        } else v[k] = get(a.x + base, k);
    }
#pragma unroll
    for (int k = 0; k < NV; k++) { y[k] = get(a.a ? a.a + base : nullptr, k); z[k] = get(a.b ? a.b + base : nullptr, k); }
#pragma unroll
    for (int k = 0; k < NV; k++) { y[k].x += z[k].x; y[k].y += z[k].y; y[k].z += z[k].z; y[k].w += z[k].w; }
    if (p.moe) {
        float4 acc[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) acc[k] = zero;
#pragma unroll 2
        for (int c = 0; c < j.top; c++) {
            const int q = t * j.top + c;
            const float wt = j.weight ? j.weight[q] : 1.f;
            const float* from = j.sel[q] < j.n_experts ? j.rows + (size_t)(j.pos ? j.pos[q] : q) * W : j.h + base;
#pragma unroll
            for (int k = 0; k < NV; k++) z[k] = get(from, k);
#pragma unroll
            for (int k = 0; k < NV; k++) {
                acc[k].x = fmaf(wt, z[k].x, acc[k].x); acc[k].y = fmaf(wt, z[k].y, acc[k].y);
                acc[k].z = fmaf(wt, z[k].z, acc[k].z); acc[k].w = fmaf(wt, z[k].w, acc[k].w);
            }
        }
#pragma unroll
        for (int k = 0; k < NV; k++) { y[k].x += acc[k].x; y[k].y += acc[k].y; y[k].z += acc[k].z; y[k].w += acc[k].w; }
    }
    const bool adds = a.a || a.b || p.moe;
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        if (at(k) >= W) break;
        if (adds) { v[k].x += y[k].x; v[k].y += y[k].y; v[k].z += y[k].z; v[k].w += y[k].w; }
        if (adds || EMBED) put(a.x + base, k, v[k]);
        if (a.x_copy) put(a.x_copy + (size_t)t * a.ld_copy, k, v[k]);
        sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
    }
    if (!a.w1 && !a.w2) {
        if constexpr (EMBED) griddep_wait();
        return;
    }
    const float mean = block_sum(sum, red) / (float)W;
    float sq = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k].x -= mean; v[k].y -= mean; v[k].z -= mean; v[k].w -= mean;
        if (at(k) < W) sq += (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
    }
    const float rstd = 1.f / sqrtf(block_sum(sq, red) / (float)W + a.eps);
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const float *w = n ? a.w2 : a.w1, *b = n ? a.b2 : a.b1;
        float* to = n ? a.y2 : a.y1;
        __nv_bfloat16* to_b = n ? a.y2_bf16 : a.y1_bf16;
        if (!w) continue;
        float4 wv[NV], bv[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) { wv[k] = get(w, k); bv[k] = get(b, k); }
#pragma unroll
        for (int k = 0; k < NV; k++) {
            if (at(k) >= W) break;
            const float4 o = make_float4(fmaf(v[k].x * rstd, wv[k].x, bv[k].x), fmaf(v[k].y * rstd, wv[k].y, bv[k].y),
                                         fmaf(v[k].z * rstd, wv[k].z, bv[k].z), fmaf(v[k].w * rstd, wv[k].w, bv[k].w));
            if (to) put(to + base, k, o);
            if (to_b) store_bf16x4(to_b + base + at(k), o);
        }
    }
    if constexpr (EMBED) griddep_wait();
}
template <bool EMBED>
static cudaError_t launch_join(const ParallelJoinArgs& a, int W, int T, cudaStream_t s) {
    ParallelJoinDev p = {};
    p.a = a;
    if (a.moe) { p.j = *a.moe; p.moe = 1; }
    if (EMBED) {
        p.e = *a.embed;
        if (p.e.bg.table && !p.e.tok_prev) return cudaErrorInvalidValue;
    }
    // few tokens: more threads per row, one CTA's latency is all there is
    if (T <= 16 && W >= 1024) return launch_chain(parallel_join_kernel<1024, EMBED>, dim3(T), dim3(1024), (size_t)W * 4, s, p, W);
    const void* const all[] = {a.x, a.a, a.b, a.w1, a.b1, a.y1, a.w2, a.b2, a.y2, a.x_copy, a.y1_bf16, a.y2_bf16, p.j.rows, p.j.h};
    uintptr_t at = 0;
    for (const void* q : all) at |= reinterpret_cast<uintptr_t>(q);
    if (W % 4 == 0 && W <= 4096 && a.ld_copy % 4 == 0 && (at & 15) == 0 && (!EMBED || embed_wide(p.e, W))) {
        if (W <= 1024) return launch_chain(parallel_join_vec_kernel<1, EMBED>, dim3(T), dim3(256), 0, s, p, W);
        if (W <= 2048) return launch_chain(parallel_join_vec_kernel<2, EMBED>, dim3(T), dim3(256), 0, s, p, W);
        return launch_chain(parallel_join_vec_kernel<4, EMBED>, dim3(T), dim3(256), 0, s, p, W);
    }
    return launch_chain(parallel_join_kernel<256, EMBED>, dim3(T), dim3(256), (size_t)W * 4, s, p, W);
}
cudaError_t parallel_join_launch(const ParallelJoinArgs& a, int W, int T, cudaStream_t s) {
    return a.embed ? launch_join<true>(a, W, T, s) : launch_join<false>(a, W, T, s);
}

// ---------------------------------------------------------------- window attention
__device__ __forceinline__ void cache_store(void* pool, int f32, size_t i, float v) {
    if (f32) reinterpret_cast<float*>(pool)[i] = v;
    else reinterpret_cast<__nv_bfloat16*>(pool)[i] = __float2bfloat16(v);
}
__device__ __forceinline__ float cache_load(const void* pool, int f32, size_t i) {
    return f32 ? reinterpret_cast<const float*>(pool)[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(pool)[i]);
}

// A warp per token and head slot, [0, H) queries, [H, H + G) key/value heads; eight to a CTA (grid (T, (H + G) / 8)): with CTAs of one
// warp an SM holds half of the warps it could, and 2048 tokens of 40 slots were 82
// thousand CTAs: 85 -> 30 us.
__global__ void __launch_bounds__(256) window_attn_store_kernel(WindowAttnArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x, hs = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (hs >= a.H + a.G) return;
    const bool is_q = hs < a.H;
    const int head = is_q ? hs : hs - a.H;
    const float* src = a.proj + (size_t)t * a.ldp + (is_q ? a.q_off : a.k_off) + head * a.d;
    const float* nw = is_q ? a.q_norm_w : a.k_norm_w;
    const int pos = r.tok_pos[t];
    float ss = 0.f;
    for (int i = lane; i < a.d; i += 32) { const float v = src[i]; ss += v * v; }
    const float rinv = 1.f / sqrtf(warp_sum(ss) / (float)a.d + a.eps);
    size_t dst = 0;
    if (!is_q) {
        const int slot = r.seg_slot[r.tok_seg[t]];
        const int page = a.block_tables[slot][pos / a.block_tokens];
        dst = (((size_t)page * a.G + head) * a.block_tokens + pos % a.block_tokens) * a.d;
    }
    float* qdst = a.q_rot + (size_t)t * a.H * a.d + (size_t)head * a.d;
    // pairs (2i, 2i+1): rotated inside the first rot_dims entries, passed through after them
    for (int p = lane; 2 * p < a.d; p += 32) {
        const int i0 = 2 * p, i1 = 2 * p + 1;
        const float r0 = src[i0], r1 = i1 < a.d ? src[i1] : 0.f;
        float u = r0 * rinv * nw[i0], v = i1 < a.d ? r1 * rinv * nw[i1] : 0.f;
        if (i1 < a.rot.rot_dims) {
            const size_t ti = (size_t)pos * (a.rot.rot_dims / 2) + p;
            const float sn = a.rot.sin[ti], cs = a.rot.cos[ti];
            const float u2 = u * cs - v * sn, v2 = v * cs + u * sn;
            u = u2; v = v2;
        }
        if (is_q) {
            qdst[i0] = u;
            if (i1 < a.d) qdst[i1] = v;
        } else {
            cache_store(a.k_pool, a.cache_f32, dst + i0, u);
            cache_store(a.v_pool, a.cache_f32, dst + i0, r0);
            if (i1 < a.d) { cache_store(a.k_pool, a.cache_f32, dst + i1, v); cache_store(a.v_pool, a.cache_f32, dst + i1, r1); }
        }
    }
}
// The same for head sizes up to 128 whose rows are whole 16-byte pieces: a lane has four neighbouring entries, read once (30 -> 22 us).
__device__ __forceinline__ void cache_store4(void* pool, int f32, size_t i, const float4& v) {
    if (f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(pool) + i) = v;
    else store_bf16x4(reinterpret_cast<__nv_bfloat16*>(pool) + i, v);
}
__global__ void __launch_bounds__(256) window_attn_store_vec_kernel(WindowAttnArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x, hs = blockIdx.y * 8 + (threadIdx.x >> 5), i = (threadIdx.x & 31) * 4;
    if (hs >= a.H + a.G) return;
    const bool is_q = hs < a.H, in = i < a.d;
    const int head = is_q ? hs : hs - a.H, pos = r.tok_pos[t];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 raw = in ? *reinterpret_cast<const float4*>(a.proj + (size_t)t * a.ldp + (is_q ? a.q_off : a.k_off) + head * a.d + i) : zero;
    const float4 w = in ? *reinterpret_cast<const float4*>((is_q ? a.q_norm_w : a.k_norm_w) + i) : zero;
    float cs[2] = {1.f, 1.f}, sn[2] = {0.f, 0.f};
#pragma unroll
    for (int p = 0; p < 2; p++)
        if (in && i + 2 * p + 1 < a.rot.rot_dims) {          // pairs (2i, 2i + 1) inside the first rot_dims entries are rotated
            const size_t at = (size_t)pos * (a.rot.rot_dims / 2) + i / 2 + p;
            cs[p] = a.rot.cos[at]; sn[p] = a.rot.sin[at];
        }
    const float rinv = 1.f / sqrtf(warp_sum(raw.x * raw.x + raw.y * raw.y + raw.z * raw.z + raw.w * raw.w) / (float)a.d + a.eps);
    if (!in) return;
    const float4 u = make_float4(raw.x * rinv * w.x, raw.y * rinv * w.y, raw.z * rinv * w.z, raw.w * rinv * w.w);
    const float4 y = make_float4(u.x * cs[0] - u.y * sn[0], u.y * cs[0] + u.x * sn[0], u.z * cs[1] - u.w * sn[1], u.w * cs[1] + u.z * sn[1]);
    if (is_q) {
        *reinterpret_cast<float4*>(a.q_rot + (size_t)t * a.H * a.d + (size_t)head * a.d + i) = y;
        return;
    }
    const int page = a.block_tables[r.seg_slot[r.tok_seg[t]]][pos / a.block_tokens];
    const size_t dst = (((size_t)page * a.G + head) * a.block_tokens + pos % a.block_tokens) * a.d + i;
    cache_store4(a.k_pool, a.cache_f32, dst, y);
    cache_store4(a.v_pool, a.cache_f32, dst, raw);
}
cudaError_t window_attn_store_launch(const WindowAttnArgs& a, const RaggedDev& r, cudaStream_t s) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(a.proj) | reinterpret_cast<uintptr_t>(a.q_norm_w) | reinterpret_cast<uintptr_t>(a.k_norm_w) |
                         reinterpret_cast<uintptr_t>(a.q_rot) | reinterpret_cast<uintptr_t>(a.k_pool) | reinterpret_cast<uintptr_t>(a.v_pool);
    const bool vec = a.d % 4 == 0 && a.d <= 128 && a.ldp % 4 == 0 && a.q_off % 4 == 0 && a.k_off % 4 == 0 && (at & 15) == 0;
    return launch_chain(vec ? window_attn_store_vec_kernel : window_attn_store_kernel, dim3(r.T, (a.H + a.G + 7) / 8), dim3(256), 0, s, a, r);
}

// grid (T, H), 4 warps: warp w takes visible keys w, w + 4, ...; a lane holds entries lane, lane + 32, ... of the head
constexpr int ATT_WARPS = 4, ATT_MAXE = 8;     // head size <= 256
__global__ void __launch_bounds__(ATT_WARPS * 32) window_attn_kernel(WindowAttnArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    __shared__ float sm_m[ATT_WARPS], sm_l[ATT_WARPS];
    __shared__ float sm_o[ATT_WARPS][ATT_MAXE * 32];
    const int t = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = r.tok_pos[t];
    const int slot = r.seg_slot[r.tok_seg[t]];
    const int* table = a.block_tables[slot];
    const int g = h / (a.H / a.G);
    const float* q = a.q_rot + (size_t)t * a.H * a.d + (size_t)h * a.d;
    float qr[ATT_MAXE], acc[ATT_MAXE];
#pragma unroll
    for (int e = 0; e < ATT_MAXE; e++) { const int i = lane + 32 * e; qr[e] = i < a.d ? q[i] * a.scale : 0.f; acc[e] = 0.f; }
    // visible: the kept prefix [0, n_keep) and the window [lo, pos]
    const int lo = max(0, pos - a.window + 1);
    const int n_keep = min(a.keep_first, lo);
    const int n_vis = n_keep + (pos - lo + 1);
    float m = -INFINITY, l = 0.f;
    for (int i = warp; i < n_vis; i += ATT_WARPS) {
        const int j = i < n_keep ? i : lo + (i - n_keep);
        const size_t base = (((size_t)table[j / a.block_tokens] * a.G + g) * a.block_tokens + j % a.block_tokens) * a.d;
        float dot = 0.f;
#pragma unroll
        for (int e = 0; e < ATT_MAXE; e++) { const int d = lane + 32 * e; if (d < a.d) dot = fmaf(qr[e], cache_load(a.k_pool, a.cache_f32, base + d), dot); }
        const float sc = warp_sum(dot);
        const float m_new = fmaxf(m, sc);
        const float corr = expf(m - m_new), p = expf(sc - m_new);
        l = l * corr + p;
#pragma unroll
        for (int e = 0; e < ATT_MAXE; e++) { const int d = lane + 32 * e; if (d < a.d) acc[e] = fmaf(p, cache_load(a.v_pool, a.cache_f32, base + d), acc[e] * corr); }
        m = m_new;
    }
    if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
#pragma unroll
    for (int e = 0; e < ATT_MAXE; e++) sm_o[warp][lane + 32 * e] = acc[e];
    __syncthreads();
    float M = -INFINITY;
    for (int w2 = 0; w2 < ATT_WARPS; w2++) M = fmaxf(M, sm_m[w2]);
    float L = 0.f;
    for (int w2 = 0; w2 < ATT_WARPS; w2++) if (sm_m[w2] > -INFINITY) L += sm_l[w2] * expf(sm_m[w2] - M);
    for (int d = threadIdx.x; d < a.d; d += blockDim.x) {
        float o = 0.f;
        for (int w2 = 0; w2 < ATT_WARPS; w2++) if (sm_m[w2] > -INFINITY) o += sm_o[w2][d] * expf(sm_m[w2] - M);
        a.out[(size_t)t * a.H * a.d + (size_t)h * a.d + d] = o / L;
    }
}
// Even head sizes: 8 warps, a warp takes 4 visible keys per round (their loads and the four dot-product reductions overlap),
// a lane holds pairs of neighbouring entries (one 4- or 8-byte load per key and 64 entries of the head).
constexpr int ATT2_WARPS = 8, ATT2_KEYS = 4, ATT2_PASS = 4;       // head size <= 256
template <bool F32>
__device__ __forceinline__ float2 cache_load2(const void* pool, size_t i) {
    if constexpr (F32) return *reinterpret_cast<const float2*>(reinterpret_cast<const float*>(pool) + i);
    const uint32_t u = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const __nv_bfloat16*>(pool) + i);
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
// of_tiles: CTA x takes the token of tile x (the one-token tiles come first) instead of token x
template <bool F32>
__global__ void __launch_bounds__(ATT2_WARPS * 32) window_attn_pairs_kernel(WindowAttnArgs a, RaggedDev r, int of_tiles) {
    griddep_launch();
    griddep_wait();
    __shared__ float sm_m[ATT2_WARPS], sm_l[ATT2_WARPS];
    __shared__ float sm_o[ATT2_WARPS][ATT2_PASS * 64];
    const int t = of_tiles ? r.tile_row0[blockIdx.x] : (int)blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = r.tok_pos[t];
    const int slot = r.seg_slot[r.tok_seg[t]];
    const int* table = a.block_tables[slot];
    const int g = h / (a.H / a.G), d = a.d;
    const float* q = a.q_rot + (size_t)t * a.H * d + (size_t)h * d;
    float2 qr[ATT2_PASS], acc[ATT2_PASS];
#pragma unroll
    for (int e = 0; e < ATT2_PASS; e++) {
        const int i = 64 * e + 2 * lane;
        qr[e] = i < d ? make_float2(q[i] * a.scale, q[i + 1] * a.scale) : make_float2(0.f, 0.f);
        acc[e] = make_float2(0.f, 0.f);
    }
    const int lo = max(0, pos - a.window + 1);
    const int n_keep = min(a.keep_first, lo);
    const int n_all = n_keep + (pos - lo + 1);
    // several CTAs per (token, head) when the step is small: CTA z takes the z-th range of the visible keys
    const int n_splits = gridDim.z, chunk = (n_all + n_splits - 1) / n_splits;
    const int i_begin = blockIdx.z * chunk, n_vis = min(n_all, i_begin + chunk);
    float m = -INFINITY, l = 0.f;
    for (int i0 = i_begin + warp * ATT2_KEYS; i0 < n_vis; i0 += ATT2_WARPS * ATT2_KEYS) {
        size_t base[ATT2_KEYS];
        float2 kv[ATT2_KEYS][ATT2_PASS], vv[ATT2_KEYS][ATT2_PASS];
        float sc[ATT2_KEYS];
#pragma unroll
        for (int u = 0; u < ATT2_KEYS; u++) {
            const int i = min(i0 + u, n_vis - 1);         // past the end: the last key again, its weight is dropped below
            const int j = i < n_keep ? i : lo + (i - n_keep);
            base[u] = (((size_t)table[j / a.block_tokens] * a.G + g) * a.block_tokens + j % a.block_tokens) * d;
        }
#pragma unroll
        for (int u = 0; u < ATT2_KEYS; u++)
#pragma unroll
            for (int e = 0; e < ATT2_PASS; e++) {
                const int i = 64 * e + 2 * lane;
                kv[u][e] = i < d ? cache_load2<F32>(a.k_pool, base[u] + i) : make_float2(0.f, 0.f);
                vv[u][e] = i < d ? cache_load2<F32>(a.v_pool, base[u] + i) : make_float2(0.f, 0.f);
            }
#pragma unroll
        for (int u = 0; u < ATT2_KEYS; u++) {
            float dot = 0.f;
#pragma unroll
            for (int e = 0; e < ATT2_PASS; e++) dot = fmaf(qr[e].x, kv[u][e].x, fmaf(qr[e].y, kv[u][e].y, dot));
            sc[u] = dot;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < ATT2_KEYS; u++) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
        float m_new = m;
#pragma unroll
        for (int u = 0; u < ATT2_KEYS; u++) if (i0 + u < n_vis) m_new = fmaxf(m_new, sc[u]);
        const float corr = expf(m - m_new);
        float p[ATT2_KEYS], ps = 0.f;
#pragma unroll
        for (int u = 0; u < ATT2_KEYS; u++) { p[u] = i0 + u < n_vis ? expf(sc[u] - m_new) : 0.f; ps += p[u]; }
        l = l * corr + ps;
#pragma unroll
        for (int e = 0; e < ATT2_PASS; e++) {
            float ax = acc[e].x * corr, ay = acc[e].y * corr;
#pragma unroll
            for (int u = 0; u < ATT2_KEYS; u++) { ax = fmaf(p[u], vv[u][e].x, ax); ay = fmaf(p[u], vv[u][e].y, ay); }
            acc[e] = make_float2(ax, ay);
        }
        m = m_new;
    }
    if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
#pragma unroll
    for (int e = 0; e < ATT2_PASS; e++) { sm_o[warp][64 * e + 2 * lane] = acc[e].x; sm_o[warp][64 * e + 2 * lane + 1] = acc[e].y; }
    __syncthreads();
    float M = -INFINITY;
    for (int w2 = 0; w2 < ATT2_WARPS; w2++) M = fmaxf(M, sm_m[w2]);
    float L = 0.f;
    for (int w2 = 0; w2 < ATT2_WARPS; w2++) if (sm_m[w2] > -INFINITY) L += sm_l[w2] * expf(sm_m[w2] - M);
    float* part = n_splits > 1 ? a.split_scratch + (((size_t)t * a.H + h) * n_splits + blockIdx.z) * (d + 2) : nullptr;
    if (part && threadIdx.x == 0) { part[0] = M; part[1] = L; }
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float o = 0.f;
        for (int w2 = 0; w2 < ATT2_WARPS; w2++) if (sm_m[w2] > -INFINITY) o += sm_o[w2][i] * expf(sm_m[w2] - M);
        if (part) part[2 + i] = o;                         // unnormalised: window_attn_merge_kernel finishes
        else a.out[(size_t)t * a.H * d + (size_t)h * d + i] = o / L;
    }
}

// sum of the key ranges of one (token, head) in range order
__global__ void __launch_bounds__(128) window_attn_merge_kernel(WindowAttnArgs a, RaggedDev r, int n_splits, int of_tiles) {
    griddep_launch();
    griddep_wait();
    const int t = of_tiles ? r.tile_row0[blockIdx.x] : (int)blockIdx.x, h = blockIdx.y, d = a.d;
    const float* part = a.split_scratch + ((size_t)t * a.H + h) * n_splits * (d + 2);
    float M = -INFINITY;
    for (int s2 = 0; s2 < n_splits; s2++) M = fmaxf(M, part[(size_t)s2 * (d + 2)]);
    float L = 0.f;
    for (int s2 = 0; s2 < n_splits; s2++) { const float ms = part[(size_t)s2 * (d + 2)]; if (ms > -INFINITY) L += part[(size_t)s2 * (d + 2) + 1] * expf(ms - M); }
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float o = 0.f;
        for (int s2 = 0; s2 < n_splits; s2++) { const float ms = part[(size_t)s2 * (d + 2)]; if (ms > -INFINITY) o += part[(size_t)s2 * (d + 2) + 2 + i] * expf(ms - M); }
        a.out[(size_t)t * a.H * d + (size_t)h * d + i] = o / L;
    }
}

// Tensor-core prompt attention (bf16 pages, head size a multiple of 16 up to 128): a CTA takes one tile of up to 64 consecutive
// queries of a segment and one head; 4 warps x 16 query rows; keys in blocks of 64 -- first the blocks that hold kept-prefix
// keys, then the blocks the tile's windows reach -- staged in shared memory once for all 64 queries. S = Q K^T and O += P V
// with mma.sync m16n8k16 (bf16 in, f32 accumulate); mask, running maximum, exponentials and the sum are 32-bit. Queries and
// probabilities enter the products as TWO bf16 each (value = leading part + remainder), so the only 16-bit rounding on this
// path is that of the cached keys and values -- the same as on the decode path.
constexpr int FA_Q = 64, FA_K = 64;
__device__ __forceinline__ void cp_async_16z(void* smem_dst, const void* gsrc, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void split_bf16(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = pack_bf16(a - __low2float(h), b - __high2float(h));
}

template <int DMAX>
__global__ void __launch_bounds__(128) window_attn_mma_kernel(WindowAttnArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    extern __shared__ __align__(16) unsigned char fa_smem[];
    const int d = a.d, LD = d + 8;
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(fa_smem);     // [64][LD] leading bf16 of the scaled query
    __nv_bfloat16* Ql = Qs + FA_Q * LD;                                 // [64][LD] what the first bf16 leaves over
    __nv_bfloat16* Ks = Ql + FA_Q * LD;
    __nv_bfloat16* Vs = Ks + FA_K * LD;
    const int tile = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int seg = r.tile_seg[tile], row0 = r.tile_row0[tile];
    const int nq = min(FA_Q, r.seg_start[seg] + r.seg_len[seg] - row0);
    const int p0 = r.tok_pos[row0], p_last = p0 + nq - 1;
    const int* table = a.block_tables[r.seg_slot[seg]];
    const int g = h / (a.H / a.G);
    const __nv_bfloat16* kp = reinterpret_cast<const __nv_bfloat16*>(a.k_pool);
    const __nv_bfloat16* vp = reinterpret_cast<const __nv_bfloat16*>(a.v_pool);
    // queries: scaled, rounded to bf16; rows past the tile are zero
    for (int i = threadIdx.x; i < FA_Q * (d / 2); i += blockDim.x) {
        const int rr = i / (d / 2), c = (i % (d / 2)) * 2;
        float2 v = make_float2(0.f, 0.f);
        if (rr < nq) {
            const float* q = a.q_rot + (size_t)(row0 + rr) * a.H * d + (size_t)h * d + c;
            v = make_float2(q[0] * a.scale, q[1] * a.scale);
        }
        const __nv_bfloat162 hi = __floats2bfloat162_rn(v.x, v.y);
        *reinterpret_cast<__nv_bfloat162*>(Qs + rr * LD + c) = hi;
        *reinterpret_cast<__nv_bfloat162*>(Ql + rr * LD + c) = __floats2bfloat162_rn(v.x - __low2float(hi), v.y - __high2float(hi));
    }
    const int lo_first = max(0, p0 - a.window + 1);
    const int n_kept_blocks = lo_first > 0 ? (min(a.keep_first, lo_first) + FA_K - 1) / FA_K : 0;
    const int win_b0 = max(lo_first / FA_K, n_kept_blocks), win_b1 = p_last / FA_K;
    const int n_blocks = n_kept_blocks + (win_b1 - win_b0 + 1);
    float o[DMAX / 8][4];
#pragma unroll
    for (int i = 0; i < DMAX / 8; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    const int gq = lane >> 2, tq = lane & 3;
    const int qrow[2] = {warp * 16 + gq, warp * 16 + gq + 8};
    for (int bi = 0; bi < n_blocks; bi++) {
        const int kb = bi < n_kept_blocks ? bi : win_b0 + (bi - n_kept_blocks);
        const int j0 = kb * FA_K;
        __syncthreads();                      // everybody is done with the previous block's K and V (and Q is written)
        for (int i = threadIdx.x; i < FA_K * (d / 8); i += blockDim.x) {
            const int rr = i / (d / 8), c = (i % (d / 8)) * 8;
            const int j = j0 + rr;
            const int jj = min(j, p_last);
            const size_t base = (((size_t)table[jj / a.block_tokens] * a.G + g) * a.block_tokens + jj % a.block_tokens) * d + c;
            cp_async_16z(Ks + rr * LD + c, kp + base, j <= p_last ? 16 : 0);
            cp_async_16z(Vs + rr * LD + c, vp + base, j <= p_last ? 16 : 0);
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
        // S = Q K^T for this warp's 16 rows
        float sacc[FA_K / 8][4];
#pragma unroll
        for (int ni = 0; ni < FA_K / 8; ni++) sacc[ni][0] = sacc[ni][1] = sacc[ni][2] = sacc[ni][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < DMAX; ks += 16) {
            if (ks < d) {
                uint32_t af[4], al[4];
                ldsm_x4(af, Qs + (warp * 16 + (lane & 15)) * LD + ks + (lane >> 4) * 8);
                ldsm_x4(al, Ql + (warp * 16 + (lane & 15)) * LD + ks + (lane >> 4) * 8);
#pragma unroll
                for (int nj = 0; nj < FA_K / 16; nj++) {
                    uint32_t bf[4];
                    ldsm_x4(bf, Ks + (nj * 16 + (lane & 7) + ((lane >> 4) << 3)) * LD + ks + ((lane >> 3) & 1) * 8);
                    mma_16816(sacc[2 * nj], al, bf[0], bf[1]);
                    mma_16816(sacc[2 * nj + 1], al, bf[2], bf[3]);
                    mma_16816(sacc[2 * nj], af, bf[0], bf[1]);
                    mma_16816(sacc[2 * nj + 1], af, bf[2], bf[3]);
                }
            }
        }
        // mask, running maximum, exponentials
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int ni = 0; ni < FA_K / 8; ni++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int rr = qrow[e >> 1], i = p0 + rr, j = j0 + ni * 8 + 2 * tq + (e & 1);
                const bool vis = rr < nq && j <= i && (i - j < a.window || j < a.keep_first);
                const float v = vis ? sacc[ni][e] : -INFINITY;
                sacc[ni][e] = v;
                mx[e >> 1] = fmaxf(mx[e >> 1], v);
            }
        float corr[2], msafe[2];
#pragma unroll
        for (int q2 = 0; q2 < 2; q2++) {
            mx[q2] = fmaxf(mx[q2], __shfl_xor_sync(0xffffffffu, mx[q2], 1));
            mx[q2] = fmaxf(mx[q2], __shfl_xor_sync(0xffffffffu, mx[q2], 2));
            const float m_new = fmaxf(m_run[q2], mx[q2]);
            msafe[q2] = m_new == -INFINITY ? 0.f : m_new;
            corr[q2] = expf(m_run[q2] - msafe[q2]);
            m_run[q2] = m_new;
            l_run[q2] *= corr[q2];
        }
#pragma unroll
        for (int ni = 0; ni < FA_K / 8; ni++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float pv = expf(sacc[ni][e] - msafe[e >> 1]);
                sacc[ni][e] = pv;
                l_run[e >> 1] += pv;
            }
#pragma unroll
        for (int i = 0; i < DMAX / 8; i++) { o[i][0] *= corr[0]; o[i][1] *= corr[0]; o[i][2] *= corr[1]; o[i][3] *= corr[1]; }
        // O += P V
#pragma unroll
        for (int kc = 0; kc < FA_K / 16; kc++) {
            uint32_t pf[4], pl[4];         // probabilities as two bf16 each (leading part + remainder): ~16 bits reach the product
            split_bf16(sacc[2 * kc][0], sacc[2 * kc][1], pf[0], pl[0]);
            split_bf16(sacc[2 * kc][2], sacc[2 * kc][3], pf[1], pl[1]);
            split_bf16(sacc[2 * kc + 1][0], sacc[2 * kc + 1][1], pf[2], pl[2]);
            split_bf16(sacc[2 * kc + 1][2], sacc[2 * kc + 1][3], pf[3], pl[3]);
#pragma unroll
            for (int nd = 0; nd < DMAX / 16; nd++) {
                if (nd * 16 < d) {
                    uint32_t vf[4];
                    ldsm_x4_t(vf, Vs + (kc * 16 + (lane & 15)) * LD + nd * 16 + (lane >> 4) * 8);
                    mma_16816(o[2 * nd], pl, vf[0], vf[1]);
                    mma_16816(o[2 * nd + 1], pl, vf[2], vf[3]);
                    mma_16816(o[2 * nd], pf, vf[0], vf[1]);
                    mma_16816(o[2 * nd + 1], pf, vf[2], vf[3]);
                }
            }
        }
    }
#pragma unroll
    for (int q2 = 0; q2 < 2; q2++) {
        l_run[q2] += __shfl_xor_sync(0xffffffffu, l_run[q2], 1);
        l_run[q2] += __shfl_xor_sync(0xffffffffu, l_run[q2], 2);
    }
#pragma unroll
    for (int i = 0; i < DMAX / 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int rr = qrow[e >> 1], c = i * 8 + 2 * tq + (e & 1);
            if (rr < nq && c < d) a.out[(size_t)(row0 + rr) * a.H * d + (size_t)h * d + c] = o[i][e] / l_run[e >> 1];
        }
}

static bool window_attn_mma(const WindowAttnArgs& a, int T) {
    static const bool no_mma = getenv("B2_NO_ATTN_MMA") != nullptr;        // tuning aid: scalar attention for prompts too
    return !no_mma && !a.cache_f32 && T > 8 && a.d % 16 == 0 && a.d <= 128;
}
static SoftmaxTcArgs window_softmax_args(const WindowAttnArgs& a) {
    SoftmaxTcArgs x = {};
    x.q = a.q_rot; x.k_pool = a.k_pool; x.v_pool = a.v_pool; x.pool_rows = a.pool_rows; x.block_tables = a.block_tables; x.block_tokens = a.block_tokens;
    x.H = a.H; x.G = a.G; x.d = x.dv = a.d; x.window = a.window; x.keep_first = a.keep_first; x.scale = a.scale; x.ld_out = a.H * a.d;
    x.out = a.out; x.out_bf16 = a.out_rounded;
    return x;
}
bool window_attn_leaves_rounded(const WindowAttnArgs& a, int T) { return window_attn_mma(a, T) && softmax_takes_tc(window_softmax_args(a)); }
// 32-bit pages, sequences that bring two tokens or more to a step of more than 8: 32 queries of one head a CTA, blocks of 64 keys and values by asynchronous
// copies one block ahead. A warp has four queries and one half of every block. Scores: a lane multiplies four queries with four keys over every fourth piece of
// four entries, 8 multiply-adds a read; the four lanes of a key group add their parts up, each ending up with one query's. Sums: a lane has four entries of the
// output of all four queries. Nothing is less than 32 bits. Blocks start at multiples of 64 keys and are summed up in ranges of 128, whose sums meet in
// the order of the keys: a row's bits depend neither on the tile that it is in nor on `company`, the CTAs of a cluster that share a tile's ranges (and then its
// queries' sums over ranges) where a step has too few tiles to fill the GPU.
// Bound by its instructions on the SMs that have a CTA (issue slots 60 %, multiply-adds 37 %, the shared-memory pipe 22 %, by counters) and by the longest
// tile. (459 tokens of 8 heads of 128 in two sequences: 105 us with a CTA per token and head, every key read from L2 by each; 60 with one warp a query group
// and blocks of 32 keys, 37 here. 900 tokens, a whole prompt of two layers: 1044 -> 622 us. A step of few tokens behind many keys, two layers with a window of
// 1024: 20 tokens 323 -> 249, 64 tokens 432 -> 306. Ranges of 256 give a window of 300 too few to share: 32 tokens 245 us against 227, of 237 before.)
constexpr int WT_Q = 32, WT_K = 64, WT_OWN = 32, WT_WARPS = 16, WT_D = 128, WT_RANGE = 2;
constexpr int WT_FEW = 4, WT_SLOTS = 16;                   // queries of a tile whose warps take ranges of their own; ranges of such a CTA between two merges

// What a warp has of a range: maxima and sums of weights of the query whose scores a lane ends up with (the sums: of the lane's keys), four entries of the
// weighted sums of all four
struct WtSums { float m, l; float4 o[4]; };
// One block's half, 32 keys, added to them. `qr`: this lane's piece of the first query; `key(u, c)`: this lane's piece c of key u of its four;
// `value(j)`: this lane's four entries of key j; `pos`, `lo`: of the lane's query; `first`: position of the warp's first query. (Explicit operations
// where a compiler could fuse: both callers' sums have the same bits.)
template <int AHEAD, typename Key, typename Value>
__device__ __forceinline__ void wt_add_half(WtSums& w, const WindowAttnArgs& a, const float* qr, int ldk, float* pw, int j0, int pos, int lo, int first, int lane, Key key, Value value) {
    const int kg = lane >> 2, part = lane & 3, d = a.d;
    float sc[4][4];                                        // [query][key of the group]
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) sc[u][v] = 0.f;
    // (AHEAD steps of 16 entries are read before the first is used: shared memory answers in time, a page does not)
#pragma unroll 1
    for (int c = 0; c < d; c += 16 * AHEAD) {
        float4 k[AHEAD][4];
#pragma unroll
        for (int i = 0; i < AHEAD; i++)
#pragma unroll
            for (int u = 0; u < 4; u++) k[i][u] = key(u, min(c + 16 * i, d - 16));
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            if (c + 16 * i >= d) break;
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = *reinterpret_cast<const float4*>(qr + u * ldk + c + 16 * i);
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int v = 0; v < 4; v++) sc[u][v] += fmaf(q[u].x, k[i][v].x, fmaf(q[u].y, k[i][v].y, fmaf(q[u].z, k[i][v].z, q[u].w * k[i][v].w)));
        }
    }
    // the four parts of every score: lane `part` ends up with query `part`
    float s[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const bool up = part & 2, odd = part & 1;
        const float x0 = (up ? sc[2][v] : sc[0][v]) + __shfl_xor_sync(0xffffffffu, up ? sc[0][v] : sc[2][v], 2);
        const float x1 = (up ? sc[3][v] : sc[1][v]) + __shfl_xor_sync(0xffffffffu, up ? sc[1][v] : sc[3][v], 2);
        s[v] = (odd ? x1 : x0) + __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 1);
    }
    float mx = w.m;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int j = j0 + kg * 4 + v;
        if (j > pos || (j < lo && j >= a.keep_first)) s[v] = -INFINITY;
        mx = fmaxf(mx, s[v]);
    }
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
    const float ref = mx > -INFINITY ? mx : 0.f, corr = w.m > -INFINITY ? expf(w.m - ref) : 0.f;      // (nothing visible yet: all weights are 0)
    w.m = mx;
    w.l = __fmul_rn(w.l, corr);
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const float e = expf(s[v] - ref);
        w.l = __fadd_rn(w.l, e);
        pw[(kg * 4 + v) * 4 + part] = e;
    }
    __syncwarp();
    float4 b[4];                                           // the block's own sums: short chains of additions
#pragma unroll
    for (int u = 0; u < 4; u++) b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](auto all) {
#pragma unroll 1
        for (int j = 0; j < WT_OWN; j += 8) {
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = value(j + i);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 p = *reinterpret_cast<const float4*>(pw + (j + i) * 4);
                const float e[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (all || e[u] != 0.f) { b[u].x = fmaf(e[u], v[i].x, b[u].x); b[u].y = fmaf(e[u], v[i].y, b[u].y); b[u].z = fmaf(e[u], v[i].z, b[u].z); b[u].w = fmaf(e[u], v[i].w, b[u].w); }
            }
        }
    };
    // (a key that some of the warp's queries do not see must not reach them, not even as 0 times infinity)
    if (j0 + WT_OWN - 1 <= first && j0 >= first + 3 - a.window + 1) add(std::true_type{});
    else add(std::false_type{});
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const float f = __shfl_sync(0xffffffffu, corr, u);
        w.o[u].x = fmaf(w.o[u].x, f, b[u].x); w.o[u].y = fmaf(w.o[u].y, f, b[u].y); w.o[u].z = fmaf(w.o[u].z, f, b[u].z); w.o[u].w = fmaf(w.o[u].w, f, b[u].w);
    }
    __syncwarp();
}

// Tiles of few queries (4 and less: portions of two to four tokens; and tokens that come alone, where they are let in) leave seven of eight warps of the above
// without any. Where a CTA has more than one range of such a tile, a warp takes half a range by itself, keys and values straight from the pages, and the
// ranges' sums wait in the place of the copies until they are merged, in the same order and to the same bits. Bound by the latency of a page's rows (twelve
// reads of a lane under way, eight for values). (Steps of two layers, 8 heads of 128, window 1024, behind 1500 keys, us: a CTA per token and head / tiles /
// here: ten sequences of two tokens 357 / 375 / 289, five 291 / 319 / 273, ten of four 429 / 374 / 288; eight lone tokens beside two 293 / 326 / 271, seven beside 20 382 / 427 / 351,
// fifteen beside 40 of 4 heads of 64 and a window of 300 289 / 299 / 259. Values read one by one in blocks at a window's edge: 353 where 271 stand.)
// CTAs x: the tiles from `first_tile` on, `cluster` for each 32 rows, then one for each of the `n_alone` tiles ahead of them.
__global__ void __launch_bounds__(WT_WARPS * 32, 1) window_attn_tile_kernel(WindowAttnArgs a, RaggedDev r, int first_tile, int cluster, int n_alone) {
    griddep_launch();
    griddep_wait();
    extern __shared__ __align__(16) float wt_sm[];
    const int tiled = (r.n_tiles - first_tile) * 2 * cluster, lone = (int)blockIdx.x - tiled;
    if (lone >= n_alone) return;
    const int d = a.d, ldk = d + 4, own_rank = blockIdx.x % cluster, rank = lone >= 0 ? 0 : own_rank, x = blockIdx.x / cluster, tile = lone >= 0 ? lone : first_tile + x / 2;
    const int h = blockIdx.y, g = h / (a.H / a.G);
    const int seg = r.tile_seg[tile], row0 = r.tile_row0[tile] + (lone >= 0 ? 0 : (x & 1) * WT_Q);
    const int nq = min(WT_Q, r.seg_start[seg] + r.seg_len[seg] - row0);
    if (nq <= 0) return;                                   // (all of a cluster)
    float* qs = wt_sm;                                     // [32][d + 4]
    float* ks = qs + WT_Q * ldk;                           // [2][64][d + 4]
    float* vs = ks + 2 * WT_K * ldk;                       // [2][64][d]
    float* ps = vs + 2 * WT_K * d;                         // [half, warp][32 keys][4 queries]
    const int warp = threadIdx.x >> 5 & 7, half = threadIdx.x >> 8, own = half * WT_OWN, lane = threadIdx.x & 31, kg = lane >> 2, part = lane & 3, w16 = threadIdx.x >> 5;
    const int p0 = r.seg_pos0[seg] + row0 - r.seg_start[seg], p_last = p0 + nq - 1;
    const int* table = a.block_tables[r.seg_slot[seg]];
    const float *k_pool = reinterpret_cast<const float*>(a.k_pool), *v_pool = reinterpret_cast<const float*>(a.v_pool);
    // key blocks: those of the kept prefix, then those of the window
    const int lo_first = max(0, p0 - a.window + 1), n_kept = lo_first > 0 ? (min(a.keep_first, lo_first) + WT_K - 1) / WT_K : 0;
    const int w0 = max(lo_first / WT_K, n_kept), w1 = p_last / WT_K + 1;
    // ranges that have any, in order; block `i` of all (the first of a range: the number of blocks before it)
    const int kept_ranges = (n_kept + WT_RANGE - 1) / WT_RANGE, w_range = max(w0 / WT_RANGE, kept_ranges), n_ranges = kept_ranges + max(0, (w1 - 1) / WT_RANGE + 1 - w_range);
    const int company = n_ranges > 1 && lone < 0 ? cluster : 1;      // (one range: one CTA)
    if (rank >= company) return;
    auto body = [&](auto is_few) {
        constexpr bool few = is_few;
        // sums of a range [half][row][d], and their maxima and sums of weights [half][row]. Rows: 32 queries, or (few) 16 ranges' 4 queries, in the place of the copies
        const int rows = few ? WT_SLOTS * WT_FEW : WT_Q;
        float* xs = few ? ks : ps + WT_WARPS * WT_OWN * 4;
        float2* xml = reinterpret_cast<float2*>(xs + 2 * rows * d);
        auto first_of = [&](int n) {
            const int at = (n < kept_ranges ? n : w_range + n - kept_ranges) * WT_RANGE;
            return min(at, n_kept) + max(0, min(at, w1) - w0);
        };
        auto end_of = [&](int n) {
            const int at = ((n < kept_ranges ? n : w_range + n - kept_ranges) + 1) * WT_RANGE;
            return min(at, n_kept) + max(0, min(at, w1) - w0);
        };
        auto block_at = [&](int i) { return (i < n_kept ? i : w0 + i - n_kept) * WT_K; };
        const int per = d / 4;
        // eight threads a row of a block, whose page is looked up a block ahead of its copies
        const int my_row = threadIdx.x / 8, my_c = threadIdx.x % 8 * 4;
        int next_range = rank, next = !few && rank < n_ranges ? first_of(rank) : -1, next_end = rank < n_ranges ? end_of(rank) : 0;      // of this CTA's blocks: the one to copy next
        auto page_of_next = [&]() { return next >= 0 ? table[min(block_at(next) + my_row, p_last) / a.block_tokens] : 0; };
        int page = page_of_next();
        auto stage = [&](int buf) {                            // keys past the last query's are zeros (their weights are)
            if (next < 0) return;
            const int pos = block_at(next) + my_row;
            const bool have = pos <= p_last;
            const size_t from = have ? (((size_t)page * a.G + g) * a.block_tokens + pos % a.block_tokens) * d : 0;
            if (++next == next_end) {
                next_range += company;
                next = next_range < n_ranges ? first_of(next_range) : -1;
                next_end = next_range < n_ranges ? end_of(next_range) : 0;
            }
            page = page_of_next();
            float *kd = ks + (buf * WT_K + my_row) * ldk, *vd = vs + (buf * WT_K + my_row) * d;
            for (int c = my_c; c < d; c += 32) {
                cp_async_16z(kd + c, k_pool + from + c, have ? 16 : 0);
                cp_async_16z(vd + c, v_pool + from + c, have ? 16 : 0);
            }
        };
        for (int e = threadIdx.x; e < (few ? WT_FEW : WT_Q) * per; e += WT_WARPS * 32) {      // (rows past the tile: the last one's, dropped at the end)
            const int q = e / per, c = e % per * 4;
            const float4 v = *reinterpret_cast<const float4*>(a.q_rot + ((size_t)(row0 + min(q, nq - 1)) * a.H + h) * d + c);
            *reinterpret_cast<float4*>(qs + q * ldk + c) = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
        }
        stage(0);
        cp_async_commit();
        if (few) __syncthreads();                              // (the queries are here; the others meet at every block)
        const int first = p0 + (few ? 0 : warp * 4), pos = first + part, lo = max(0, pos - a.window + 1);      // of the query whose scores this lane ends up with
        float* pw = ps + (half * 8 + warp) * WT_OWN * 4;
        auto start = [](WtSums& w) {
            w.m = -INFINITY; w.l = 0.f;
#pragma unroll
            for (int u = 0; u < 4; u++) w.o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto leave = [&](WtSums& w, int row) {                 // a range's sums, to rows `row` ... of its half
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) w.l += __shfl_xor_sync(0xffffffffu, w.l, x);
            if (4 * lane < d)
#pragma unroll
                for (int u = 0; u < 4; u++) *reinterpret_cast<float4*>(xs + (half * rows + row + u) * d + 4 * lane) = w.o[u];
            if (kg == 0) xml[half * rows + row + part] = make_float2(w.m, w.l);
        };
        // state over ranges: this warp has queries rank + company * (its number of 16, and 16 more)
        float M[2] = {-INFINITY, -INFINITY}, L[2] = {0.f, 0.f};
        float4 O[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        int count = 0;
        const int slots = few ? WT_SLOTS : 1;
        for (int n0 = 0; n0 < n_ranges; n0 += company * slots) {
            WtSums w;
            if constexpr (few) {
                for (int slot = warp; slot < WT_SLOTS; slot += 8) {
                    const int n = n0 + slot * company + rank;
                    if (n >= n_ranges) break;
                    start(w);
                    const int i0 = first_of(n), i1 = end_of(n);
                    auto row_of = [&](int i) {                     // of this lane's key (keys past the last query: that one's, whose weight is dropped)
                        const int j = min(block_at(i) + own + lane, p_last);
                        return ((unsigned)table[j / a.block_tokens] * a.G + g) * a.block_tokens + j % a.block_tokens;
                    };
                    unsigned ahead = row_of(i0);
                    for (int i = i0; i < i1; i++) {
                        const int j0 = block_at(i) + own;
                        const unsigned at = ahead;
                        if (i + 1 < i1) ahead = row_of(i + 1);
                        const float* k_at[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) k_at[u] = k_pool + (size_t)__shfl_sync(0xffffffffu, at, kg * 4 + u) * d + part * 4;
                        const float* v_lane = v_pool + (4 * lane < d ? 4 * lane : 0);
                        wt_add_half<3>(w, a, qs + part * 4, ldk, pw, j0, pos, lo, first, lane, [&](int u, int c) { return *reinterpret_cast<const float4*>(k_at[u] + c); },
                                    [&](int jj) { return *reinterpret_cast<const float4*>(v_lane + (size_t)__shfl_sync(0xffffffffu, at, jj) * d); });
                    }
                    leave(w, slot * WT_FEW);
                }
            } else {
                const int n = n0 + rank, i0 = n < n_ranges ? first_of(n) : 0, i1 = n < n_ranges ? end_of(n) : 0;
                start(w);
                for (int i = i0; i < i1; i++) {
                    const int buf = count++ & 1, j0 = block_at(i) + own;
                    cp_async_wait_all();
                    __syncthreads();                           // this block has come, everybody has left the other buffer
                    stage(buf ^ 1);
                    cp_async_commit();
                    if (warp * 4 >= nq) continue;              // (none of the tile's)
                    const float *kr = ks + (buf * WT_K + own + kg * 4) * ldk + part * 4, *vr = vs + (buf * WT_K + own) * d + (4 * lane < d ? 4 * lane : 0);
                    wt_add_half<1>(w, a, qs + warp * 4 * ldk + part * 4, ldk, pw, j0, pos, lo, first, lane, [&](int u, int c) { return *reinterpret_cast<const float4*>(kr + u * ldk + c); },
                                [&](int jj) { return *reinterpret_cast<const float4*>(vr + jj * d); });
                }
                if (n < n_ranges) leave(w, warp * 4);
            }
            if (company > 1) cluster_sync();
            else __syncthreads();
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int q = rank + company * (w16 + WT_WARPS * k);
                if (q >= nq) break;
                for (int i = 0; i < company * slots && n0 + i < n_ranges; i++) {
                    const int c = i & (company - 1), row = few ? (i >> __ffs(company) - 1) * WT_FEW + q : q;
                    const int of = lone < 0 ? c : own_rank;
                    const uint32_t at = cluster_address(smem_u32(xs + row * d + (4 * lane < d ? 4 * lane : 0)), of), at_ml = cluster_address(smem_u32(xml + row), of);
                    const float2 x0 = cluster_load2(at_ml), x1 = cluster_load2(at_ml + rows * 8);
                    const float4 y0 = cluster_load4(at), y1 = cluster_load4(at + rows * d * 4);
                    const float top = fmaxf(M[k], fmaxf(x0.x, x1.x)), ref = top > -INFINITY ? top : 0.f;      // (nothing visible yet: all factors are 0)
                    const float f = expf(M[k] - ref), f0 = expf(x0.x - ref), f1 = expf(x1.x - ref);
                    M[k] = top;
                    L[k] = fmaf(L[k], f, fmaf(x0.y, f0, x1.y * f1));
                    O[k].x = fmaf(O[k].x, f, fmaf(y0.x, f0, y1.x * f1)); O[k].y = fmaf(O[k].y, f, fmaf(y0.y, f0, y1.y * f1));
                    O[k].z = fmaf(O[k].z, f, fmaf(y0.z, f0, y1.z * f1)); O[k].w = fmaf(O[k].w, f, fmaf(y0.w, f0, y1.w * f1));
                }
            }
            if (company > 1) cluster_sync();                       // (nobody overwrites, or leaves, what another still reads)
            else __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int q = rank + company * (w16 + WT_WARPS * k);
            if (q < nq && 4 * lane < d)
                *reinterpret_cast<float4*>(a.out + ((size_t)(row0 + q) * a.H + h) * d + 4 * lane) = make_float4(O[k].x / L[k], O[k].y / L[k], O[k].z / L[k], O[k].w / L[k]);
        }
    };
    if (nq <= WT_FEW && n_ranges > company) body(std::true_type{});
    else body(std::false_type{});
}
// Heads of whole 16-entry pieces up to 128, rows on 16-byte boundaries.
static bool window_attn_tiles(const WindowAttnArgs& a, int T) {
    return a.cache_f32 && T > 8 && a.d % 16 == 0 && a.d <= WT_D && ((reinterpret_cast<uintptr_t>(a.q_rot) | reinterpret_cast<uintptr_t>(a.out)) & 15) == 0;
}

cudaError_t window_attn_launch(const WindowAttnArgs& a, const RaggedDev& r, cudaStream_t s) {
    if (a.d > ATT_MAXE * 32 || (a.out_rounded && !window_attn_leaves_rounded(a, r.T))) return cudaErrorInvalidValue;
    if (window_attn_mma(a, r.T)) {
        const SoftmaxTcArgs x = window_softmax_args(a);
        if (softmax_takes_tc(x)) return softmax_tc_launch(x, r, s);
        if (!allow_smem<window_attn_mma_kernel<128>>(4 * 64 * (128 + 8) * 2)) return cudaErrorInvalidValue;
        const size_t smem = (size_t)4 * 64 * (a.d + 8) * 2;
        if (a.d <= 64) return launch_chain(window_attn_mma_kernel<64>, dim3(r.n_tiles, a.H), dim3(128), smem, s, a, r);
        return launch_chain(window_attn_mma_kernel<128>, dim3(r.n_tiles, a.H), dim3(128), smem, s, a, r);
    }
    const int alone = r.n_upto[0];                         // (tokens that come alone: a CTA per token and head, below)
    const bool tiles = window_attn_tiles(a, r.T) && r.n_tiles > alone;
    if (tiles) {
        constexpr int most = ((WT_Q + 2 * WT_K) * (WT_D + 4) + 2 * WT_K * WT_D + WT_WARPS * WT_OWN * 4 + 2 * WT_Q * (WT_D + 2)) * 4;
        if (!allow_smem<window_attn_tile_kernel>(most)) return cudaErrorInvalidValue;
        const size_t smem = (size_t)((WT_Q + 2 * WT_K) * (a.d + 4) + 2 * WT_K * a.d + WT_WARPS * WT_OWN * 4 + 2 * WT_Q * (a.d + 2)) * 4;
        // as many CTAs a tile as fit side by side in clusters (of 2: 148, of 8: 128), and no more than a window has ranges
        const int ranges = (int)std::min<long long>(8, ((long long)a.window + a.keep_first + WT_Q) / (WT_RANGE * WT_K) + 2);
        auto company_of = [&](int n) {
            int c = 1;
            while (c < 8 && c < ranges && n * a.H * c * 2 <= (c == 1 ? 148 : 128)) c *= 2;
            return c;
        };
        int n = (r.n_tiles - alone) * 2 - (r.n_upto[5] - alone), first = alone, company = company_of(n), lone = 0;
        auto fits = [&](int c) { return (n * c + (alone + c - 1) / c * c) * a.H <= 128; };
        if (alone > 0 && r.n_tiles == r.n_upto[2] && r.n_tiles * a.H <= (ranges < 8 ? 1 : 4) * 148) {
            // none of more than four tokens: those that come alone are tiles like the others (eight beside two: 271 us, with one CTA each 317). Several waves
            // of them where a window holds enough ranges to keep their warps busy (16 heads of 128, 31 beside two behind 1500: window 1024 591 us apart
            // from the others, 490 as tiles; window 300 376, 397)
            first = 0; n = r.n_tiles; company = company_of(n);
        } else if (alone > 0 && (fits(company) || (company > 1 && fits(company / 2)))) {
            // a CTA for each of them beside the tiles, or beside half as many for each tile. (Where they do not fit they take a launch of their own, which holds
            // many to an SM: fifteen beside 256 1145 us with a CTA per token and head, 622 so)
            if (!fits(company)) company /= 2;
            lone = alone;
        }
        const dim3 grid((r.n_tiles - first) * 2 * company + (lone + company - 1) / company * company, a.H), block(WT_WARPS * 32);
        const cudaError_t e = company > 1 ? launch_chain_cluster(window_attn_tile_kernel, company, grid, block, smem, s, a, r, first, company, lone)
                                          : launch_chain(window_attn_tile_kernel, grid, block, smem, s, a, r, first, company, lone);
        const bool joined = first == 0 || lone > 0;
        if (e != cudaSuccess || joined) return e;
    }
    if (a.d % 2 == 0) {
        // a step of a few tokens does not fill the GPU with one CTA per (token, head): split the keys (up to 16 ranges)
        int splits = 1;
        if (a.split_scratch && r.T * a.H < 148) {
            splits = std::min(16, (2 * 148) / (r.T * a.H));
            while (splits > 1 && (size_t)r.T * a.H * splits * (a.d + 2) > (size_t)a.split_capacity) splits--;
        }
        const dim3 grid(tiles ? alone : r.T, a.H, splits);
        cudaError_t ce = a.cache_f32 ? launch_chain(window_attn_pairs_kernel<true>, grid, dim3(ATT2_WARPS * 32), 0, s, a, r, tiles ? 1 : 0)
                                     : launch_chain(window_attn_pairs_kernel<false>, grid, dim3(ATT2_WARPS * 32), 0, s, a, r, 0);
        if (ce != cudaSuccess || splits == 1) return ce;
        return launch_chain(window_attn_merge_kernel, dim3(grid.x, a.H), dim3(128), 0, s, a, r, splits, tiles ? 1 : 0);
    }
    return launch_chain(window_attn_kernel, dim3(r.T, a.H), dim3(ATT_WARPS * 32), 0, s, a, r);
}

// ---------------------------------------------------------------- selective scan
// xc[t][c] = silu(bias[c] + sum_j w[c][j] * in[t - (taps-1) + j][c]); inputs before the segment come from the slot's state
__global__ void __launch_bounds__(256) scan_conv_kernel(ScanArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x;
    const int seg = r.tok_seg[t], slot = r.seg_slot[seg], i = t - r.seg_start[seg];
    const int hist = a.taps - 1;
    for (int c = threadIdx.x; c < a.inner; c += blockDim.x) {
        float acc = a.conv_b[c];
        for (int j = 0; j < a.taps; j++) {
            const int srci = i - hist + j;
            const float v = srci >= 0 ? a.proj[(size_t)(t - i + srci) * a.ldp + a.x_off + c]
                                      : a.conv_state[((size_t)slot * a.inner + c) * hist + (hist + srci)];
            acc = fmaf(a.conv_w[(size_t)c * a.taps + j], v, acc);
        }
        const float y = silu_inline(acc);
        a.xc[(size_t)t * a.inner + c] = y;
        if (a.xc_rounded) a.xc_rounded[(size_t)t * a.inner + c] = __float2bfloat16(y);
    }
}
// The usual tap counts: a thread makes SCV_T consecutive tokens of one channel, whose inputs it reads once and all ahead of the first
// use. Runs inside one sequence and past its first taps - 1 tokens, nearly all of them, look at no state and no segment. (2048 tokens of 8192
// channels: 120 us with a thread per token and channel, 65 with runs that all looked for their state (117 instructions an output), 40 here,
// with the copy that is left rounded for the next product.)
constexpr int SCV_T = 8;
template <int TAPS>
__global__ void __launch_bounds__(256) scan_conv_taps_kernel(ScanArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    constexpr int hist = TAPS - 1;
    const int t0 = blockIdx.x * SCV_T, c = blockIdx.y * 256 + threadIdx.x;
    if (c >= a.inner) return;
    float w[TAPS], v[SCV_T + hist];
#pragma unroll
    for (int j = 0; j < TAPS; j++) w[j] = a.conv_w[(size_t)c * TAPS + j];
    const float* from = a.proj + (long)(t0 - hist) * a.ldp + a.x_off + c;
#pragma unroll
    for (int k = 0; k < SCV_T + hist; k++, from += a.ldp) {
        const int t = t0 + k - hist;
        v[k] = t >= 0 && t < r.T ? *from : 0.f;
    }
    const float bias = a.conv_b[c];
    float* xc = a.xc + (size_t)t0 * a.inner + c;
    __nv_bfloat16* xb = a.xc_rounded ? a.xc_rounded + (size_t)t0 * a.inner + c : nullptr;
    auto put = [&](float acc) {
        const float y = silu_inline(acc);
        *xc = y;
        xc += a.inner;
        if (xb) { *xb = __float2bfloat16(y); xb += a.inner; }
    };
    const int seg0 = r.tok_seg[t0];
    if (t0 + SCV_T <= r.T && r.tok_seg[t0 + SCV_T - 1] == seg0 && t0 - r.seg_start[seg0] >= hist) {
#pragma unroll
        for (int k = 0; k < SCV_T; k++) {
            float acc = bias;
#pragma unroll
            for (int j = 0; j < TAPS; j++) acc = fmaf(w[j], v[k + j], acc);
            put(acc);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < SCV_T; k++) {
        const int t = t0 + k;
        if (t >= r.T) break;
        const int seg = r.tok_seg[t], i = t - r.seg_start[seg];
        float acc = bias;
#pragma unroll
        for (int j = 0; j < TAPS; j++) {
            const int src = i - hist + j;
            const float in = src >= 0 ? v[k + j] : a.conv_state[((size_t)r.seg_slot[seg] * a.inner + c) * hist + hist + src];
            acc = fmaf(w[j], in, acc);
        }
        put(acc);
    }
}
cudaError_t scan_conv_launch(const ScanArgs& a, const RaggedDev& r, cudaStream_t s) {
    // steps of a few tokens have too few runs of SCV_T to spread over: a CTA per token
    if (r.T >= 64 && a.taps >= 2 && a.taps <= 4) {
        const dim3 grid((r.T + SCV_T - 1) / SCV_T, (a.inner + 255) / 256);
        if (a.taps == 2) return launch_chain(scan_conv_taps_kernel<2>, grid, dim3(256), 0, s, a, r);
        if (a.taps == 3) return launch_chain(scan_conv_taps_kernel<3>, grid, dim3(256), 0, s, a, r);
        return launch_chain(scan_conv_taps_kernel<4>, grid, dim3(256), 0, s, a, r);
    }
    return launch_chain(scan_conv_kernel, dim3(r.T), dim3(256), 0, s, a, r);
}

// grid (n_seg, inner / 8): a warp per channel, lanes over the states (SCAN_MAXS per lane)
constexpr int SCAN_MAXS = 8;       // state size <= 256
__global__ void __launch_bounds__(256) scan_recurrence_kernel(ScanArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    const int seg = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.y * 8 + warp;
    if (c >= a.inner) return;
    const int slot = r.seg_slot[seg], start = r.seg_start[seg], len = r.seg_len[seg];
    const int hist = a.taps - 1;
    // the convolution's memory moves on: the last taps-1 inputs of the sequence (read before written: index k + len > k)
    if (lane == 0) {
        float* st = a.conv_state + ((size_t)slot * a.inner + c) * hist;
        for (int k = 0; k < hist; k++) {
            const int srci = len + k - hist;
            st[k] = srci >= 0 ? a.proj[(size_t)(start + srci) * a.ldp + a.x_off + c] : st[k + len];
        }
    }
    float A[SCAN_MAXS], S[SCAN_MAXS];
    float* sst = a.ssm_state + ((size_t)slot * a.inner + c) * a.N;
#pragma unroll
    for (int e = 0; e < SCAN_MAXS; e++) {
        const int n = lane + 32 * e;
        A[e] = n < a.N ? -expf(a.A_log[(size_t)c * a.N + n]) : 0.f;
        S[e] = n < a.N ? sst[n] : 0.f;
    }
    const float Dc = a.D[c], dtb = a.dt_bias[c];
    for (int i = 0; i < len; i++) {
        const int t = start + i;
        const float dt = softplus_f(a.dt_raw[(size_t)t * a.inner + c] + dtb);
        const float xv = a.xc[(size_t)t * a.inner + c];
        const float* Bp = a.xproj + (size_t)t * a.ldx + a.R;
        const float* Cp = Bp + a.N;
        float part = 0.f;
#pragma unroll
        for (int e = 0; e < SCAN_MAXS; e++) {
            const int n = lane + 32 * e;
            if (n < a.N) {
                S[e] = expf(dt * A[e]) * S[e] + dt * xv * Bp[n];
                part = fmaf(S[e], Cp[n], part);
            }
        }
        const float yv = warp_sum(part) + Dc * xv;
        if (lane == 0) a.y[(size_t)t * a.inner + c] = yv * silu_f(a.proj[(size_t)t * a.ldp + a.z_off + c]);
    }
#pragma unroll
    for (int e = 0; e < SCAN_MAXS; e++) { const int n = lane + 32 * e; if (n < a.N) sst[n] = S[e]; }
}
// Small states (N <= NMAX <= 64): a thread per channel keeps its N states in registers, the step's B and C rows are staged in
// shared memory for a block of tokens, and the next token's inputs are fetched while the current one is computed. No
// shuffles, every global access is coalesced over the channels. grid (n_seg, inner / SCAN_CH).
constexpr int SCAN_CH = 64, SCAN_TB = 16;
template <int NMAX>
__global__ void __launch_bounds__(SCAN_CH) scan_recurrence_chan_kernel(ScanArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    extern __shared__ float bc[];          // [SCAN_TB][2 N]
    const int seg = blockIdx.x, c = blockIdx.y * SCAN_CH + threadIdx.x;
    const bool ok = c < a.inner;
    const int cc = ok ? c : a.inner - 1;    // idle threads shadow the last channel (they still take part in the barriers)
    const int slot = r.seg_slot[seg], start = r.seg_start[seg], len = r.seg_len[seg];
    const int hist = a.taps - 1, N = a.N;
    if (ok) {
        float* st = a.conv_state + ((size_t)slot * a.inner + c) * hist;
        for (int k = 0; k < hist; k++) {
            const int srci = len + k - hist;
            st[k] = srci >= 0 ? a.proj[(size_t)(start + srci) * a.ldp + a.x_off + c] : st[k + len];
        }
    }
    float A[NMAX], S[NMAX];
    float* sst = a.ssm_state + ((size_t)slot * a.inner + cc) * N;
#pragma unroll
    for (int n = 0; n < NMAX; n++) {
        A[n] = n < N ? -expf(a.A_log[(size_t)cc * N + n]) : 0.f;
        S[n] = n < N ? sst[n] : 0.f;
    }
    const float Dc = a.D[cc], dtb = a.dt_bias[cc];
    float n_dt = a.dt_raw[(size_t)start * a.inner + cc], n_x = a.xc[(size_t)start * a.inner + cc];
    float n_z = a.proj[(size_t)start * a.ldp + a.z_off + cc];
    for (int i0 = 0; i0 < len; i0 += SCAN_TB) {
        const int nb = min(SCAN_TB, len - i0);
        __syncthreads();
        for (int j = threadIdx.x; j < nb * 2 * N; j += SCAN_CH) {
            const int tt = j / (2 * N), e = j % (2 * N);
            bc[j] = a.xproj[(size_t)(start + i0 + tt) * a.ldx + a.R + e];
        }
        __syncthreads();
        for (int ii = 0; ii < nb; ii++) {
            const int t = start + i0 + ii;
            const float dt = softplus_f(n_dt + dtb), xv = n_x, zv = n_z;
            if (i0 + ii + 1 < len) {
                n_dt = a.dt_raw[(size_t)(t + 1) * a.inner + cc];
                n_x = a.xc[(size_t)(t + 1) * a.inner + cc];
                n_z = a.proj[(size_t)(t + 1) * a.ldp + a.z_off + cc];
            }
            const float* Bp = bc + ii * 2 * N;
            const float* Cp = Bp + N;
            const float dx = dt * xv;
            float yv = 0.f;
#pragma unroll
            for (int n = 0; n < NMAX; n++)
                if (n < N) {
                    S[n] = expf(dt * A[n]) * S[n] + dx * Bp[n];
                    yv = fmaf(S[n], Cp[n], yv);
                }
            if (ok) a.y[(size_t)t * a.inner + c] = (yv + Dc * xv) * silu_f(zv);
        }
    }
    if (ok) {
#pragma unroll
        for (int n = 0; n < NMAX; n++) if (n < N) sst[n] = S[n];
    }
}

// States up to a warp wide (N <= 32): four or eight lanes per channel, two or four states each (lane q: states q, q + LANES, ...), so that
// what a token costs beside its states -- inputs, loop, read-out -- is paid once per lane, not once per state. A CTA owns blockDim / LANES <=
// SC_CH channels, as few (8 at least) as give every SM one. Blocks of SC_TB tokens (step size, convolved input and gate of its channels, the B
// and C rows, ordered so that a lane's states are one read) arrive in shared memory as asynchronous copies two blocks ahead; softplus(dt +
// bias) and silu(z) are applied once per entry, a block ahead. Every global access is a run of the CTA's channels. What a token does to a
// channel is the same wherever the token stands in a step.
// Bound by its instructions and shared reads: 2048 tokens of 8192 channels with 16 states keep 70 % of the issue slots and 57 % of the shared-memory
// pipe busy (ncu), three to four warps a scheduler; the exponentials alone would take 70 us. The same on a B200: 995 us with a lane per state, 416 with
// four lanes and softplus and gate in a phase of their own, 273 here. (The decays stay expf: one approximate power of two each takes 248 us, but errs to one
// side, and the states sum that up. Step sizes 0.01 to 0.02, A 0.5 to 1, 4000 tokens: output off by 6.8e-7 of its norm, 1.7e-7 here; step sizes
// 0.001 to 0.1, A 1 to 16, 2048 tokens: 1.19e-7 and 0.84e-7.)
constexpr int SC_CH = 64, SC_TB = 16;
template <int LANES, int SPL>
__global__ void __launch_bounds__(SC_CH * LANES) scan_recurrence_lanes_kernel(ScanArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    constexpr int ROW = LANES * 2 * SPL;                 // a token's B and C: per lane its states' B, then their C
    extern __shared__ __align__(16) float sc_smem[];
    float2* dd = reinterpret_cast<float2*>(sc_smem);     // [3][SC_TB][SC_CH]: dt, x as they come; then step size, step size times x
    const int step = blockDim.x, n_ch = step / LANES;
    constexpr int blk = SC_TB * SC_CH;
    float2* gh = dd + 3 * blk;                           // the same of z, -; then gate, x
    float* bc = reinterpret_cast<float*>(gh + 3 * blk);  // [3][SC_TB][ROW]
    const int seg = blockIdx.x, q = threadIdx.x % LANES, lc = threadIdx.x / LANES, c0 = blockIdx.y * n_ch, c = c0 + lc;
    const int N = a.N;
    const bool c_ok = c < a.inner;
    const int cc = c_ok ? c : a.inner - 1;
    const int slot = r.seg_slot[seg], start = r.seg_start[seg], len = r.seg_len[seg];
    const int hist = a.taps - 1;
    if (c_ok && q == 0) {
        float* st = a.conv_state + ((size_t)slot * a.inner + c) * hist;
        for (int k = 0; k < hist; k++) {
            const int srci = len + k - hist;
            st[k] = srci >= 0 ? a.proj[(size_t)(start + srci) * a.ldp + a.x_off + c] : st[k + len];
        }
    }
    float* sst = a.ssm_state + ((size_t)slot * a.inner + cc) * N;
    float A[SPL], S[SPL];
#pragma unroll
    for (int j = 0; j < SPL; j++) {
        const int n = q + LANES * j;
        A[j] = n < N ? -expf(a.A_log[(size_t)cc * N + n]) : 0.f;
        S[j] = n < N && c_ok ? sst[n] : 0.f;
    }
    const int fch = threadIdx.x % n_ch, fu = threadIdx.x / n_ch, fcc = min(c0 + fch, a.inner - 1);      // the channel this thread fetches for, every LANES-th token
    // (channels past the end: nothing. Many lanes that copy one address took the last CTA 346 us where the others took 244.)
    const bool f_ok = c0 + fch < a.inner;
    const float dtb = a.dt_bias[fcc], Dc = a.D[cc];
    if (N < LANES * SPL) {                               // states past the end stay zero (what idle channels hold goes nowhere)
        for (int j = threadIdx.x; j < 3 * SC_TB * ROW; j += step) bc[j] = 0.f;
        __syncthreads();
    }
    // the next block's first entries of this thread: its channel's inputs, and one column of the B and C rows (threads past the last whole token fetch none)
    const int bc_e = threadIdx.x % (2 * N), bc_u = threadIdx.x / (2 * N), bc_du = step / (2 * N), bc_n = bc_e < N ? bc_e : bc_e - N;
    const int bc_at = bc_n % LANES * 2 * SPL + (bc_e < N ? 0 : SPL) + bc_n / LANES;
    const float *g_dt = a.dt_raw + (size_t)(start + fu) * a.inner + fcc, *g_x = a.xc + (size_t)(start + fu) * a.inner + fcc;
    const float *g_z = a.proj + (size_t)(start + fu) * a.ldp + a.z_off + fcc, *g_bc = a.xproj + (size_t)(start + bc_u) * a.ldx + a.R + bc_e;
    const size_t by_inner = (size_t)LANES * a.inner, by_ldp = (size_t)LANES * a.ldp, by_bc = (size_t)bc_du * a.ldx;
    auto stage = [&](int i0, int buf) {                  // blocks in order
        const int nb = min(SC_TB, len - i0);
        float2 *d = dd + buf * blk + fu * SC_CH + fch, *g = gh + buf * blk + fu * SC_CH + fch;
#pragma unroll
        for (int u = 0; u < SC_TB; u += LANES) {
            if (f_ok && u + fu < nb) {
                cp_async_4(&d[u * SC_CH].x, g_dt);
                cp_async_4(&d[u * SC_CH].y, g_x);
                cp_async_4(&g[u * SC_CH].x, g_z);
            }
            g_dt += by_inner; g_x += by_inner; g_z += by_ldp;
        }
        float* w = bc + buf * SC_TB * ROW + bc_at;
        const float* p = g_bc;
        if (bc_u < bc_du)
            for (int u = bc_u; u < nb; u += bc_du, p += by_bc) cp_async_4(w + u * ROW, p);
        g_bc += SC_TB * (size_t)a.ldx;
    };
    // what this thread fetched of a token, made ready in place
    auto ready = [&](int at) {
        const float2 v = dd[at];
        const float dt = softplus_f(v.x + dtb);
        dd[at] = make_float2(dt, dt * v.y);
        gh[at] = make_float2(silu_inline(gh[at].x), v.y);
    };
    // a token's update of this lane's states; their sum times C
    auto token = [&](const float2* d, const float* b) {
        float2 v = *d;
        float B[SPL], C[SPL];
        if constexpr (SPL == 1) { const float2 w = *reinterpret_cast<const float2*>(b); B[0] = w.x; C[0] = w.y; }
        else {
#pragma unroll
            for (int j = 0; j < 2 * SPL; j += 4) {
                const float4 w = *reinterpret_cast<const float4*>(b + j);
                const float k[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; i++) { if (j + i < SPL) B[(j + i) % SPL] = k[i]; else C[(j + i) % SPL] = k[i]; }
            }
        }
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < SPL; j++) {
            S[j] = fmaf(expf(v.x * A[j]), S[j], v.y * B[j]);
            sum = j == 0 ? S[j] * C[j] : fmaf(S[j], C[j], sum);
        }
        return sum;
    };
    auto store = [&](int t, float y) {
        if (!c_ok) return;
        if (a.y_rounded) a.y_rounded[(size_t)t * a.inner + c] = __float2bfloat16(y);
        else a.y[(size_t)t * a.inner + c] = y;
    };
    stage(0, 0);
    cp_async_commit();
    if (SC_TB < len) stage(SC_TB, 1);
    cp_async_commit();
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    for (int u = fu; u < min(SC_TB, len); u += LANES) ready(u * SC_CH + fch);
    int buf = 0;
    for (int i0 = 0; i0 < len; i0 += SC_TB) {
        const int nb = min(SC_TB, len - i0), next = buf == 2 ? 0 : buf + 1;
        cp_async_wait_all();           // this thread's part of the next block has come; of this block it is ready, everybody's after the barrier
        __syncthreads();
        if (i0 + 2 * SC_TB < len) stage(i0 + 2 * SC_TB, buf == 0 ? 2 : buf - 1);        // everybody has left that buffer
        cp_async_commit();
        // LANES tokens at a time: their exponentials do not wait for one another, and the sums over the lanes are exchanged in halves, each
        // lane ending up with the token it stores. In between, what this thread fetched for one token of the next block is made ready (behind the
        // last block: what stands in that buffer, for nothing; without a branch the two run side by side).
        const float2 *d = dd + buf * blk + lc, *g = gh + buf * blk + lc;
        const float* b = bc + buf * SC_TB * ROW + q * 2 * SPL;
        int u = 0;
        for (; u + LANES <= nb; u += LANES) {
            float part[LANES];
#pragma unroll
            for (int t = 0; t < LANES; t++) part[t] = token(d + (u + t) * SC_CH, b + (u + t) * ROW);
            ready(next * blk + (u + fu) * SC_CH + fch);
#pragma unroll
            for (int w = LANES / 2; w > 0; w >>= 1) {
                const bool up = q & w;
#pragma unroll
                for (int t = 0; t < w; t++) part[t] = (up ? part[t + w] : part[t]) + __shfl_xor_sync(0xffffffffu, up ? part[t] : part[t + w], w);
            }
            const float2 gate = g[(u + q) * SC_CH];
            store(start + i0 + u + q, fmaf(Dc, gate.y, part[0]) * gate.x);
        }
        for (; u < nb; u++) {
            float sum = token(d + u * SC_CH, b + u * ROW);
#pragma unroll
            for (int w = LANES / 2; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            const float2 gate = g[u * SC_CH];
            if (q == 0) store(start + i0 + u, fmaf(Dc, gate.y, sum) * gate.x);
        }
        buf = next;
    }
    if (c_ok) {
#pragma unroll
        for (int j = 0; j < SPL; j++) { const int n = q + LANES * j; if (n < N) sst[n] = S[j]; }
    }
}
template <int LANES, int SPL>
static cudaError_t launch_scan_lanes(const ScanArgs& a, const RaggedDev& r, cudaStream_t s) {
    const int per_sm = (int)(((long)a.inner * r.n_seg + 147) / 148), n_ch = std::min(SC_CH, std::max(8, (per_sm + 7) / 8 * 8));
    constexpr int smem = 3 * SC_TB * (SC_CH * 16 + LANES * 2 * SPL * 4);
    if (!allow_smem<scan_recurrence_lanes_kernel<LANES, SPL>>(smem)) return cudaErrorInvalidValue;
    return launch_chain(scan_recurrence_lanes_kernel<LANES, SPL>, dim3(r.n_seg, (a.inner + n_ch - 1) / n_ch), dim3(n_ch * LANES), smem, s, a, r);
}

bool scan_leaves_rounded(const ScanArgs& a) { return a.N <= 32; }
cudaError_t scan_recurrence_launch(const ScanArgs& a, const RaggedDev& r, cudaStream_t s) {
    if (a.N > SCAN_MAXS * 32 || (a.y_rounded && !scan_leaves_rounded(a))) return cudaErrorInvalidValue;
    PlainLaunch pl;        // latency-bound over the prompt: CTAs spread over all SMs (see kernels.h)
    if (a.N <= 4) return launch_scan_lanes<4, 1>(a, r, s);
    if (a.N <= 8) return launch_scan_lanes<4, 2>(a, r, s);
    if (a.N <= 16) return launch_scan_lanes<8, 2>(a, r, s);
    if (a.N <= 32) return launch_scan_lanes<8, 4>(a, r, s);
    if (a.N <= 64) {
        const dim3 grid(r.n_seg, (a.inner + SCAN_CH - 1) / SCAN_CH), block(SCAN_CH);
        const size_t smem = (size_t)SCAN_TB * 2 * a.N * 4;
        return launch_chain(scan_recurrence_chan_kernel<64>, grid, block, smem, s, a, r);
    }
    return launch_chain(scan_recurrence_kernel, dim3(r.n_seg, (a.inner + 7) / 8), dim3(256), 0, s, a, r);
}

// ---------------------------------------------------------------- matrix memory (mLSTM)
// Everything of the recurrence that the memory itself does not enter, ahead of it: per (sequence, head) the log gates
// i = cap tanh((i + b_i) / cap) and f = logsigmoid(cap tanh((f + b_f) / cap)), the running maximum m_t = max(f + m_(t-1), i) and the two
// factors exp(f + m_(t-1) - m_t) and exp(i - m_t) that a token's update takes. The maximum is one thread's serial chain over a block
// of tokens in shared memory (two dependent operations a token); the rest is one token per thread. Left in place: decay over the
// projection's f column, write weight over its i column; exp(-m_t) in m_scale [T][H].
// Bound by that chain (2048 tokens: 10 us) and, per block of tokens, by a read, two gates and a write in a row: long steps take blocks of 1024
// tokens (57 us in blocks of 256, 28 here).
constexpr int MG_TB = 1024;
__global__ void __launch_bounds__(MG_TB) matrix_mem_gates_kernel(MatrixMemArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    __shared__ float2 g[MG_TB];                // log gates f, i
    __shared__ float ms[MG_TB + 1];
    const int seg = blockIdx.x, h = blockIdx.y, block = blockDim.x, u = threadIdx.x;
    const int slot = r.seg_slot[seg], start = r.seg_start[seg], len = r.seg_len[seg];
    const float ib = a.i_bias[h], fb = a.f_bias[h];
    if (u == 0) ms[0] = a.m[(size_t)slot * a.H + h];
    for (int i0 = 0; i0 < len; i0 += block) {
        const int nb = min(block, len - i0);
        float* p = const_cast<float*>(a.proj) + (size_t)(start + i0 + min(u, nb - 1)) * a.ldp;
        float2 mine = make_float2(0.f, 0.f);
        if (u < nb) {
            const float ri = p[a.i_off + h], rf = p[a.f_off + h];
            mine.y = a.cap * tanhf((ri + ib) / a.cap);
            mine.x = log_sigmoid_f(a.cap * tanhf((rf + fb) / a.cap));
            g[u] = mine;
        }
        __syncthreads();
        if (u == 0) {
            float m = ms[0];
            int k = 0;
            for (; k + 8 <= nb; k += 8) {      // read ahead of the chain
                float2 v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = g[k + j];
#pragma unroll
                for (int j = 0; j < 8; j++) { m = fmaxf(v[j].x + m, v[j].y); ms[k + j + 1] = m; }
            }
            for (; k < nb; k++) { m = fmaxf(g[k].x + m, g[k].y); ms[k + 1] = m; }
        }
        __syncthreads();
        if (u < nb) {
            const float m_new = ms[u + 1];
            p[a.f_off + h] = expf(mine.x + ms[u] - m_new);
            p[a.i_off + h] = expf(mine.y - m_new);
            a.m_scale[(size_t)(start + i0 + u) * a.H + h] = expf(-m_new);
        }
        const float last = ms[nb];
        __syncthreads();
        if (u == 0) ms[0] = last;
    }
    if (u == 0) a.m[(size_t)slot * a.H + h] = ms[0];
}

// grid (n_seg, H, ceil(dv / 32) + 1): a CTA owns 32 columns of one head's d x dv memory, two neighbouring ones and MM_ROWS rows a thread, in
// registers as pairs of rows. A warp is 16 such column pairs by 2 row groups; a token's k and q are read from shared memory as they lie, in pairs of
// rows: a read brings 4 bytes a cycle to every lane, whether lanes want the same or not, so the columns a thread has decide how many reads
// a multiply-add costs. Tokens go in blocks of MM_TB: a state update needs only the thread's own registers, so the block barrier is paid
// once per block -- for the inputs (q, k, v and the two factors of the next block arrive in shared memory as asynchronous copies while this
// block is computed) and for the partial read-outs of the row groups, which all threads then sum in a fixed order.
// The CTA past the last columns carries the normaliser n as one column whose v is 1, and leaves n . q; the division by it waits for
// matrix_mem_out_kernel.
// Bound by multiply-adds (24 pairs a token and warp, two cycles each; 31 % of the pipe's instruction rate) and shared reads (18 cycles a token and
// warp, eight warps a pipe; 44 % of its rate), and by their latency with two warps a scheduler (issue slots 52 %). A 2048-token prompt of 16 heads of 128 x 256 (B200): 966 us with one column a thread, 428 with two columns of 16 rows
// and one warp a scheduler, 315 here (four columns a thread and one warp: 400; two tokens side by side, single multiply-adds: the same).
constexpr int MM_ROWS = 8, MM_COLS = 32, MM_TB = 16, MM_MAX_D = 256;      // (16 warps at most)
__global__ void __launch_bounds__(512, 1) matrix_mem_kernel(MatrixMemArgs a, RaggedDev r) {
    griddep_launch();
    griddep_wait();
    extern __shared__ __align__(16) float sm[];
    const int d = a.d, dv = a.dv, n_warps = blockDim.x / 32;
    const int dp = n_warps * 2 * MM_ROWS, red_tok = 2 * n_warps * MM_COLS;      // rows, with those past the end; partial read-outs of a token
    float* qs = sm;                                // [2][MM_TB][dp]
    float* ks = qs + 2 * MM_TB * dp;               // [2][MM_TB][dp]
    float* vs = ks + 2 * MM_TB * dp;               // [2][MM_TB][MM_COLS]
    float* gs = vs + 2 * MM_TB * MM_COLS;          // [2][MM_TB][2]: write weight, decay
    float* red = gs + 2 * MM_TB * 2;               // [2][MM_TB][2 n_warps][MM_COLS]: partial read-outs of the row groups
    const bool norm_cta = blockIdx.z == gridDim.z - 1;
    const int seg = blockIdx.x, h = blockIdx.y, c0 = norm_cta ? 0 : blockIdx.z * MM_COLS, n_cols = norm_cta ? 1 : min(MM_COLS, dv - c0);
    const int slot = r.seg_slot[seg], start = r.seg_start[seg], len = r.seg_len[seg];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, col = (lane & 15) * 2, row = (warp * 2 + (lane >> 4)) * MM_ROWS;
    // this thread's part of the memory (or, one column, of the normaliser)
    float* Sg = norm_cta ? a.n + ((size_t)slot * a.H + h) * d : a.S + (((size_t)slot * a.H + h) * d) * dv + c0;
    const int lds = norm_cta ? 1 : dv;
    uint64_t S[MM_ROWS / 2][2];
    auto at = [&](int i, int j) { return Sg + (size_t)(row + i) * lds + col + j; };
    auto own = [&](int i, int j) { return row + i < d && col + j < n_cols; };
#pragma unroll
    for (int i = 0; i < MM_ROWS / 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) S[i][j] = f2_pack(own(2 * i, j) ? *at(2 * i, j) : 0.f, own(2 * i + 1, j) ? *at(2 * i + 1, j) : 0.f);
    const float qscale = 1.f / sqrtf((float)d);
    // q and k rows as 16-byte copies where they start on 16 bytes
    const bool wide = d % 4 == 0 && a.ldp % 4 == 0 && a.q_off % 4 == 0 && a.k_off % 4 == 0 && (reinterpret_cast<uintptr_t>(a.proj) & 15) == 0;
    const int per = wide ? d / 4 : d, piece = wide ? 4 : 1;
    const int f_e = (threadIdx.x % per) * piece, f_u = threadIdx.x / per, f_du = blockDim.x / per;      // (only when per divides the CTA)
    const bool even = blockDim.x % per == 0;
    auto stage = [&](int i0, int buf) {                  // tokens i0 .. of the segment into buffer `buf`
        const int nb = min(MM_TB, len - i0);
        auto copy = [&](int u, int e) {
            const float* p = a.proj + (size_t)(start + i0 + u) * a.ldp + h * d + e;
            float *qd = &qs[(buf * MM_TB + u) * dp + e], *kd = &ks[(buf * MM_TB + u) * dp + e];
            if (wide) { cp_async_16z(qd, p + a.q_off, 16); cp_async_16z(kd, p + a.k_off, 16); }
            else { cp_async_4(qd, p + a.q_off); cp_async_4(kd, p + a.k_off); }
        };
        if (even) for (int u = f_u; u < nb; u += f_du) copy(u, f_e);
        else for (int j = threadIdx.x; j < nb * per; j += blockDim.x) copy(j / per, (j % per) * piece);
        for (int j = threadIdx.x; j < nb * MM_COLS; j += blockDim.x) {
            const int u = j / MM_COLS, e = j % MM_COLS;
            const float* p = a.proj + (size_t)(start + i0 + u) * a.ldp;
            if (e < n_cols && !norm_cta) cp_async_4(&vs[(buf * MM_TB + u) * MM_COLS + e], p + a.v_off + h * dv + c0 + e);
            if (e < 2) cp_async_4(&gs[(buf * MM_TB + u) * 2 + e], p + (e == 0 ? a.i_off : a.f_off) + h);
        }
    };
    auto finish = [&](int i0, int buf) {                 // sum over the row groups in a fixed order
        const int nb = min(MM_TB, len - i0), u0 = threadIdx.x / MM_COLS, e = threadIdx.x % MM_COLS;
        if (e >= n_cols) return;
        for (int u = u0; u < nb; u += n_warps) {
            const float* rd = red + (size_t)(buf * MM_TB + u) * red_tok + e;
            float sum = 0.f;
#pragma unroll 8
            for (int w = 0; w < 2 * n_warps; w++) sum += rd[w * MM_COLS];
            const size_t t = start + i0 + u;
            if (norm_cta) a.nq[t * a.H + h] = sum * qscale;
            else a.o_raw[t * a.H * dv + (size_t)h * dv + c0 + e] = sum * qscale;
        }
    };
    // what no copy brings: rows past the end stay zero, the normaliser's one column is 1 (what idle columns hold goes nowhere)
    if (d < dp || norm_cta) {
        if (d < dp) for (int j = threadIdx.x; j < 4 * MM_TB * dp; j += blockDim.x) qs[j] = 0.f;
        if (norm_cta) for (int j = threadIdx.x; j < 2 * MM_TB; j += blockDim.x) vs[j * MM_COLS] = 1.f;
        __syncthreads();
    }
    if (len > 0) stage(0, 0);
    cp_async_commit();
    for (int i0 = 0; i0 < len; i0 += MM_TB) {
        const int nb = min(MM_TB, len - i0), buf = (i0 / MM_TB) & 1;
        cp_async_wait_all();
        __syncthreads();
        if (i0 + MM_TB < len) stage(i0 + MM_TB, buf ^ 1);
        cp_async_commit();
        if (i0 > 0) finish(i0 - MM_TB, buf ^ 1);
        // the next token's row pieces and factors are read while this one is computed: latency hides only behind a warp's own work
        const float *kr = ks + buf * MM_TB * dp + row, *qr = qs + buf * MM_TB * dp + row, *vr = vs + buf * MM_TB * MM_COLS + col, *gr = gs + buf * MM_TB * 2;
        float* out = red + (size_t)buf * MM_TB * red_tok + (warp * 2 + (lane >> 4)) * MM_COLS + col;
        ulonglong2 kn[2], qn[2];
        float2 vn, gn;
        auto fetch = [&]() {
            const ulonglong2 *k = reinterpret_cast<const ulonglong2*>(kr), *q = reinterpret_cast<const ulonglong2*>(qr);
            kn[0] = k[0]; kn[1] = k[1]; qn[0] = q[0]; qn[1] = q[1];
            vn = *reinterpret_cast<const float2*>(vr); gn = *reinterpret_cast<const float2*>(gr);
        };
        fetch();
        uint64_t decay = f2_pack(gn.y, gn.y), vv[2] = {f2_pack(gn.x * vn.x, gn.x * vn.x), f2_pack(gn.x * vn.y, gn.x * vn.y)};
#pragma unroll 4
        for (int u = 0; u < nb; u++) {
            const uint64_t kk[4] = {kn[0].x, kn[0].y, kn[1].x, kn[1].y}, qq[4] = {qn[0].x, qn[0].y, qn[1].x, qn[1].y};
            if (u + 1 < nb) { kr += dp; qr += dp; vr += MM_COLS; gr += 2; }
            fetch();
            float p[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
#pragma unroll
                for (int i = 0; i < 4; i++) S[i][j] = f2_fma(decay, S[i][j], f2_mul(kk[i], vv[j]));
                const uint64_t s0 = f2_fma(S[2][j], qq[2], f2_mul(S[0][j], qq[0])), s1 = f2_fma(S[3][j], qq[3], f2_mul(S[1][j], qq[1]));
                const float2 x = f2_unpack(s0), y = f2_unpack(s1);
                p[j] = (x.x + x.y) + (y.x + y.y);
            }
            *reinterpret_cast<float2*>(out) = make_float2(p[0], p[1]);
            out += red_tok;
            decay = f2_pack(gn.y, gn.y);
            vv[0] = f2_pack(gn.x * vn.x, gn.x * vn.x); vv[1] = f2_pack(gn.x * vn.y, gn.x * vn.y);
        }
    }
    __syncthreads();
    if (len > 0) { const int last0 = (len - 1) / MM_TB * MM_TB; finish(last0, (last0 / MM_TB) & 1); }
#pragma unroll
    for (int i = 0; i < MM_ROWS / 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float2 v = f2_unpack(S[i][j]);
            if (own(2 * i, j)) *at(2 * i, j) = v.x;
            if (own(2 * i + 1, j)) *at(2 * i + 1, j) = v.y;
        }
}

// per (token, head): o = read-out / normaliser; out = o / rms(o) * norm_w * sigmoid(gate). A warp each; a lane keeps its entries (MO_U reads of
// four ahead of the first use) where the head has at most 128 MO_U of them and rows start on 16 bytes, else reads them again. Bound by memory: 100 MB
// for 2048 tokens of 16 x 256 (53 us with a CTA per token and head and one entry a read, 37 here).
constexpr int MO_U = 4;
__global__ void __launch_bounds__(256) matrix_mem_out_kernel(MatrixMemArgs a, int T, int wide) {
    griddep_launch();
    griddep_wait();
    const int lane = threadIdx.x & 31;
    const long i = blockIdx.x * 8l + (threadIdx.x >> 5);
    if (i >= (long)T * a.H) return;
    const int t = (int)(i / a.H), h = (int)(i % a.H);
    const size_t base = (size_t)t * a.H * a.dv + (size_t)h * a.dv;
    const float nq = a.nq[i], m_scale = a.m_scale[i];
    auto inverse = [&] { return 1.f / (fmaxf(fabsf(nq), m_scale) + 1e-6f); };
    const float* gate = a.proj + (size_t)t * a.ldp + a.g_off + h * a.dv;
    const float *o = a.o_raw + base, *w = a.norm_w + h * a.dv;
    float ss = 0.f;
    if (wide) {
        float4 v[MO_U], z[MO_U], n[MO_U];
#pragma unroll
        for (int k = 0; k < MO_U; k++) {
            const int e = (k * 32 + lane) * 4;
            if (e < a.dv) { v[k] = *reinterpret_cast<const float4*>(o + e); z[k] = *reinterpret_cast<const float4*>(gate + e); n[k] = *reinterpret_cast<const float4*>(w + e); }
            else v[k] = z[k] = n[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float inv = inverse();
#pragma unroll
        for (int k = 0; k < MO_U; k++) {
            if (k * 128 >= a.dv) break;
            v[k].x *= inv; v[k].y *= inv; v[k].z *= inv; v[k].w *= inv;
            ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
        }
        const float rinv = 1.f / sqrtf(warp_sum(ss) / (float)a.dv + a.eps);
#pragma unroll
        for (int k = 0; k < MO_U; k++) {
            const int e = (k * 32 + lane) * 4;
            if (e >= a.dv) break;
            const float4 y = make_float4(v[k].x * rinv * n[k].x * sigmoid_f(z[k].x), v[k].y * rinv * n[k].y * sigmoid_f(z[k].y),
                                         v[k].z * rinv * n[k].z * sigmoid_f(z[k].z), v[k].w * rinv * n[k].w * sigmoid_f(z[k].w));
            if (a.out_rounded) store_bf16x4(a.out_rounded + base + e, y);
            else *reinterpret_cast<float4*>(a.out + base + e) = y;
        }
    } else {
        const float inv = inverse();
        for (int e = lane; e < a.dv; e += 32) { const float v = o[e] * inv; ss += v * v; }
        const float rinv = 1.f / sqrtf(warp_sum(ss) / (float)a.dv + a.eps);
        for (int e = lane; e < a.dv; e += 32) {
            const float y = o[e] * inv * rinv * w[e] * sigmoid_f(gate[e]);
            if (a.out_rounded) a.out_rounded[base + e] = __float2bfloat16(y);
            else a.out[base + e] = y;
        }
    }
}

cudaError_t matrix_mem_launch(const MatrixMemArgs& a, const RaggedDev& r, cudaStream_t s) {
    if (a.dv <= 0 || a.d <= 0 || a.d > MM_MAX_D) return cudaErrorInvalidValue;
    cudaError_t ce = launch_chain(matrix_mem_gates_kernel, dim3(r.n_seg, a.H), dim3(r.T >= 512 ? MG_TB : 256), 0, s, a, r);
    if (ce != cudaSuccess) return ce;
    {
        PlainLaunch pl;    // latency-bound over the prompt: CTAs spread over all SMs (see kernels.h)
        const int n_warps = (a.d + 2 * MM_ROWS - 1) / (2 * MM_ROWS);
        const size_t smem = (size_t)2 * MM_TB * (2 * n_warps * 2 * MM_ROWS + MM_COLS + 2 + 2 * n_warps * MM_COLS) * 4;
        if (!allow_smem<matrix_mem_kernel>(200 * 1024)) return cudaErrorInvalidValue;
        ce = launch_chain(matrix_mem_kernel, dim3(r.n_seg, a.H, (a.dv + MM_COLS - 1) / MM_COLS + 1), dim3(n_warps * 32), smem, s, a, r);
    }
    if (ce != cudaSuccess) return ce;
    const uintptr_t rows = reinterpret_cast<uintptr_t>(a.o_raw) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.out_rounded) |
                           reinterpret_cast<uintptr_t>(a.proj) | reinterpret_cast<uintptr_t>(a.norm_w);
    const int wide = a.dv % 4 == 0 && a.dv <= 128 * MO_U && a.ldp % 4 == 0 && a.g_off % 4 == 0 && (rows & 15) == 0;
    return launch_chain(matrix_mem_out_kernel, dim3((unsigned)(((long)r.T * a.H + 7) / 8)), dim3(256), 0, s, a, r.T, wide);
}

}  // namespace b2
