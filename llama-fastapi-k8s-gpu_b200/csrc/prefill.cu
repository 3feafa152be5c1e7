// Prompt-processing (prefill) kernels around the tensor-core GEMM (gemm.cu): T tokens of one sequence at once.
// Replaces the batch > 1 side of ggml-cuda that llama.cpp runs for the prompt under create_chat_completion
// (api.py:55-63): get_rows (K1), rms_norm_f32 (K2), rope_f32 + the KV-cache copy (K6/K7),
// the attention mat-muls + soft_max (K8-K10 at batch T), silu/mul (K11).
//
// f16 activation matrices that feed the GEMM are written in its operand order [K/8][T_pad][8]; the GEMM's
// outputs arrive as n_parts K-split partial sums that the consumer adds in a fixed order.
//   embed_rows      x[t][:]      = dequantised row tokens[t] of the embedding table          (f32)
//   resid_norm_half x[t] += sum(parts); xn[t] = f16( x[t] / sqrt(mean(x[t]^2) + eps) * w )
//   rope_store      sum(parts) -> q rotated f16 [T][n_head*hd]; k rotated, v -> paged f16 KV cache
//   attn_prefill    causal flash attention over the paged cache, mma.sync m16n8k16 (f16 in, f32 accumulate),
//                   one warp per 16 queries of one head, the G heads of a KV group share the K/V tiles
//   silu_mul_half   h[t][:]      = f16( silu(gate) * up )
//   prefill_finish  pushes the prompt tokens into the penalty history and leaves token / position of the
//                   last prompt token in the slot registers
#include "kernels.h"
#include "ptx.cuh"
#include "quant_blocks.cuh"
#include <cuda_fp16.h>

namespace b2 {

// ---------------------------------------------------------------- embedding rows
__global__ void embed_rows_kernel(int type, const uint8_t* table, int K, const int* tokens, float* x) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x;
    const int be = block_elems(type), bb = block_bytes(type);
    const uint8_t* row = table + (size_t)tokens[t] * (K / be) * bb;
    for (int i = threadIdx.x; i < K; i += blockDim.x)
        x[(size_t)t * K + i] = dequant_elem(type, row + (size_t)(i / be) * bb, i % be);
}
cudaError_t embed_rows_launch(int type, const uint8_t* table, int K, const int* tokens, int T, float* x, cudaStream_t s) {
    return launch_chain(embed_rows_kernel, dim3(T), dim3(T > 148 ? 256 : 1024), 0, s, type, table, K, tokens, x);
}

__device__ __forceinline__ size_t op_index(int t, int k, int T_pad) { return ((size_t)(k >> 3) * T_pad + t) * 8 + (k & 7); }

// ---------------------------------------------------------------- residual add + RMSNorm -> f16
constexpr int RN_THREADS = 1024;
__global__ void __launch_bounds__(RN_THREADS) resid_norm_half_kernel(float* x, const float* parts, int n_parts, long part_stride,
                                                                     const float* w, float eps, int K, int T_pad, __half* xn) {
    griddep_launch();
    griddep_wait();
    __shared__ float red[RN_THREADS / 32];
    const int t = blockIdx.x;
    float* xr = x + (size_t)t * K;
    // a thread's float4s stay in registers between the sum of squares and the normalisation (K <= 2 * 4 * RN_THREADS = 8192;
    // longer rows re-read what they wrote)
    constexpr int KEEP = 2;
    float4 keep[KEEP];
    float ss = 0.f;
    auto sum_parts = [&](int i) -> float4 {                             // float4 per thread: the split sums are independent loads
        float4 v = *reinterpret_cast<const float4*>(xr + 4 * i);
        const float* pp = parts + (size_t)t * K + 4 * i;
#pragma unroll 4
        for (int s = 0; s < n_parts; s++) {
            const float4 q = *reinterpret_cast<const float4*>(pp + (size_t)s * part_stride);
            v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
        }
        if (n_parts) *reinterpret_cast<float4*>(xr + 4 * i) = v;
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        return v;
    };
#pragma unroll
    for (int it = 0; it < KEEP; it++) {
        const int i = threadIdx.x + it * RN_THREADS;
        keep[it] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < K / 4) keep[it] = sum_parts(i);
    }
    for (int i = threadIdx.x + KEEP * RN_THREADS; i < K / 4; i += RN_THREADS) sum_parts(i);
    if (!w) return;
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < RN_THREADS / 32; i++) tot += red[i];
    const float r = rsqrtf(tot / (float)K + eps);
    auto emit = [&](int i, const float4& a) {                           // 4 consecutive k = half of a 16-byte run in operand order
        const float4 wa = *reinterpret_cast<const float4*>(w + 4 * i);
        const __half2 h0 = __floats2half2_rn(a.x * r * wa.x, a.y * r * wa.y), h1 = __floats2half2_rn(a.z * r * wa.z, a.w * r * wa.w);
        *reinterpret_cast<uint2*>(xn + ((size_t)(i >> 1) * T_pad + t) * 8 + 4 * (i & 1)) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
    };
#pragma unroll
    for (int it = 0; it < KEEP; it++) {
        const int i = threadIdx.x + it * RN_THREADS;
        if (i < K / 4) emit(i, keep[it]);
    }
    for (int i = threadIdx.x + KEEP * RN_THREADS; i < K / 4; i += RN_THREADS) emit(i, *reinterpret_cast<const float4*>(xr + 4 * i));
}
// The same for long prompts, four tokens a CTA (256 threads each, rows of at most 4096): a thread has four reads of every plane in flight, and the operand
// order's 16-byte pieces of the four tokens lie side by side, so that they leave as 64-byte runs. The sums are those of the kernel above, bit for bit:
// entry i belongs to "thread" i, whose warp sums first. (512 rows of 4096: 12.5 us a row a CTA, which is two waves of one read and one half-filled
// sector each; 8.5 here.)
constexpr int RN_TOK = 4;
__global__ void __launch_bounds__(RN_THREADS) resid_norm_half_rows_kernel(float* x, const float* parts, int n_parts, long part_stride,
                                                                          const float* w, float eps, int K, int T, int T_pad, __half* xn) {
    griddep_launch();
    griddep_wait();
    extern __shared__ __align__(16) uint8_t rn_rows[];                  // [K / 8][RN_TOK][8] f16
    __shared__ float red[RN_TOK][RN_THREADS / 32];
    constexpr int NT = RN_THREADS / RN_TOK, U = 4;
    const int tok = threadIdx.x / NT, j = threadIdx.x % NT, t = blockIdx.x * RN_TOK + tok;
    const bool in = t < T;
    float* xr = x + (size_t)min(t, T - 1) * K;
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int i = j + u * NT;
        v[u] = i < K / 4 ? *reinterpret_cast<const float4*>(xr + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int s = 0; s < n_parts; s++) {
        const float* pp = parts + (size_t)s * part_stride + (size_t)min(t, T - 1) * K;
        float4 q[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = j + u * NT;
            q[u] = i < K / 4 ? *reinterpret_cast<const float4*>(pp + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < U; u++) { v[u].x += q[u].x; v[u].y += q[u].y; v[u].z += q[u].z; v[u].w += q[u].w; }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int i = j + u * NT;
        if (n_parts && in && i < K / 4) *reinterpret_cast<float4*>(xr + 4 * i) = v[u];
        float ss = 0.f;
        ss += v[u].x * v[u].x + v[u].y * v[u].y + v[u].z * v[u].z + v[u].w * v[u].w;
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) red[tok][(j + u * NT) / 32] = ss;
    }
    if (!w) return;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < RN_THREADS / 32; i++) tot += red[tok][i];
    const float r = rsqrtf(tot / (float)K + eps);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int i = j + u * NT;
        if (i >= K / 4) break;
        const float4 wa = *reinterpret_cast<const float4*>(w + 4 * i);
        const __half2 h0 = __floats2half2_rn(v[u].x * r * wa.x, v[u].y * r * wa.y), h1 = __floats2half2_rn(v[u].z * r * wa.z, v[u].w * r * wa.w);
        *reinterpret_cast<uint2*>(rn_rows + ((size_t)(i >> 1) * RN_TOK + tok) * 16 + 8 * (i & 1)) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < K / 8 * RN_TOK; i += RN_THREADS) {
        const int to = blockIdx.x * RN_TOK + i % RN_TOK;
        if (to < T) *reinterpret_cast<uint4*>(xn + ((size_t)(i / RN_TOK) * T_pad + to) * 8) = *reinterpret_cast<const uint4*>(rn_rows + (size_t)i * 16);
    }
}
cudaError_t resid_norm_half_launch(float* x, const float* parts, int n_parts, long part_stride, const float* w, float eps,
                                   int K, int T, int T_pad, __half* xn, cudaStream_t s) {
    // from where a CTA per token no longer fits two to an SM; below, a row's latency is all there is
    if (T >= 256 && K % 8 == 0 && K <= 4 * RN_THREADS)
        return launch_chain(resid_norm_half_rows_kernel, dim3((T + RN_TOK - 1) / RN_TOK), dim3(RN_THREADS), (size_t)K * RN_TOK * 2, s, x, parts, n_parts, part_stride, w, eps, K, T, T_pad, xn);
    return launch_chain(resid_norm_half_kernel, dim3(T), dim3(RN_THREADS), 0, s, x, parts, n_parts, part_stride, w, eps, K, T_pad, xn);
}

// ---------------------------------------------------------------- RoPE + KV store
// parts: [T][n_head*hd | n_kv*hd | n_kv*hd] f32. Pair (2i, 2i+1) rotated by pos * freq[i] (ggml "norm" RoPE). A CTA per token; the position's
// hd / 2 turns are made once, while the row's sums are on their way (a sincosf per pair and head before: 512 tokens 11.5 -> 9 us, 32 slots 8.4 -> 6.5).
template <typename StoreQ>
__device__ __forceinline__ void rope_row(const float* r, int n_parts, long part_stride, int pos, int page, int n_head, int n_kv, int hd, int bt,
                                         const float* rope_freq, __half* k_cache, __half* v_cache, StoreQ store_q) {
    __shared__ float2 turn[128];                             // cos, sin; hd <= 256
    constexpr int U = 2;
    const unsigned nq = n_head * hd, nk = n_kv * hd, units = (nq + 2 * nk) / 4, slot = pos % bt;      // a unit: two pairs
    bool ready = false;
    for (unsigned u0 = threadIdx.x; u0 - threadIdx.x < units; u0 += U * blockDim.x) {
        float4 v[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const unsigned i = u0 + k * blockDim.x;
            v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i >= units) continue;
#pragma unroll 4
            for (int s = 0; s < n_parts; s++) {
                const float4 q = *reinterpret_cast<const float4*>(r + (size_t)s * part_stride + 4 * i);
                v[k].x += q.x; v[k].y += q.y; v[k].z += q.z; v[k].w += q.w;
            }
        }
        if (!ready) {
            if (2 * threadIdx.x < hd) {
                float sn, cs;
                sincosf((float)pos * rope_freq[threadIdx.x], &sn, &cs);
                turn[threadIdx.x] = make_float2(cs, sn);
            }
            __syncthreads();
            ready = true;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
            const unsigned i = u0 + k * blockDim.x, e = 4 * i;
            if (i >= units) continue;
            if (e < nq + nk) {
                const float2 c0 = turn[e % hd / 2], c1 = turn[e % hd / 2 + 1];
                v[k] = make_float4(v[k].x * c0.x - v[k].y * c0.y, v[k].x * c0.y + v[k].y * c0.x, v[k].z * c1.x - v[k].w * c1.y, v[k].z * c1.y + v[k].w * c1.x);
            }
            if (e < nq) { store_q(e, v[k]); continue; }
            const unsigned ee = e < nq + nk ? e - nq : e - nq - nk, kvh = ee / hd, d = ee % hd;
            const __half2 h0 = __floats2half2_rn(v[k].x, v[k].y), h1 = __floats2half2_rn(v[k].z, v[k].w);
            *reinterpret_cast<uint2*>((e < nq + nk ? k_cache : v_cache) + (((size_t)page * n_kv + kvh) * bt + slot) * hd + d) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
        }
    }
}
__global__ void __launch_bounds__(1024) rope_store_kernel(const float* parts, int n_parts, long part_stride, int T, int pos0, int n_head, int n_kv,
                                                          int hd, int bt, const int* block_table, const float* rope_freq, __half* qh,
                                                          __half* k_cache, __half* v_cache) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x, pos = pos0 + t, nq = n_head * hd;
    rope_row(parts + (size_t)t * (nq + 2 * n_kv * hd), n_parts, part_stride, pos, block_table[pos / bt], n_head, n_kv, hd, bt, rope_freq, k_cache, v_cache,
             [&](unsigned e, const float4& v) {
                 const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
                 *reinterpret_cast<uint2*>(qh + (size_t)t * nq + e) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
             });
}
cudaError_t rope_store_launch(const float* parts, int n_parts, long part_stride, int T, int pos0, int n_head, int n_kv, int hd,
                              int bt, const int* block_table, const float* rope_freq, __half* qh, __half* k_cache,
                              __half* v_cache, cudaStream_t s) {
    if (hd % 4 || hd > 256 || part_stride % 4) return cudaErrorInvalidValue;
    return launch_chain(rope_store_kernel, dim3(T), dim3(T > 148 ? 512 : 1024), 0, s, parts, n_parts, part_stride, T, pos0, n_head, n_kv, hd, bt, block_table, rope_freq, qh, k_cache, v_cache);
}

// ---------------------------------------------------------------- SiLU(gate) * up -> f16
__global__ void silu_mul_half_kernel(const float* parts, int n_parts, long part_stride, int F, int T, int T_pad, __half* h) {
    griddep_launch();
    griddep_wait();
    // thread <-> (8 consecutive f, token): one 16-byte store in operand order. A warp is 8 such pieces of f by 4 tokens: rows are read in runs of 256
    // bytes and the pieces leave in runs of 64 (32 tokens by one piece, a row each, read 32 bytes here and there: 512 tokens 27 us, 15 here)
    const int lane = threadIdx.x & 31, t = blockIdx.y * 4 + (lane >> 3), ch = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 8 + (lane & 7);
    if (t >= T || ch >= F / 8) return;
    float g[8] = {0, 0, 0, 0, 0, 0, 0, 0}, u[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int s = 0; s < n_parts; s++) {
        const float* row = parts + (size_t)s * part_stride + (size_t)t * 2 * F + ch * 8;
        const float4 g0 = *reinterpret_cast<const float4*>(row), g1 = *reinterpret_cast<const float4*>(row + 4);
        const float4 u0 = *reinterpret_cast<const float4*>(row + F), u1 = *reinterpret_cast<const float4*>(row + F + 4);
        g[0] += g0.x; g[1] += g0.y; g[2] += g0.z; g[3] += g0.w; g[4] += g1.x; g[5] += g1.y; g[6] += g1.z; g[7] += g1.w;
        u[0] += u0.x; u[1] += u0.y; u[2] += u0.z; u[3] += u0.w; u[4] += u1.x; u[5] += u1.y; u[6] += u1.z; u[7] += u1.w;
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float a = g[2 * j] / (1.f + __expf(-g[2 * j])) * u[2 * j], b = g[2 * j + 1] / (1.f + __expf(-g[2 * j + 1])) * u[2 * j + 1];
        const __half2 hh = __floats2half2_rn(a, b);
        o[j] = *reinterpret_cast<const uint32_t*>(&hh);
    }
    *reinterpret_cast<uint4*>(h + ((size_t)ch * T_pad + t) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}
cudaError_t silu_mul_half_launch(const float* parts, int n_parts, long part_stride, int F, int T, int T_pad, __half* h, cudaStream_t s) {
    return launch_chain(silu_mul_half_kernel, dim3((F / 8 + 63) / 64, (T + 3) / 4), dim3(256), 0, s, parts, n_parts, part_stride, F, T, T_pad, h);
}

// ---------------------------------------------------------------- batched decode step: one token per slot
// (a token that the caller has set, and its position, go into the slot's registers here)
__global__ void embed_batch_kernel(int type, const uint8_t* table, int K, const SlotDev* tab, const BatchIdx b, const BatchTokens set, float* x) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x, given = set.token[t];
    int* ints = tab[b.slot[t]].ints;
    const int tok = given >= 0 ? given : ints[0];
    if (given >= 0 && threadIdx.x == 0) { ints[0] = given; ints[1] = set.pos[t]; }
    const int be = block_elems(type), bb = block_bytes(type);
    const uint8_t* row = table + (size_t)tok * (K / be) * bb;
    for (int i = threadIdx.x; i < K; i += blockDim.x)
        x[(size_t)t * K + i] = dequant_elem(type, row + (size_t)(i / be) * bb, i % be);
}
cudaError_t embed_batch_launch(int type, const uint8_t* table, int K, const SlotDev* tab, const BatchIdx& b, const BatchTokens& set, float* x, cudaStream_t s) {
    return launch_chain(embed_batch_kernel, dim3(b.n), dim3(1024), 0, s, type, table, K, tab, b, set, x);
}

// like rope_store, but row t belongs to slot b.slot[t] at that slot's own position; q stays float32 for flash-decode
__global__ void __launch_bounds__(1024) rope_store_batch_kernel(const float* parts, int n_parts, long part_stride, const SlotDev* tab, const BatchIdx b,
                                                                int n_head, int n_kv, int hd, int bt, const float* rope_freq, float* q_out,
                                                                __half* k_cache, __half* v_cache) {
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x;
    const SlotDev sd = tab[b.slot[t]];
    const int pos = sd.ints[1], nq = n_head * hd;
    rope_row(parts + (size_t)t * (nq + 2 * n_kv * hd), n_parts, part_stride, pos, sd.block_table[pos / bt], n_head, n_kv, hd, bt, rope_freq, k_cache, v_cache,
             [&](unsigned e, const float4& v) { *reinterpret_cast<float4*>(q_out + (size_t)t * nq + e) = v; });
}
cudaError_t rope_store_batch_launch(const float* parts, int n_parts, long part_stride, const SlotDev* tab, const BatchIdx& b,
                                    int n_head, int n_kv, int hd, int bt, const float* rope_freq, float* q_out,
                                    __half* k_cache, __half* v_cache, cudaStream_t s) {
    if (hd % 4 || hd > 256 || part_stride % 4) return cudaErrorInvalidValue;
    return launch_chain(rope_store_batch_kernel, dim3(b.n), dim3(1024), 0, s, parts, n_parts, part_stride, tab, b, n_head, n_kv, hd, bt, rope_freq, q_out, k_cache, v_cache);
}

// ---------------------------------------------------------------- slot registers after a prompt chunk
__global__ void prefill_finish_kernel(const int* prompt, int n, int pos_last, int* ints, SamplerState* st) {
    griddep_launch();
    griddep_wait();
    // only the last HISTORY_LEN tokens stay in the ring: one thread each (one thread walking 512 tokens took 27 us)
    const int nh = st->n_hist, i = n - HISTORY_LEN + (int)threadIdx.x;
    if (i >= 0) st->history[(nh + i) & (HISTORY_LEN - 1)] = prompt[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        st->n_hist = nh + n;
        ints[0] = prompt[n - 1];
        ints[1] = pos_last;
    }
}
cudaError_t prefill_finish_launch(const int* prompt, int n, int pos_last, int* ints, SamplerState* st, cudaStream_t s) {
    return launch_chain(prefill_finish_kernel, dim3(1), dim3(HISTORY_LEN), 0, s, prompt, n, pos_last, ints, st);
}

// ---------------------------------------------------------------- causal attention for T queries
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void cp_async_16(void* dst, const void* src, bool have) {       // zeros where there is nothing to read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

constexpr int PA_KT = 64;        // keys per tile

// grid (query tiles, n_kv), the tiles with the most keys first; block = G * QW warps: warp w -> head kvh*G + w % G, queries 16 * (w / G) .. +15 of the
// tile. The next tile of keys and values arrives as asynchronous copies while one is used. Bound by the chain of a tile's scores, softmax and sums,
// four warps a CTA. (512 tokens, 32 heads of 128: 44 us with one buffer and single fragment reads, 29.5 here, the same bits.)
template <int HD>
__global__ void __launch_bounds__(256) attn_prefill_kernel(const __half* qh, const __half* k_cache, const __half* v_cache,
                                                           const int* block_table, int T, int T_pad, int pos0, int n_head,
                                                           int n_kv, int bt, int QW, float scale_log2, __half* out) {
    griddep_launch();
    griddep_wait();
    constexpr int LD = HD + 8;                                  // padded row: conflict-free fragment loads
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __half* const kv = reinterpret_cast<__half*>(smem_raw);     // [2][keys, values][PA_KT][LD]
    const int G = n_head / n_kv, q_tile = gridDim.x - 1 - blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int kvh = blockIdx.y, head = kvh * G + warp % G;
    const int q0 = q_tile * 16 * QW + 16 * (warp / G);          // first query (chunk-relative) of this warp
    const int nq = n_head * HD;
    const bool active = q0 < T;

    // Q fragments: rows q0+g and q0+g+8 (clamped; rows >= T are dropped at the end)
    uint32_t qa[HD / 16][4];
    {
        const int r0 = min(q0 + g, T - 1), r1 = min(q0 + g + 8, T - 1);
        const __half* p0 = qh + (size_t)r0 * nq + head * HD, * p1 = qh + (size_t)r1 * nq + head * HD;
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
            qa[kk][0] = *reinterpret_cast<const uint32_t*>(p0 + kk * 16 + 2 * tq);
            qa[kk][1] = *reinterpret_cast<const uint32_t*>(p1 + kk * 16 + 2 * tq);
            qa[kk][2] = *reinterpret_cast<const uint32_t*>(p0 + kk * 16 + 8 + 2 * tq);
            qa[kk][3] = *reinterpret_cast<const uint32_t*>(p1 + kk * 16 + 8 + 2 * tq);
        }
    }
    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;   // running max / sum of rows g, g+8 (log2 domain)

    // keys needed by the CTA: positions 0 .. pos0 + (last query of the tile)
    const int last_q = min(q_tile * 16 * QW + 16 * QW - 1, T - 1);
    const int n_keys = pos0 + last_q + 1;
    const int my_last = pos0 + min(q0 + 15, T - 1);             // last key this warp needs
    auto stage = [&](int k0, int buf) {
        __half *ks = kv + (size_t)buf * 2 * PA_KT * LD, *vs = ks + PA_KT * LD;
        for (int i = threadIdx.x; i < PA_KT * (HD / 8); i += blockDim.x) {
            const int j = i / (HD / 8), ch = i % (HD / 8), pos = k0 + j;
            const bool have = pos < n_keys;
            const size_t base = have ? (((size_t)block_table[pos / bt] * n_kv + kvh) * bt + pos % bt) * HD + ch * 8 : 0;
            cp_async_16(ks + j * LD + ch * 8, k_cache + base, have);
            cp_async_16(vs + j * LD + ch * 8, v_cache + base, have);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, 0);
    for (int k0 = 0, buf = 0; k0 < n_keys; k0 += PA_KT, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                        // this tile has come; everybody has left the other buffer
        if (k0 + PA_KT < n_keys) stage(k0 + PA_KT, buf ^ 1);
        if (!active || k0 > my_last) continue;
        const __half *ks = kv + (size_t)buf * 2 * PA_KT * LD, *vs = ks + PA_KT * LD;
        // ---- S = Q K^T for 64 keys: 8 n-tiles of 8 keys
        float sc[PA_KT / 8][4];
#pragma unroll
        for (int nt = 0; nt < PA_KT / 8; nt++) {
            sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
            const __half* kr = ks + (nt * 8 + (lane & 7)) * LD + (lane >> 3) * 8;
#pragma unroll
            for (int kk = 0; kk < HD / 16; kk += 2) {
                uint32_t b[4];                                  // dims kk * 16 .. + 31 of eight keys
                ldmatrix_x4(b, kr + kk * 16);
                mma16816(sc[nt], qa[kk], b[0], b[1]);
                mma16816(sc[nt], qa[kk + 1], b[2], b[3]);
            }
        }
        // ---- causal mask + online softmax (rows g and g+8; columns 2tq, 2tq+1 of every n-tile)
        const int p_row0 = pos0 + q0 + g, p_row1 = p_row0 + 8;
        float mx0 = m0, mx1 = m1;
#pragma unroll
        for (int nt = 0; nt < PA_KT / 8; nt++) {
            const int kp = k0 + nt * 8 + 2 * tq;
            sc[nt][0] = kp <= p_row0 ? sc[nt][0] * scale_log2 : -INFINITY;
            sc[nt][1] = kp + 1 <= p_row0 ? sc[nt][1] * scale_log2 : -INFINITY;
            sc[nt][2] = kp <= p_row1 ? sc[nt][2] * scale_log2 : -INFINITY;
            sc[nt][3] = kp + 1 <= p_row1 ? sc[nt][3] * scale_log2 : -INFINITY;
            mx0 = fmaxf(mx0, fmaxf(sc[nt][0], sc[nt][1]));
            mx1 = fmaxf(mx1, fmaxf(sc[nt][2], sc[nt][3]));
        }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        // key 0 is visible to every query, so after the first tile the maxima are finite
        const float f0 = exp2f(m0 - mx0), f1 = exp2f(m1 - mx1);
        m0 = mx0; m1 = mx1;
        float s0 = 0.f, s1 = 0.f;
        uint32_t pa[PA_KT / 16][4];
#pragma unroll
        for (int nt = 0; nt < PA_KT / 8; nt++) {
            const float e0 = exp2f(sc[nt][0] - mx0), e1 = exp2f(sc[nt][1] - mx0);
            const float e2 = exp2f(sc[nt][2] - mx1), e3 = exp2f(sc[nt][3] - mx1);
            s0 += e0 + e1; s1 += e2 + e3;
            pa[nt >> 1][(nt & 1) * 2 + 0] = pack_half2(e0, e1);
            pa[nt >> 1][(nt & 1) * 2 + 1] = pack_half2(e2, e3);
        }
        l0 = l0 * f0 + s0; l1 = l1 * f1 + s1;
#pragma unroll
        for (int i = 0; i < HD / 8; i++) { o[i][0] *= f0; o[i][1] *= f0; o[i][2] *= f1; o[i][3] *= f1; }
        // ---- O += P V : k = keys (4 k-tiles of 16), n = head dims (HD / 8 n-tiles)
#pragma unroll
        for (int kt = 0; kt < PA_KT / 16; kt++) {
#pragma unroll
            for (int nt = 0; nt < HD / 8; nt += 2) {
                // 16 keys x 16 dims, transposed on load
                uint32_t b[4];
                ldmatrix_x4_trans(b, vs + (kt * 16 + (lane & 15)) * LD + nt * 8 + (lane >> 4) * 8);
                mma16816(o[nt], pa[kt], b[0], b[1]);
                mma16816(o[nt + 1], pa[kt], b[2], b[3]);
            }
        }
    }
    if (!active) return;
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    const float i0 = 1.f / l0, i1 = 1.f / l1;
    const int r0 = q0 + g, r1 = q0 + g + 8;
#pragma unroll
    for (int nt = 0; nt < HD / 8; nt++) {
        const int d = head * HD + nt * 8 + 2 * tq;      // column of the [T][n_head*hd] matrix, stored in operand order
        if (r0 < T) *reinterpret_cast<uint32_t*>(out + op_index(r0, d, T_pad)) = pack_half2(o[nt][0] * i0, o[nt][1] * i0);
        if (r1 < T) *reinterpret_cast<uint32_t*>(out + op_index(r1, d, T_pad)) = pack_half2(o[nt][2] * i1, o[nt][3] * i1);
    }
}

cudaError_t attn_prefill_launch(const __half* qh, const __half* k_cache, const __half* v_cache, const int* block_table,
                                int T, int T_pad, int pos0, int n_head, int n_kv, int hd, int bt, __half* out, cudaStream_t s) {
    if (n_kv <= 0 || n_head % n_kv) return cudaErrorInvalidValue;
    const int G = n_head / n_kv;
    if (G > 8) return cudaErrorInvalidValue;
    const int QW = G >= 4 ? 1 : 4 / G;
    const int q_tile = 16 * QW;
    dim3 grid((T + q_tile - 1) / q_tile, n_kv), block(32 * G * QW);
    const float scale_log2 = 1.4426950408889634f / sqrtf((float)hd);
    const size_t smem = (size_t)2 * 2 * PA_KT * (hd + 8) * 2;
    if (!allow_smem<attn_prefill_kernel<128>>(4 * PA_KT * (128 + 8) * 2)) return cudaErrorInvalidValue;
    if (hd == 64) return launch_chain(attn_prefill_kernel<64>, grid, block, smem, s, qh, k_cache, v_cache, block_table, T, T_pad, pos0, n_head, n_kv, bt, QW, scale_log2, out);
    if (hd == 128) return launch_chain(attn_prefill_kernel<128>, grid, block, smem, s, qh, k_cache, v_cache, block_table, T, T_pad, pos0, n_head, n_kv, bt, QW, scale_log2, out);
    return cudaErrorInvalidValue;
}

}  // namespace b2
