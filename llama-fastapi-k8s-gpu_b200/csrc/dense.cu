// Dense products for the layer-list models: Y[T][N] = epi(X[T][K] . W[N][K]^T + bias), weights bf16 or f32 as stored
// in the file, activations f32 in memory. Five kernels:
//   dense_rows_kernel   T <= 8 (decode steps): one warp per weight row, the row is streamed once for all tokens
//   dense_tc_kernel     T > 8, bf16 weights: tensor cores (dense_tc.cu), X rounded to bf16
//   dense_mma_kernel    the same for rows that tensor copies cannot take (K % 8 != 0): mma.sync m16n8k16 bf16, f32 accumulate
//   dense_split_kernel  T > 8, exact mode, bf16 weights: tensor cores, X as three bf16 parts that add up to it (dense_split.cu)
//   dense_fma_kernel    T > 8, exact mode, weights or rows that the former does not take: 32-bit multiply-adds, nothing rounded
// Every output element is one sum over k in a fixed order that depends only on the matrix and the kernel, never on the
// other rows, so a token's result is the same whatever else shares the step. Arbitrary T, N, K (edges are guarded).
// The llama graph's counterpart (quantised blocks, tcgen05) is gemm.cu / matvec.cu.
#include "kernels.h"
#include "dense_dev.cuh"
#include "layered.h"
#include "ptx.cuh"
#include "quant_blocks.cuh"

#include <algorithm>
#include <array>

namespace b2 {

__device__ __forceinline__ float ld_w(const __nv_bfloat16* w, size_t i) { return __bfloat162float(w[i]); }
__device__ __forceinline__ float ld_w(const float* w, size_t i) { return w[i]; }

// ---------------------------------------------------------------- few tokens: a warp per R weight rows
// TT = compiled token count (1, 2, 4 or 8 >= T), R = rows per warp (the activations a lane loads serve R rows: with several
// tokens the activation loads, not the weights, fill the load pipe). Fast path (K % 8 == 0, 16-byte aligned rows): a lane takes
// 8 consecutive weights per load and keeps R x U = 4 loads in flight, 2 KB per warp on the wire. Each output is still one sum
// over k in an order that depends on K alone.
constexpr int ROWS_MAX_T = 8;
template <typename TW, int TT, int R>
__device__ __forceinline__ void dense_rows_cta(const DenseDev& a, unsigned bx, unsigned by, unsigned bz) {
    constexpr int U = 4 / R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = a.N, K = a.K, ldx = a.ldx;
    const int n0 = (bx * 8 + warp) * R;
    if (n0 >= N) return;
    const float* x; const TW* w; float* y; const float* aux; int t0, t1;
    if (!dense_tile<TW>(a, ROWS_MAX_T, x, w, y, aux, t0, t1, by, bz)) return;
    const int T = a.grouped ? 1 : a.T;
    const float* rs = a.g.row_scale;
    if (a.grouped) { x += (size_t)x_row(a, t0) * ldx; y += (size_t)t0 * a.ldy; if (aux) aux += (size_t)t0 * a.ldaux; if (rs) rs += t0; }
    const TW* rows[R];
#pragma unroll
    for (int r = 0; r < R; r++) rows[r] = w + (size_t)min(n0 + r, N - 1) * K;      // past the end: the last row again, not stored
    float acc[TT][R];
#pragma unroll
    for (int t = 0; t < TT; t++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[t][r] = 0.f;
    const bool vec = (K % 8 == 0) && (ldx % 4 == 0) && ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(x)) & 15) == 0;
    if (vec) {
        auto load8 = [&](const TW* row, int k, float (&wv)[8]) {
            if constexpr (sizeof(TW) == 2) {
                const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(row + k));       // streamed once: do not keep in L1
                const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int i = 0; i < 4; i++) { wv[2 * i] = __uint_as_float(u[i] << 16); wv[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
            } else {
                const float4 a = __ldcs(reinterpret_cast<const float4*>(row + k)), b = __ldcs(reinterpret_cast<const float4*>(row + k + 4));
                wv[0] = a.x; wv[1] = a.y; wv[2] = a.z; wv[3] = a.w; wv[4] = b.x; wv[5] = b.y; wv[6] = b.z; wv[7] = b.w;
            }
        };
        auto fma8 = [&](const float (&wv)[R][8], int k) {
#pragma unroll
            for (int t = 0; t < TT; t++)
                if (t < T) {
                    const float4 a = *reinterpret_cast<const float4*>(x + (size_t)t * ldx + k);
                    const float4 b = *reinterpret_cast<const float4*>(x + (size_t)t * ldx + k + 4);
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        float v = acc[t][r];
                        v = fmaf(a.x, wv[r][0], v); v = fmaf(a.y, wv[r][1], v); v = fmaf(a.z, wv[r][2], v); v = fmaf(a.w, wv[r][3], v);
                        v = fmaf(b.x, wv[r][4], v); v = fmaf(b.y, wv[r][5], v); v = fmaf(b.z, wv[r][6], v); v = fmaf(b.w, wv[r][7], v);
                        acc[t][r] = v;
                    }
                }
        };
        int k = lane * 8;
        for (; k + (U - 1) * 256 < K; k += U * 256) {
            float wv[U][R][8];
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int r = 0; r < R; r++) load8(rows[r], k + u * 256, wv[u][r]);
#pragma unroll
            for (int u = 0; u < U; u++) fma8(wv[u], k + u * 256);
        }
        for (; k < K; k += 256) {
            float wv[R][8];
#pragma unroll
            for (int r = 0; r < R; r++) load8(rows[r], k, wv[r]);
            fma8(wv, k);
        }
    } else {
        // lanes take k = lane, lane + 32, ...: neighbouring lanes read neighbouring weights
        for (int k = lane; k < K; k += 32) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float wv = ld_w(rows[r], k);
#pragma unroll
                for (int t = 0; t < TT; t++)
                    if (t < T) acc[t][r] = fmaf(x[(size_t)t * ldx + k], wv, acc[t][r]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < TT; t++) {
        if (t >= T) continue;
        float v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = warp_sum(acc[t][r]);
        if (lane != 0) continue;
        if constexpr (R % 2 == 0) {
#pragma unroll
            for (int r = 0; r < R; r += 2) epi_store2(a, y, aux, rs, t, n0 + r, v[r], v[r + 1]);
        } else {
            epi_store(a, y, aux, t, n0, v[0]);
        }
    }
}
template <typename TW, int TT, int R>
__global__ void __launch_bounds__(256) dense_rows_kernel(DenseDev a) {
    griddep_launch();
    griddep_wait();
    dense_rows_cta<TW, TT, R>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}
// two independent products in one launch: the CTAs of a, then those of b (grouped pairs, `nb` CTAs each)
template <typename TW, int TT, int R>
__global__ void __launch_bounds__(256) dense_rows_pair_kernel(DenseDev a, DenseDev b, unsigned na, unsigned nb) {
    griddep_launch();
    griddep_wait();
    if (blockIdx.x < na) dense_rows_cta<TW, TT, R>(a, blockIdx.x, 0, 0);
    else dense_rows_cta<TW, 1, 1>(b, (blockIdx.x - na) % nb, (blockIdx.x - na) / nb, 0);
}

template <typename TW>
static cudaError_t launch_rows(const DenseDev& d, int batch, cudaStream_t s) {
    dim3 block(256);
    const unsigned gy = d.grouped ? d.T : 1, gz = d.grouped ? 1 : batch;       // grouped: one pair row per blockIdx.y
    const int N = d.N;
    if (d.grouped || d.T == 1) {
        if (d.epi == EPI_GLU_SILU || d.epi == EPI_GLU_GELU || d.epi == EPI_GLU_CLAMP) return launch_chain(dense_rows_kernel<TW, 1, 2>, dim3((N + 15) / 16, gy, gz), block, 0, s, d);
        return launch_chain(dense_rows_kernel<TW, 1, 1>, dim3((N + 7) / 8, gy, gz), block, 0, s, d);
    }
    if (d.T == 2) return launch_chain(dense_rows_kernel<TW, 2, 2>, dim3((N + 15) / 16, gy, gz), block, 0, s, d);
    if (d.T <= 4) return launch_chain(dense_rows_kernel<TW, 4, 4>, dim3((N + 31) / 32, gy, gz), block, 0, s, d);
    return launch_chain(dense_rows_kernel<TW, 8, 4>, dim3((N + 31) / 32, gy, gz), block, 0, s, d);
}

// ---------------------------------------------------------------- exact: 64 x 64 tile, 32-deep, 4 x 4 per thread
// Bound by the multiply-adds once the loads are out of the way: the next slice of both operands is in registers while the current one
// is used (16-byte loads along K where rows allow), both live in shared memory as rows padded by 16 bytes, and four K steps cost
// eight 16-byte shared loads for 64 multiply-adds. A thread's rows and columns are 16 apart: neighbouring lanes read neighbouring
// rows, on different banks. The order of every sum is that of k.
template <typename TW>
__global__ void __launch_bounds__(256) dense_fma_kernel(DenseDev a) {
    griddep_launch();
    griddep_wait();
    constexpr int BM = 64, BN = 64, BK = 32, LD = BK + 4;
    __shared__ __align__(16) float xs[2][BM][LD];
    __shared__ __align__(16) float ws[2][BN][LD];
    const float* x; const TW* w; float* y; const float* aux; int t0, T;
    if (!dense_tile<TW>(a, BM, x, w, y, aux, t0, T, blockIdx.y, blockIdx.z)) return;
    const int N = a.N, K = a.K, ldx = a.ldx;
    const int n0 = blockIdx.x * BN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;      // rows ty + 16 i, columns tx + 16 j
    // a thread fetches 8 consecutive K entries of one row of each operand
    const int fr = threadIdx.x >> 2, fk = (threadIdx.x & 3) * 8;
    const int xt = t0 + fr, wn = n0 + fr;
    const bool x_in = xt < T, w_in = wn < N;
    const float* xr = x + (size_t)(x_in ? x_row(a, xt) : 0) * ldx;
    const TW* wr = w + (size_t)(w_in ? wn : 0) * K;
    const bool vec = K % 8 == 0 && ldx % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    float xv[8], wv[8];
    auto fetch = [&](int k0) {
        const int k = k0 + fk;
        if (vec) {
            const bool in = k < K;
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
            if (x_in && in) { p = *reinterpret_cast<const float4*>(xr + k); q = *reinterpret_cast<const float4*>(xr + k + 4); }
            xv[0] = p.x; xv[1] = p.y; xv[2] = p.z; xv[3] = p.w; xv[4] = q.x; xv[5] = q.y; xv[6] = q.z; xv[7] = q.w;
            if constexpr (sizeof(TW) == 2) {
                uint4 u = make_uint4(0u, 0u, 0u, 0u);
                if (w_in && in) u = *reinterpret_cast<const uint4*>(wr + k);
                const uint32_t h[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 4; i++) { wv[2 * i] = __uint_as_float(h[i] << 16); wv[2 * i + 1] = __uint_as_float(h[i] & 0xffff0000u); }
            } else {
                p = make_float4(0.f, 0.f, 0.f, 0.f); q = p;
                if (w_in && in) { p = *reinterpret_cast<const float4*>(wr + k); q = *reinterpret_cast<const float4*>(wr + k + 4); }
                wv[0] = p.x; wv[1] = p.y; wv[2] = p.z; wv[3] = p.w; wv[4] = q.x; wv[5] = q.y; wv[6] = q.z; wv[7] = q.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                xv[i] = x_in && k + i < K ? xr[k + i] : 0.f;
                wv[i] = w_in && k + i < K ? ld_w(wr, k + i) : 0.f;
            }
        }
    };
    auto put = [&](int buf) {
        *reinterpret_cast<float4*>(&xs[buf][fr][fk]) = make_float4(xv[0], xv[1], xv[2], xv[3]);
        *reinterpret_cast<float4*>(&xs[buf][fr][fk + 4]) = make_float4(xv[4], xv[5], xv[6], xv[7]);
        *reinterpret_cast<float4*>(&ws[buf][fr][fk]) = make_float4(wv[0], wv[1], wv[2], wv[3]);
        *reinterpret_cast<float4*>(&ws[buf][fr][fk + 4]) = make_float4(wv[4], wv[5], wv[6], wv[7]);
    };
    float acc[4][4] = {};
    fetch(0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float4 p[4], q[4];
#pragma unroll
            for (int i = 0; i < 4; i++) { p[i] = *reinterpret_cast<const float4*>(&xs[buf][ty + 16 * i][kk]); q[i] = *reinterpret_cast<const float4*>(&ws[buf][tx + 16 * i][kk]); }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[i][j] = fmaf(p[i].x, q[j].x, acc[i][j]);
                    acc[i][j] = fmaf(p[i].y, q[j].y, acc[i][j]);
                    acc[i][j] = fmaf(p[i].z, q[j].z, acc[i][j]);
                    acc[i][j] = fmaf(p[i].w, q[j].w, acc[i][j]);
                }
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
    const float* rs = a.g.row_scale;
    const bool glu = a.epi == EPI_GLU_SILU || a.epi == EPI_GLU_GELU || a.epi == EPI_GLU_CLAMP;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + ty + 16 * i;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx + 16 * j;
            const float other = __shfl_xor_sync(0xffffffffu, acc[i][j], 1);      // the neighbouring column
            if (t < T) {
                if (!glu) { if (n < N) epi_store(a, y, aux, t, n, acc[i][j]); }
                else if (!(tx & 1)) epi_store2(a, y, aux, rs, t, n, acc[i][j], other);
            }
        }
    }
}

// ---------------------------------------------------------------- tensor cores: 64 x 64 tile, 32-deep, 4 warps of 32 x 32
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__global__ void __launch_bounds__(128) dense_mma_kernel(DenseDev a) {
    griddep_launch();
    griddep_wait();
    constexpr int BM = 64, BN = 64, BK = 32, LD = BK + 8;      // rows padded by 16 bytes: fragment reads hit 32 banks
    __shared__ __align__(16) __nv_bfloat16 xs[BM][LD];
    __shared__ __align__(16) __nv_bfloat16 ws[BN][LD];
    const float* x; const __nv_bfloat16* w; float* y; const float* aux; int t0, T;
    if (!dense_tile<__nv_bfloat16>(a, BM, x, w, y, aux, t0, T, blockIdx.y, blockIdx.z)) return;
    const int N = a.N, K = a.K, ldx = a.ldx;
    const int n0 = blockIdx.x * BN;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int g = lane >> 2, tq = lane & 3;
    float acc[2][4][4] = {};
    const bool w_vec = (K % 8 == 0) && ((reinterpret_cast<uintptr_t>(w) & 15) == 0);
    for (int k0 = 0; k0 < K; k0 += BK) {
        // X tile: f32 -> bf16 (round to nearest even), 64 x 32
        for (int i = threadIdx.x; i < BM * BK / 2; i += 128) {
            const int r = i / (BK / 2), kk = (i % (BK / 2)) * 2;
            const int t = t0 + r, k = k0 + kk;
            float v0 = 0.f, v1 = 0.f;
            if (t < T) {
                const float* xr = x + (size_t)x_row(a, t) * ldx;
                if (k < K) v0 = xr[k];
                if (k + 1 < K) v1 = xr[k + 1];
            }
            *reinterpret_cast<__nv_bfloat162*>(&xs[r][kk]) = __floats2bfloat162_rn(v0, v1);
        }
        // W tile: 64 rows x 32 bf16
        if (w_vec) {
            for (int i = threadIdx.x; i < BN * BK / 8; i += 128) {
                const int r = i / (BK / 8), kk = (i % (BK / 8)) * 8;
                const int n = n0 + r, k = k0 + kk;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (n < N && k < K) v = *reinterpret_cast<const uint4*>(w + (size_t)n * K + k);
                *reinterpret_cast<uint4*>(&ws[r][kk]) = v;
            }
        } else {
            for (int i = threadIdx.x; i < BN * BK; i += 128) {
                const int r = i / BK, kk = i % BK;
                const int n = n0 + r, k = k0 + kk;
                ws[r][kk] = (n < N && k < K) ? w[(size_t)n * K + k] : __float2bfloat16(0.f);
            }
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < BK; ks += 16) {
            uint32_t af[2][4], bf[4][2];
#pragma unroll
            for (int mi = 0; mi < 2; mi++) {
                const int r = wm + mi * 16 + g;
                af[mi][0] = *reinterpret_cast<const uint32_t*>(&xs[r][ks + 2 * tq]);
                af[mi][1] = *reinterpret_cast<const uint32_t*>(&xs[r + 8][ks + 2 * tq]);
                af[mi][2] = *reinterpret_cast<const uint32_t*>(&xs[r][ks + 2 * tq + 8]);
                af[mi][3] = *reinterpret_cast<const uint32_t*>(&xs[r + 8][ks + 2 * tq + 8]);
            }
#pragma unroll
            for (int ni = 0; ni < 4; ni++) {
                const int c = wn + ni * 8 + g;
                bf[ni][0] = *reinterpret_cast<const uint32_t*>(&ws[c][ks + 2 * tq]);
                bf[ni][1] = *reinterpret_cast<const uint32_t*>(&ws[c][ks + 2 * tq + 8]);
            }
#pragma unroll
            for (int mi = 0; mi < 2; mi++)
#pragma unroll
                for (int ni = 0; ni < 4; ni++) mma_bf16_16816(acc[mi][ni], af[mi], bf[ni]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int mi = 0; mi < 2; mi++)
#pragma unroll
        for (int ni = 0; ni < 4; ni++)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const int t = t0 + wm + mi * 16 + g + (e >> 1) * 8;
                if (t < T) epi_store2(a, y, aux, a.g.row_scale, t, n0 + wn + ni * 8 + 2 * tq, acc[mi][ni][e], acc[mi][ni][e + 1]);
            }
}

// The tcgen05 kernel reads a rounded copy of the input: [T][K]; batched: [T][x_span] with batch b at column b * x_bs; grouped: the rows of
// the sorted pairs. Its operands are tensor maps: rows of whole 16-byte pieces on 16-byte boundaries.
bool dense_takes_rounded(const DenseArgs& a) {
    const int span = a.batch > 1 ? a.x_span : a.K;
    const bool tiled = a.groups && a.groups->tile_group;
    const bool ok = a.w_type == T_BF16 && !a.exact && a.xb && a.K % 8 == 0 && (reinterpret_cast<uintptr_t>(a.w) & 15) == 0 && span % 8 == 0 &&
                    (a.batch == 1 || (a.x_span > 0 && a.x_bs % 8 == 0 && a.w_bs % 8 == 0));
    return ok && (a.groups ? tiled : a.T > ROWS_MAX_T);
}

static DenseDev dense_dev(const DenseArgs& a) {
    DenseDev d = {};
    d.x = a.x; d.ldx = a.ldx; d.w = a.w; d.bias = a.bias; d.y = a.y; d.ldy = a.ldy; d.T = a.T; d.N = a.N; d.K = a.K; d.epi = a.epi;
    d.n_act = a.n_act; d.n_act_end = a.n_act_end; d.yb = a.y_rounded; d.scale = a.scale; d.p0 = a.p0; d.p1 = a.p1;
    d.aux = a.aux; d.ldaux = a.ldaux; d.aux_ns = a.aux_one ? 0 : 1; d.x_bs = a.x_bs; d.w_bs = a.w_bs; d.y_bs = a.y_bs; d.aux_bs = a.aux_bs;
    if (a.groups) { d.g = *a.groups; d.grouped = a.groups->tile_group ? 2 : 1; }
    return d;
}

static bool glu_epi(int epi) { return epi == EPI_GLU_SILU || epi == EPI_GLU_GELU || epi == EPI_GLU_CLAMP; }
bool dense_pairs(const DenseArgs& a, const DenseArgs& b) {
    return !a.groups && a.batch == 1 && a.T >= 1 && a.T <= ROWS_MAX_T && b.groups && !b.groups->tile_group && a.w_type == b.w_type &&
           !glu_epi(a.epi) && !glu_epi(b.epi) && !a.x_rounded && !a.y_rounded && !b.x_rounded && !b.y_rounded;
}
template <typename TW>
static cudaError_t launch_rows_pair(const DenseDev& a, const DenseDev& b, cudaStream_t s) {
    const unsigned per = a.T == 1 ? 8 : a.T == 2 ? 16 : 32, na = (a.N + per - 1) / per, nb = (b.N + 7) / 8;      // rows per CTA as in launch_rows
    const dim3 grid(na + nb * b.T), block(256);
    if (a.T == 1) return launch_chain(dense_rows_pair_kernel<TW, 1, 1>, grid, block, 0, s, a, b, na, nb);
    if (a.T == 2) return launch_chain(dense_rows_pair_kernel<TW, 2, 2>, grid, block, 0, s, a, b, na, nb);
    if (a.T <= 4) return launch_chain(dense_rows_pair_kernel<TW, 4, 4>, grid, block, 0, s, a, b, na, nb);
    return launch_chain(dense_rows_pair_kernel<TW, 8, 4>, grid, block, 0, s, a, b, na, nb);
}
cudaError_t dense_pair_launch(const DenseArgs& a, const DenseArgs& b, cudaStream_t s) {
    if (!dense_pairs(a, b) || a.N <= 0 || a.K <= 0 || b.T <= 0 || b.N <= 0 || b.K <= 0) return cudaErrorInvalidValue;
    return a.w_type == T_BF16 ? launch_rows_pair<__nv_bfloat16>(dense_dev(a), dense_dev(b), s) : launch_rows_pair<float>(dense_dev(a), dense_dev(b), s);
}

cudaError_t dense_launch(const DenseArgs& a, cudaStream_t s) {
    if (a.T <= 0 || a.N <= 0 || a.K <= 0 || a.batch <= 0) return cudaErrorInvalidValue;
    if (a.w_type != T_BF16 && a.w_type != T_F32) return cudaErrorInvalidValue;
    if (glu_epi(a.epi) && a.N % 2) return cudaErrorInvalidValue;
    if (a.groups && a.batch != 1) return cudaErrorInvalidValue;
    const bool wb = a.w_type == T_BF16;
    const DenseDev d = dense_dev(a);
    if (d.grouped == 1 || (!d.grouped && a.T <= ROWS_MAX_T)) return wb ? launch_rows<__nv_bfloat16>(d, a.batch, s) : launch_rows<float>(d, a.batch, s);
    // few output columns in 32-bit (router scores): the tiled kernel would run a handful of CTAs over the whole K; the
    // few-token kernel over chunks of 8 rows keeps every SM busy and streams the small matrix from L2
    if (a.exact && !d.grouped && a.batch == 1 && a.N <= 64) {
        const int chunks = a.T / ROWS_MAX_T, rem = a.T % ROWS_MAX_T;
        DenseDev c = d;
        c.T = ROWS_MAX_T; c.x_bs = (long)ROWS_MAX_T * a.ldx; c.y_bs = (long)ROWS_MAX_T * a.ldy; c.aux_bs = (long)ROWS_MAX_T * a.ldaux; c.w_bs = 0;
        cudaError_t ce = wb ? launch_rows<__nv_bfloat16>(c, chunks, s) : launch_rows<float>(c, chunks, s);
        if (ce != cudaSuccess || rem == 0) return ce;
        c = d;
        c.T = rem; c.x += (size_t)chunks * ROWS_MAX_T * a.ldx; c.y += (size_t)chunks * ROWS_MAX_T * a.ldy;
        if (c.aux) c.aux += (size_t)chunks * ROWS_MAX_T * a.ldaux;
        return wb ? launch_rows<__nv_bfloat16>(c, 1, s) : launch_rows<float>(c, 1, s);
    }
    if (dense_takes_split(a)) return dense_split_launch(a, d, s);
    const unsigned gz = d.grouped ? 1 : a.batch;
    if (dense_takes_rounded(a)) return dense_tc_launch(a, d, s);
    if (a.x_rounded || a.y_rounded || (d.grouped == 2 && a.groups->tile_max != 64)) return cudaErrorInvalidValue;
    dim3 grid((a.N + 63) / 64, d.grouped ? (unsigned)a.groups->max_tiles : (unsigned)((a.T + 63) / 64), gz);
    if (wb && !a.exact) return launch_chain(dense_mma_kernel, grid, dim3(128), 0, s, d);
    if (wb) return launch_chain(dense_fma_kernel<__nv_bfloat16>, grid, dim3(256), 0, s, d);
    return launch_chain(dense_fma_kernel<float>, grid, dim3(256), 0, s, d);
}

}  // namespace b2
