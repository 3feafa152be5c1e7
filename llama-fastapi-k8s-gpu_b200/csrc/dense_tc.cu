// Dense products of more than 8 tokens on the 5th-generation tensor cores:
//     Y[t][n] = epi(sum_k X[t][k] * W[n][k])      X rounded to bf16 [rows][K], W bf16 [N][K], f32 sums in tensor memory.
//
// Both operands come by 3-D tensor copies (K, row, batch entry or expert) of 64-wide K slices into a ring of 128-byte-swizzled
// stages; rows and K past the end arrive as zeros. Six warps: 0-3 epilogue (one tensor-memory lane a thread), 4 copies, 5 matrix
// instructions. A CTA walks its tiles with two accumulators, so the epilogue of a tile runs under the products of the next one.
//
// Two orientations:
//   long steps    weights are the MMA's A operand (128 rows = the 128 lanes of tensor memory), tokens its N (up to 256 columns): an
//                 epilogue warp writes 32 neighbouring outputs of one token per store.
//   short steps   (at most 256 tokens, and the 64-row tiles of experts) tokens are the A operand, weight rows the N, as few a tile
//                 (16 at least) as spread a matrix over all SMs: these products are bound by the weight stream, and 128-row tiles of
//                 a 2048-row matrix would leave 132 of 148 SMs idle. K is not split, so each sum keeps its order whatever the step.
// (bf16 products of 2048 tokens, start of these figures: 128 x 128 tiles of mma.sync. 4096 wide layer pass of mLSTM + attention/scan/feed-forward:
// products 4.9 -> 1.3 ms; 32 sequences of 1 token: a 2048 x 2048 product 60 -> 7 us; the sums are the same bit for bit.)
// The weights of the first stages are requested before the dependency wait: they do not depend on the previous kernel.
#include "dense_tc.cuh"
#include "quant_blocks.cuh"
#include "tc05.cuh"
#include "tensor_map.h"

#include <algorithm>

namespace b2 {

constexpr int TC_MAX_STAGES = 24;
constexpr int TC_THREADS = 192;
constexpr int TC_SMEM = TC_RING + TC_M * TC_K * 2 + 1024;      // + what a short step's MMA reads past the last stage, alignment

// short steps: 16 (or fewer) weight rows n.. of token t, which is this lane's; `have`: the lane has a token
template <int EPI, bool ROUNDED>
__device__ __forceinline__ void tc_store_rows(const DenseDev& a, float* y, __nv_bfloat16* yb, const float* aux, bool have, int n, int n_end, int t,
                                              const float (&acc)[16]) {
    constexpr bool GLU = EPI == EPI_GLU_SILU || EPI == EPI_GLU_GELU || EPI == EPI_GLU_CLAMP;
    if (!have) return;
    float v[16];
    if constexpr (GLU) {
        const float s = a.g.row_scale ? a.g.row_scale[t] : 1.f;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            float gate = acc[j], up = acc[j + 1];
            if (a.g.row_scale) { gate *= s; up *= s; }
            if (EPI == EPI_GLU_CLAMP) {
                const float g = fminf(gate, a.p0), u = fminf(fmaxf(up, -a.p0), a.p0);
                v[j >> 1] = g / (1.f + expf(-a.p1 * g)) * (u + 1.f);
            } else v[j >> 1] = (EPI == EPI_GLU_SILU ? silu_act(gate) : gelu_tanh_act(gate)) * up;
            v[j >> 1] *= a.scale;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int c = min(n + j, a.N - 1);
            v[j] = acc[j];
            if ((EPI == EPI_BIAS || EPI == EPI_BIAS_RELU2 || EPI == EPI_BIAS_PART_RELU2) && a.bias) v[j] += a.bias[c];
            if (EPI == EPI_BIAS_RELU2 || (EPI == EPI_BIAS_PART_RELU2 && c >= a.n_act && c < a.n_act_end)) { v[j] = fmaxf(v[j], 0.f); v[j] = v[j] * v[j]; }
            if (EPI == EPI_MUL_SIGMOID) v[j] *= sigmoid_act(aux[(size_t)t * a.ldaux + c * a.aux_ns]);
            if (EPI == EPI_PIECEWISE) v[j] = v[j] > 0.f ? fmaf(a.p0 * v[j], v[j], 0.5f * v[j]) : fmaf(a.p1, expm1f(v[j]) - v[j], 0.5f * v[j]);
            v[j] *= a.scale;
        }
    }
    constexpr int W = GLU ? 8 : 16;                               // outputs of the 16 rows
    const int c0 = GLU ? n >> 1 : n, left = (GLU ? n_end >> 1 : n_end) - c0;
    if constexpr (ROUNDED) {
        __nv_bfloat16* out = yb + (size_t)t * a.ldy + c0;
        if (left >= W && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < W; j += 8) {
                uint32_t u[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(v[j + 2 * i], v[j + 2 * i + 1]);
                    u[i] = *reinterpret_cast<const uint32_t*>(&h);
                }
                *reinterpret_cast<uint4*>(out + j) = make_uint4(u[0], u[1], u[2], u[3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < W; j++) if (j < left) out[j] = __float2bfloat16(v[j]);
        }
    } else {
        float* out = y + (size_t)t * a.ldy + c0;
        if (left >= W && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < W; j += 4) *reinterpret_cast<float4*>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < W; j++) if (j < left) out[j] = v[j];
        }
    }
}

template <int EPI, bool ROUNDED, bool SHORT>
__global__ void __launch_bounds__(TC_THREADS, 1) dense_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                 const __grid_constant__ TcParams p) {
    extern __shared__ uint8_t tc_smem[];
    __shared__ uint64_t full[TC_MAX_STAGES], empty[TC_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_at;
    const DenseDev& a = p.a;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp: known to be uniform)
    uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)tc_smem + 1023) & ~(uintptr_t)1023);
    const int S = p.stages;
    // a stage: weights, then tokens (short steps: the MMA reads 128 token rows whatever NT is; what it finds there is dropped)
    const int ks = SHORT ? p.ks : 1;
    const uint32_t w_slice = (uint32_t)p.NW * TC_K * 2, x_slice = (uint32_t)p.NT * TC_K * 2, w_bytes = ks * w_slice, stage_bytes = w_bytes + ks * x_slice;
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < 2 * p.cols) tmem_cols <<= 1;
    if (warp == 5) {
        if (lane == 0) {
            for (int i = 0; i < S; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
            for (int i = 0; i < 2; i++) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 128); }
            fence_mbar_init();
        }
        __syncwarp();
        tc_alloc(&tmem_at, tmem_cols);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    griddep_launch();
    const uint32_t tmem = tmem_at;
    const int slices = (a.K + TC_K - 1) / TC_K, nk = (slices + ks - 1) / ks, first = blockIdx.x, step = gridDim.x;
    auto load_w = [&](uint8_t* st, int k, const TcTile& w, uint64_t* bar) {
        if (SHORT && ks > 1) tma_load_4d(st, &map_w, 0, w.n0, k * ks, w.z, bar);
        else tma_load_3d(st, &map_w, k * TC_K, w.n0, w.z, bar);
    };

    // The loops of the two issuing warps are run by all lanes, one of which issues: what the instructions take from uniform registers is
    // computed there (as loops of one lane, each instruction was preceded by moves).
    if (warp == 4) {
        // ================= copies
        const bool one = elect_one();
        int s = 0, ahead = 0;
        uint32_t use = 0;
        bool waited = false;
        if (!a.grouped && first < p.n_work) {                      // weights of the first stages: no need to wait for the previous kernel
            TcTile w;
            tc_tile(p, first, 0, w);
            for (; ahead < S && ahead < nk; ahead++)
                if (one) {
                    mbar_arrive_expect_tx(&full[ahead], stage_bytes);
                    load_w(ring + (size_t)ahead * stage_bytes, ahead, w, &full[ahead]);
                }
        }
        griddep_wait();
        const int n_tiles = a.grouped ? *a.g.n_tiles : 0;
        for (int i = first; i < p.n_work; i += step) {
            TcTile w;
            if (!tc_tile(p, i, n_tiles, w)) continue;
            for (int k = 0; k < nk; k++) {
                uint8_t* st = ring + (size_t)s * stage_bytes;
                const bool weights = waited || k >= ahead;         // else they are on their way
                if (weights && use > 0) mbar_wait_warp(&empty[s], (use - 1) & 1, p.err, 0x50001u, (unsigned)k);
                if (one && weights) {
                    mbar_arrive_expect_tx(&full[s], stage_bytes);
                    load_w(st, k, w, &full[s]);
                }
                if (!one) {
                } else if (SHORT && ks > 1) tma_load_4d(st + w_bytes, &map_x, 0, w.t0, k * ks, a.grouped ? 0 : w.z, &full[s]);
                else tma_load_3d(st + w_bytes, &map_x, k * TC_K, w.t0, a.grouped ? 0 : w.z, &full[s]);
                if (++s == S) { s = 0; use++; }
            }
            waited = true;
        }
    } else if (warp == 5) {
        // ================= matrix instructions
        const bool one = elect_one();
        griddep_wait();
        const int n_tiles = a.grouped ? *a.g.n_tiles : 0;
        const uint32_t idesc = tc_idesc_bf16(TC_M, SHORT ? p.NW : p.NT);
        int s = 0, tile = 0;
        uint32_t use = 0;
        for (int i = first; i < p.n_work; i += step) {
            TcTile w;
            if (!tc_tile(p, i, n_tiles, w)) continue;
            const int b = tile & 1;
            if (tile >= 2) mbar_wait_warp(&acc_empty[b], ((tile >> 1) - 1) & 1, p.err, 0x50002u, (unsigned)tile);
            tc_after_sync();
            for (int k = 0; k < nk; k++) {
                mbar_wait_warp(&full[s], use & 1, p.err, 0x50003u, (unsigned)k);
                tc_after_sync();
                const uint32_t at = smem_u32(ring + (size_t)s * stage_bytes);
                const int n_slices = min(ks, slices - k * ks);
                if (one) for (int q = 0; q < n_slices; q++) {
                    const uint64_t dw = tc_desc(at + q * w_slice), dx = tc_desc(at + w_bytes + q * x_slice);
#pragma unroll
                    for (int kk = 0; kk < TC_K / 16; kk++)
                        tc_mma(tmem + b * p.cols, (SHORT ? dx : dw) + 2 * kk, (SHORT ? dw : dx) + 2 * kk, idesc, (k | q | kk) ? 1u : 0u);
                }
                if (one) tc_commit(&empty[s]);
                if (++s == S) { s = 0; use++; }
            }
            if (one) tc_commit(&acc_full[b]);
            tile++;
        }
    } else if (warp < 4) {
        // ================= epilogue
        griddep_wait();
        const int n_tiles = a.grouped ? *a.g.n_tiles : 0;
        int tile = 0;
        for (int i = first; i < p.n_work; i += step) {
            TcTile w;
            if (!tc_tile(p, i, n_tiles, w)) continue;
            const int b = tile & 1;
            mbar_wait(&acc_full[b], (tile >> 1) & 1, p.err, 0x50004u, (unsigned)tile);
            tc_after_sync();
            const uint32_t acc = tmem + b * p.cols + ((uint32_t)(warp * 32) << 16);
            float* y = a.y;
            const float* aux = a.aux;
            __nv_bfloat16* yb = a.yb;
            if (!a.grouped) { y += w.z * a.y_bs; yb += w.z * a.y_bs; if (aux) aux += w.z * a.aux_bs; }
            if constexpr (SHORT) {
                const int t = w.t0 + threadIdx.x, n_end = min(w.n0 + p.NW, a.N);
                if (w.t0 + warp * 32 < w.t1) {
                    for (int c = 0; c < p.NW; c += 16) {
                        float v[16];
                        __syncwarp();
                        tc_ld16(acc + c, v);
                        if (w.n0 + c < n_end) tc_store_rows<EPI, ROUNDED>(a, y, yb, aux, (int)threadIdx.x < p.NT && t < w.t1, w.n0 + c, n_end, t, v);
                    }
                }
            } else {
                const int n = w.n0 + threadIdx.x, left = w.t1 - w.t0;
                const float bias = (EPI == EPI_BIAS || EPI == EPI_BIAS_RELU2 || EPI == EPI_BIAS_PART_RELU2) && a.bias && n < a.N ? a.bias[n] : 0.f;
                for (int c = 0; c < p.NT && c < left; c += 16) {
                    float v[16];
                    __syncwarp();
                    tc_ld16(acc + c, v);
                    tc_store<EPI, ROUNDED>(a, y, yb, aux, bias, n, w.t0 + c, min(16, left - c), v);
                }
            }
            tc_before_sync();
            mbar_arrive(&acc_empty[b]);
            tile++;
        }
    }
    tc_before_sync();
    __syncthreads();
    if (warp == 5) tc_dealloc(tmem, tmem_cols);
}

// ---------------------------------------------------------------- rounded inputs
// y[r][0..K) = bf16(x[rows ? rows[r] : r][0..K)), 8 entries a thread; TX float or bf16 (the latter only gathers). K % 8 == 0
template <typename TX>
__global__ void rows_to_bf16_kernel(const TX* __restrict__ x, int ldx, const int* __restrict__ rows, int n_src, int T, int K, __nv_bfloat16* __restrict__ y) {
    griddep_launch();
    griddep_wait();
    const int per = K / 8;
    const long n = (long)T * per;
    const bool wide = sizeof(TX) == 2 || (ldx % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int t = (int)(i / per), k = (int)(i % per) * 8;
        const int src = rows ? min(max(rows[t], 0), n_src - 1) : t;
        const TX* from = x + (size_t)src * ldx + k;
        uint4 o;
        if constexpr (sizeof(TX) == 2) o = *reinterpret_cast<const uint4*>(from);
        else {
            float v[8];
            if (wide) {
                const float4 p = *reinterpret_cast<const float4*>(from), q = *reinterpret_cast<const float4*>(from + 4);
                v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = from[j];
            }
            uint32_t u[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                u[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
            o = make_uint4(u[0], u[1], u[2], u[3]);
        }
        *reinterpret_cast<uint4*>(y + (size_t)t * K + k) = o;
    }
}

// ---------------------------------------------------------------- host side
typedef CUresult (*TcEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

template <int N>
static bool encode_map(CUtensorMap* m, const void* base, const cuuint64_t (&dims)[N], const cuuint64_t (&strides)[N - 1], const cuuint32_t (&box)[N]) {
    static const TcEncodeFn encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) fn = nullptr;
        cudaGetLastError();
        return (TcEncodeFn)fn;
    }();
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return encode && encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, N, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool bf16_rows_map(CUtensorMap* m, const void* base, long cols, long rows, long ld, long nb, long bs, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)nb};
    const cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)(nb > 1 ? bs * 2 : ld * 2)};
    const cuuint32_t box[3] = {TC_K, (cuuint32_t)box_rows, 1};
    return encode_map(m, base, dims, strides, box);
}
bool bf16_slices_map(CUtensorMap* m, const void* base, long cols, long rows, long ld, long nb, long bs, int box_rows, int slices) {
    const cuuint64_t dims[4] = {TC_K, (cuuint64_t)rows, (cuuint64_t)(cols / TC_K), (cuuint64_t)nb};
    const cuuint64_t strides[3] = {(cuuint64_t)ld * 2, TC_K * 2, (cuuint64_t)(nb > 1 ? bs * 2 : ld * 2)};
    const cuuint32_t box[4] = {TC_K, (cuuint32_t)box_rows, (cuuint32_t)slices, 1};
    return cols % TC_K == 0 && encode_map(m, base, dims, strides, box);
}
bool bf16_parts_map(CUtensorMap* m, const void* base, long cols, long rows, long ld, long nb, long bs, int parts, int box_rows) {
    const cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)parts, (cuuint64_t)nb};
    const cuuint64_t strides[3] = {(cuuint64_t)ld * 2, (cuuint64_t)(rows * ld) * 2, (cuuint64_t)(nb > 1 ? bs * 2 : ld * 2)};
    const cuuint32_t box[4] = {TC_K, (cuuint32_t)box_rows, (cuuint32_t)parts, 1};
    return encode_map(m, base, dims, strides, box);
}
bool bf16_heads_map(CUtensorMap* m, const void* base, long cols, long heads, long rows, int box_heads, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)heads, (cuuint64_t)rows};
    const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)(cols * heads) * 2};
    const cuuint32_t box[3] = {TC_K, (cuuint32_t)box_heads, (cuuint32_t)box_rows};
    return encode_map(m, base, dims, strides, box);
}

typedef void (*TcKernel)(const CUtensorMap, const CUtensorMap, const TcParams);
template <int EPI, bool ROUNDED = false>
static TcKernel tc_kernel_of(bool short_step) {
    if (short_step) return allow_smem<dense_tc_kernel<EPI, ROUNDED, true>>(TC_SMEM) ? dense_tc_kernel<EPI, ROUNDED, true> : nullptr;
    return allow_smem<dense_tc_kernel<EPI, ROUNDED, false>>(TC_SMEM) ? dense_tc_kernel<EPI, ROUNDED, false> : nullptr;
}
static TcKernel tc_kernel(int epi, bool rounded, bool short_step) {
    if (rounded) {
        switch (epi) {
            case EPI_NONE: return tc_kernel_of<EPI_NONE, true>(short_step);
            case EPI_MUL_SIGMOID: return tc_kernel_of<EPI_MUL_SIGMOID, true>(short_step);
            case EPI_BIAS_RELU2: return tc_kernel_of<EPI_BIAS_RELU2, true>(short_step);
            case EPI_GLU_GELU: return tc_kernel_of<EPI_GLU_GELU, true>(short_step);
            case EPI_PIECEWISE: return tc_kernel_of<EPI_PIECEWISE, true>(short_step);
            case EPI_GLU_SILU: return tc_kernel_of<EPI_GLU_SILU, true>(short_step);
            case EPI_GLU_CLAMP: return tc_kernel_of<EPI_GLU_CLAMP, true>(short_step);
            default: return nullptr;
        }
    }
    switch (epi) {
        case EPI_NONE: return tc_kernel_of<EPI_NONE>(short_step);
        case EPI_BIAS: return tc_kernel_of<EPI_BIAS>(short_step);
        case EPI_BIAS_RELU2: return tc_kernel_of<EPI_BIAS_RELU2>(short_step);
        case EPI_GLU_SILU: return tc_kernel_of<EPI_GLU_SILU>(short_step);
        case EPI_MUL_SIGMOID: return tc_kernel_of<EPI_MUL_SIGMOID>(short_step);
        case EPI_GLU_CLAMP: return tc_kernel_of<EPI_GLU_CLAMP>(short_step);
        case EPI_PIECEWISE: return tc_kernel_of<EPI_PIECEWISE>(short_step);
        case EPI_GLU_GELU: return tc_kernel_of<EPI_GLU_GELU>(short_step);
        case EPI_BIAS_PART_RELU2: return tc_kernel_of<EPI_BIAS_PART_RELU2>(short_step);
    }
    return nullptr;
}

cudaError_t dense_tc_launch(const DenseArgs& a, const DenseDev& d, cudaStream_t s) {
    const int SMS = 148;
    const bool grouped = d.grouped == 2;
    if (d.grouped == 1 || !a.xb) return cudaErrorInvalidValue;
    // ---- the input, rounded (and gathered into the order of the sorted pairs)
    const int span = a.batch > 1 ? a.x_span : a.K;
    const int* gather = grouped ? a.groups->x_rows : nullptr;
    const int src_rows = grouped ? a.groups->x_total_rows : a.T, rows = gather ? a.T : src_rows;
    const __nv_bfloat16* xb = a.x_rounded;
    if (!xb || gather) {
        const long n = (long)rows * (span / 8);
        const dim3 grid((unsigned)std::min<long>((n + 255) / 256, SMS * 8));
        cudaError_t e;
        if (xb) e = launch_chain(rows_to_bf16_kernel<__nv_bfloat16>, grid, dim3(256), 0, s, xb, span, gather, src_rows, rows, span, a.xb);
        else e = launch_chain(rows_to_bf16_kernel<float>, grid, dim3(256), 0, s, a.x, a.ldx, gather, src_rows, rows, span, a.xb);
        if (e != cudaSuccess) return e;
        xb = a.xb;
    }
    // ---- tiles
    TcParams p = {};
    p.a = d;
    p.err = kernel_error_word();
    // grouped: 64-row tiles are short (a 128-row tile of a long prompt fills the other orientation's columns as well)
    const bool short_step = grouped ? a.groups->tile_max <= 64 : a.T <= 256;
    if (short_step) {
        p.NT = grouped ? a.groups->tile_max : std::min(TC_M, (a.T + 15) / 16 * 16);
        p.nT = grouped ? a.groups->max_tiles : (a.T + p.NT - 1) / p.NT;
        // weight rows a tile: one wave over the SMs (of as many expert tiles as have rows, which the device alone knows: at most one per
        // expert when the pairs are few)
        const long parts = grouped ? std::min(a.groups->max_tiles, a.groups->n_groups) : (long)a.batch * p.nT, rows_per = (a.N * parts + SMS - 1) / SMS;
        p.NW = (int)std::min<long>(256, std::max<long>(16, (rows_per + 15) / 16 * 16));
    } else {
        p.NW = TC_M;
        if (grouped) {
            p.NT = a.groups->tile_max;
            p.nT = a.groups->max_tiles;
        } else {
            // waves x (columns + the share of a tile's time that its 128 weight rows cost whatever the columns)
            long best = -1;
            const long nN = (a.N + TC_M - 1) / TC_M;
            for (int nt = 256; nt >= 64; nt -= 32) {
                const long tiles = nN * a.batch * ((a.T + nt - 1) / nt), cost = (tiles + SMS - 1) / SMS * (nt + 96);
                if (best < 0 || cost < best) { best = cost; p.NT = nt; }
            }
            p.nT = (a.T + p.NT - 1) / p.NT;
        }
    }
    p.nN = (a.N + p.NW - 1) / p.NW;
    p.n_work = p.nN * p.nT * (grouped ? 1 : a.batch);
    p.cols = ((short_step ? p.NW : p.NT) + 31) / 32 * 32;
    // short steps: several K slices per copy and barrier while a stage stays within 32 KB (with one, a 16-row tile moved 2 KB per copy and the
    // copying thread set the pace)
    p.ks = 1;
    if (short_step && a.K % TC_K == 0) while (p.ks < 4 && (p.NW + p.NT) * TC_K * 2 * p.ks * 2 <= 32 * 1024 && a.K / TC_K >= 4 * p.ks) p.ks *= 2;
    const int stage_bytes = (p.NW + p.NT) * TC_K * 2 * p.ks;
    p.stages = std::min(TC_MAX_STAGES, TC_RING / stage_bytes);
    TcKernel kernel = tc_kernel(a.epi, a.y_rounded != nullptr, short_step);
    if (!kernel) return cudaErrorInvalidValue;
    CUtensorMap mw, mx;
    const long w_entries = grouped ? a.groups->n_groups : a.batch, w_bs = grouped ? a.groups->w_stride : a.w_bs;
    const long x_entries = grouped ? 1 : a.batch;
    if (p.ks > 1 ? !bf16_slices_map(&mw, a.w, a.K, a.N, a.K, w_entries, w_bs, p.NW, p.ks) : !bf16_rows_map(&mw, a.w, a.K, a.N, a.K, w_entries, w_bs, p.NW)) return cudaErrorInvalidValue;
    if (p.ks > 1 ? !bf16_slices_map(&mx, xb, a.K, rows, span, x_entries, a.x_bs, p.NT, p.ks) : !bf16_rows_map(&mx, xb, a.K, rows, span, x_entries, a.x_bs, p.NT)) return cudaErrorInvalidValue;
    return launch_chain(kernel, dim3(std::min(p.n_work, SMS)), dim3(TC_THREADS), (size_t)p.stages * stage_bytes + TC_M * TC_K * 2 + 1024, s, mw, mx, p);
}

}  // namespace b2
