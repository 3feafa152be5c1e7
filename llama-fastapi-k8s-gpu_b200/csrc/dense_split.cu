// 32-bit products of more than 8 tokens with bf16 weights on the 5th-generation tensor cores:
//     Y[t][n] = epi(sum_k X[t][k] * W[n][k])      X, Y f32, W bf16 as stored.
//
// An f32 value of 2^-110 and more is the sum of three bf16 values, exactly: its 24 significant bits cut into runs of 8 (truncated, not rounded, so
// that nothing overflows; the split of Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for higher-precision
// computations", 2019). Of smaller values what lies below bf16's last subnormal bit is cut off, less than 2^-133: a row whose largest entry is
// 2^-120 is off by 7e-5, beside larger entries it does not show. A product of two bf16 values is exact in f32, so X . W is three bf16 products whose terms are the terms of the 32-bit
// product; only the sums round. Tensor memory sums without rounding to nearest, and over a whole K that would show; so a sum stays there for
// 64 entries of K only (three parts, the smallest first) and is then added to a 32-bit register in the order of k, as the multiply-add kernel
// adds single terms. Errors against 64 bits are below that kernel's (below).
// (An infinite input stays one. An infinite WEIGHT would meet the zeros behind an input's leading part as NaN, where multiply-adds keep the
// infinity: models with one never come here, see bf16_any_infinite.)
//
// Tiles of 128 weight rows (the lanes of tensor memory) and NT tokens, one after another per CTA. Ten warps: 0-7 add up and store (four
// lanes' quarters, two halves of the token columns), 8 copies, 9 matrix instructions. Four accumulators of NT columns: the products of up to
// three K slices run ahead of the additions.
// Bound by the chain of a slice (its copy, twelve products, the read-out of its sums), a CTA an SM and K / 64 slices in a row: the tensor pipe is
// busy 9 to 29 % of the time, issue slots 17 to 22 %, L2 9 to 13 % (ncu). 459 tokens of two layers of 1024 (B200): ten products 1320 us as multiply-adds, 20 to 37 each here, the whole step 1820 -> 550; against 64 bits the
// logits are off by 4.8e-7 of their norm, 1.5e-6 before.
#include "dense_tc.cuh"
#include "quant_blocks.cuh"
#include "tc05.cuh"
#include "tensor_map.h"

#include <algorithm>

namespace b2 {

constexpr int SP_PARTS = 3, SP_ADDERS = 8, SP_THREADS = (SP_ADDERS + 2) * 32, SP_BUFS = 4, SP_MAX_NT = 128, SP_MAX_STAGES = 8;

template <int EPI>
__global__ void __launch_bounds__(SP_THREADS, 1) dense_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                    const __grid_constant__ TcParams p) {
    extern __shared__ uint8_t sp_smem[];
    __shared__ uint64_t full[SP_MAX_STAGES], empty[SP_MAX_STAGES], acc_full[SP_BUFS], acc_empty[SP_BUFS];
    __shared__ uint32_t tmem_at;
    const DenseDev& a = p.a;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)sp_smem + 1023) & ~(uintptr_t)1023);
    const int S = p.stages;
    const uint32_t w_bytes = TC_M * TC_K * 2, x_part = (uint32_t)p.NT * TC_K * 2, stage_bytes = w_bytes + SP_PARTS * x_part;
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < SP_BUFS * p.cols) tmem_cols <<= 1;
    if (warp == SP_ADDERS + 1) {
        if (lane == 0) {
            for (int i = 0; i < S; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
            for (int i = 0; i < SP_BUFS; i++) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], SP_ADDERS * 32); }
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
    const int nk = (a.K + TC_K - 1) / TC_K, first = blockIdx.x, step = gridDim.x;
    if (warp == SP_ADDERS) {
        // ================= copies: the weights of the first stages do not wait for the previous kernel
        const bool one = elect_one();
        int s = 0, ahead = 0;
        uint32_t use = 0;
        if (!a.grouped && first < p.n_work) {
            TcTile w;
            tc_tile(p, first, 0, w);
            for (; ahead < S && ahead < nk; ahead++)
                if (one) {
                    mbar_arrive_expect_tx(&full[ahead], stage_bytes);
                    tma_load_3d(ring + (size_t)ahead * stage_bytes, &map_w, ahead * TC_K, w.n0, w.z, &full[ahead]);
                }
        }
        griddep_wait();
        const int n_tiles = a.grouped ? *a.g.n_tiles : 0;
        for (int i = first; i < p.n_work; i += step) {
            TcTile w;
            if (!tc_tile(p, i, n_tiles, w)) continue;
            for (int k = 0; k < nk; k++) {
                uint8_t* st = ring + (size_t)s * stage_bytes;
                if (ahead > 0) ahead--;                            // its weights are on their way
                else {
                    if (use > 0) mbar_wait_warp(&empty[s], (use - 1) & 1, p.err, 0x51001u, (unsigned)k);
                    if (one) {
                        mbar_arrive_expect_tx(&full[s], stage_bytes);
                        tma_load_3d(st, &map_w, k * TC_K, w.n0, w.z, &full[s]);
                    }
                }
                if (one) tma_load_4d(st + w_bytes, &map_x, k * TC_K, w.t0, 0, a.grouped ? 0 : w.z, &full[s]);
                if (++s == S) { s = 0; use++; }
            }
        }
    } else if (warp == SP_ADDERS + 1) {
        // ================= matrix instructions
        const bool one = elect_one();
        griddep_wait();
        const int n_tiles = a.grouped ? *a.g.n_tiles : 0;
        const uint32_t idesc = tc_idesc_bf16(TC_M, p.NT);
        int s = 0, b = 0;
        uint32_t use = 0, turn = 0;
        for (int i = first; i < p.n_work; i += step) {
            TcTile w;
            if (!tc_tile(p, i, n_tiles, w)) continue;
            for (int k = 0; k < nk; k++) {
                if (turn > 0) mbar_wait_warp(&acc_empty[b], (turn - 1) & 1, p.err, 0x51002u, (unsigned)k);
                mbar_wait_warp(&full[s], use & 1, p.err, 0x51003u, (unsigned)k);
                tc_after_sync();
                const uint32_t at = smem_u32(ring + (size_t)s * stage_bytes);
                if (one) {
                    const uint64_t dw = tc_desc(at);
                    for (int part = SP_PARTS - 1; part >= 0; part--) {
                        const uint64_t dx = tc_desc(at + w_bytes + part * x_part);
#pragma unroll
                        for (int kk = 0; kk < TC_K / 16; kk++) tc_mma(tmem + b * p.cols, dw + 2 * kk, dx + 2 * kk, idesc, (part < SP_PARTS - 1 || kk) ? 1u : 0u);
                    }
                    tc_commit(&empty[s]);
                    tc_commit(&acc_full[b]);
                }
                __syncwarp();
                if (++s == S) { s = 0; use++; }
                if (++b == SP_BUFS) { b = 0; turn++; }
            }
        }
    } else {
        // ================= additions, epilogue
        griddep_wait();
        const int n_tiles = a.grouped ? *a.g.n_tiles : 0, half = p.NT / 2, c0 = warp < 4 ? 0 : half;
        const uint32_t quarter = tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0;
        int b = 0;
        uint32_t turn = 0;
        for (int i = first; i < p.n_work; i += step) {
            TcTile w;
            if (!tc_tile(p, i, n_tiles, w)) continue;
            float acc[SP_MAX_NT / 32][16];
#pragma unroll
            for (int g = 0; g < SP_MAX_NT / 32; g++)
#pragma unroll
                for (int j = 0; j < 16; j++) acc[g][j] = 0.f;
            for (int k = 0; k < nk; k++) {
                mbar_wait_warp(&acc_full[b], turn & 1, p.err, 0x51004u, (unsigned)k);
                tc_after_sync();
#pragma unroll
                for (int g = 0; g < SP_MAX_NT / 32; g++) {
                    if (16 * g >= half) break;
                    float v[16];
                    tc_ld16(quarter + b * p.cols + 16 * g, v);
#pragma unroll
                    for (int j = 0; j < 16; j++) acc[g][j] += v[j];
                }
                tc_before_sync();
                mbar_arrive(&acc_empty[b]);
                if (++b == SP_BUFS) { b = 0; turn++; }
            }
            float* y = a.y;
            const float* aux = a.aux;
            if (!a.grouped) { y += w.z * a.y_bs; if (aux) aux += w.z * a.aux_bs; }
            const int n = w.n0 + (warp & 3) * 32 + lane, left = w.t1 - w.t0 - c0;
            const float bias = (EPI == EPI_BIAS || EPI == EPI_BIAS_RELU2 || EPI == EPI_BIAS_PART_RELU2) && a.bias && n < a.N ? a.bias[n] : 0.f;
#pragma unroll
            for (int g = 0; g < SP_MAX_NT / 32; g++) {
                if (16 * g >= half || 16 * g >= left) break;
                __syncwarp();
                tc_store<EPI, false>(a, y, nullptr, aux, bias, n, w.t0 + c0 + 16 * g, min(16, left - 16 * g), acc[g]);
            }
        }
    }
    tc_before_sync();
    __syncthreads();
    if (warp == SP_ADDERS + 1) tc_dealloc(tmem, tmem_cols);
}

// ---------------------------------------------------------------- inputs in three parts
// parts[j][r][0..K), j = 0 .. 2: leading, middle and last 8 significant bits (as far as bf16 reaches) of x[rows ? rows[r] : r][0..K), 8 entries a thread. K % 8 == 0.
// Infinities and NaN stay what they are in the leading part, with zeros behind them.
__global__ void rows_to_parts_kernel(const float* __restrict__ x, int ldx, const int* __restrict__ rows, int n_src, int T, int K, __nv_bfloat16* __restrict__ parts) {
    griddep_launch();
    griddep_wait();
    const int per = K / 8;
    const long n = (long)T * per, plane = (long)T * K;
    const bool wide = ldx % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int t = (int)(i / per), k = (int)(i % per) * 8;
        const int src = rows ? min(max(rows[t], 0), n_src - 1) : t;
        const float* from = x + (size_t)src * ldx + k;
        float v[8];
        if (wide) {
            const float4 f = *reinterpret_cast<const float4*>(from), g = *reinterpret_cast<const float4*>(from + 4);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; v[4] = g.x; v[5] = g.y; v[6] = g.z; v[7] = g.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = from[j];
        }
        uint32_t u[SP_PARTS][4];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t bits = __float_as_uint(v[j]);
            const bool finite = (bits & 0x7f800000u) != 0x7f800000u;
            uint32_t h[SP_PARTS] = {bits & 0xffff0000u, 0u, 0u};
            if (finite) {
                const float r1 = v[j] - __uint_as_float(h[0]);
                h[1] = __float_as_uint(r1) & 0xffff0000u;
                h[2] = __float_as_uint(r1 - __uint_as_float(h[1])) & 0xffff0000u;
            } else if (bits & 0x007fffffu) h[0] |= 0x00400000u;       // a NaN whose cut payload is zero would read as an infinity
#pragma unroll
            for (int q = 0; q < SP_PARTS; q++) u[q][j >> 1] = (j & 1) ? (u[q][j >> 1] | h[q]) : (h[q] >> 16);
        }
#pragma unroll
        for (int q = 0; q < SP_PARTS; q++) *reinterpret_cast<uint4*>(parts + q * plane + (size_t)t * K + k) = make_uint4(u[q][0], u[q][1], u[q][2], u[q][3]);
    }
}

__global__ void any_infinite_kernel(const uint16_t* __restrict__ w, size_t n, int* found) {
    bool any = false;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) any |= (w[i] & 0x7fff) == 0x7f80;
    if (any) *found = 1;
}

// ---------------------------------------------------------------- host side
cudaError_t bf16_any_infinite(const void* w, size_t n, int* found, cudaStream_t s) {
    any_infinite_kernel<<<148 * 8, 256, 0, s>>>(static_cast<const uint16_t*>(w), n, found);
    return cudaGetLastError();
}

typedef void (*SplitKernel)(const CUtensorMap, const CUtensorMap, const TcParams);
template <int EPI>
static SplitKernel split_kernel_of() {
    return allow_smem<dense_split_kernel<EPI>>(TC_RING + 1024) ? dense_split_kernel<EPI> : nullptr;
}
static SplitKernel split_kernel(int epi) {
    switch (epi) {
        case EPI_NONE: return split_kernel_of<EPI_NONE>();
        case EPI_BIAS: return split_kernel_of<EPI_BIAS>();
        case EPI_BIAS_RELU2: return split_kernel_of<EPI_BIAS_RELU2>();
        case EPI_GLU_SILU: return split_kernel_of<EPI_GLU_SILU>();
        case EPI_MUL_SIGMOID: return split_kernel_of<EPI_MUL_SIGMOID>();
        case EPI_GLU_CLAMP: return split_kernel_of<EPI_GLU_CLAMP>();
        case EPI_PIECEWISE: return split_kernel_of<EPI_PIECEWISE>();
        case EPI_GLU_GELU: return split_kernel_of<EPI_GLU_GELU>();
        case EPI_BIAS_PART_RELU2: return split_kernel_of<EPI_BIAS_PART_RELU2>();
    }
    return nullptr;
}

// operands are tensor maps: rows of whole 16-byte pieces on 16-byte boundaries
bool dense_takes_split(const DenseArgs& a) {
    const int span = a.batch > 1 ? a.x_span : a.K;
    return a.x_parts && a.exact && a.w_type == T_BF16 && a.K % 8 == 0 && (reinterpret_cast<uintptr_t>(a.w) & 15) == 0 && span % 8 == 0 &&
           (a.batch == 1 || (a.x_span > 0 && a.x_bs % 8 == 0 && a.w_bs % 8 == 0)) && (!a.groups || (a.groups->tile_group && a.groups->tile_max == 64)) &&
           !a.x_rounded && !a.y_rounded;
}

cudaError_t dense_split_launch(const DenseArgs& a, const DenseDev& d, cudaStream_t s) {
    const int SMS = 148;
    const bool grouped = d.grouped == 2;
    if (d.grouped == 1 || !dense_takes_split(a)) return cudaErrorInvalidValue;
    const int span = a.batch > 1 ? a.x_span : a.K;
    const int* gather = grouped ? a.groups->x_rows : nullptr;
    const int src_rows = grouped ? a.groups->x_total_rows : a.T, rows = gather ? a.T : src_rows;
    const long n = (long)rows * (span / 8);
    cudaError_t e = launch_chain(rows_to_parts_kernel, dim3((unsigned)std::min<long>((n + 255) / 256, SMS * 8)), dim3(256), 0, s, a.x, a.ldx, gather, src_rows,
                                 rows, span, a.x_parts);
    if (e != cudaSuccess) return e;
    TcParams p = {};
    p.a = d;
    p.err = kernel_error_word();
    p.NW = TC_M;
    p.nN = (a.N + TC_M - 1) / TC_M;
    if (grouped) {
        p.NT = a.groups->tile_max;
        p.nT = a.groups->max_tiles;
    } else {
        // waves x (token columns + what a slice costs whatever the columns: the copy of its weights and their reads by every product)
        long best = -1;
        for (int nt = SP_MAX_NT; nt >= 32; nt -= 32) {
            const long tiles = (long)p.nN * a.batch * ((a.T + nt - 1) / nt), cost = (tiles + SMS - 1) / SMS * (nt + 64);
            if (best < 0 || cost < best) { best = cost; p.NT = nt; }
        }
        p.nT = (a.T + p.NT - 1) / p.NT;
    }
    p.n_work = p.nN * p.nT * (grouped ? 1 : a.batch);
    p.cols = p.NT;
    const int stage_bytes = (TC_M + SP_PARTS * p.NT) * TC_K * 2;
    p.stages = std::min(SP_MAX_STAGES, TC_RING / stage_bytes);
    SplitKernel kernel = split_kernel(a.epi);
    CUtensorMap mw, mx;
    if (!kernel || !bf16_rows_map(&mw, a.w, a.K, a.N, a.K, grouped ? a.groups->n_groups : a.batch, grouped ? a.groups->w_stride : a.w_bs, TC_M) ||
        !bf16_parts_map(&mx, a.x_parts, a.K, rows, span, grouped ? 1 : a.batch, a.x_bs, SP_PARTS, p.NT)) return cudaErrorInvalidValue;
    return launch_chain(kernel, dim3(std::min(p.n_work, SMS)), dim3(SP_THREADS), (size_t)p.stages * stage_bytes + 1024, s, mw, mx, p);
}

}  // namespace b2
