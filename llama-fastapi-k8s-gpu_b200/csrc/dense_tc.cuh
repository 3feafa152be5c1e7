// What the kernels that multiply on the 5th-generation tensor cores share (dense_tc.cu, dense_split.cu): tiles, the walk over them, the
// stores of tiles whose lanes are weight rows.
#pragma once
#include "dense_dev.cuh"
#include "ptx.cuh"

namespace b2 {

constexpr int TC_M = 128, TC_K = 64;             // rows of the A operand, K entries of a stage (128 bytes: one swizzle row)
constexpr int TC_RING = 208 * 1024;              // shared memory for the stages

struct TcParams {
    DenseDev a;
    int NT, NW;              // tokens and weight rows of a tile (multiples of 16; the A operand's side at most 128)
    int nN, nT;              // weight-row tiles; token tiles (grouped: tiles of the sorted pairs)
    int n_work;              // tiles in all
    int stages, cols;        // ring stages; tensor-memory columns of one accumulator
    int ks;                  // 64-wide K slices of a stage (1; short steps also 2 and 4: a copy, a wait and a commit cost the same for all of
                             // them, and few-row tiles are small. 32 sequences, 12 steps of two layers: 6.85 -> 6.1 ms)
    unsigned int* err;
};

struct TcTile { int n0, t0, t1, z; };

// tiles that share weights are neighbours: token tiles (or the sorted tiles of the experts) run fastest
__device__ __forceinline__ bool tc_tile(const TcParams& p, int i, int n_tiles, TcTile& w) {
    const int t = i % p.nT, rest = i / p.nT;
    w.n0 = (rest % p.nN) * p.NW;
    if (p.a.grouped) {
        if (t >= n_tiles) return false;
        w.t0 = p.a.g.tile_row0[t];
        w.t1 = w.t0 + p.a.g.tile_rows[t];
        w.z = p.a.g.tile_group[t];
        return true;
    }
    w.z = rest / p.nN;
    w.t0 = t * p.NT;
    w.t1 = p.a.T;
    return true;
}

// long steps: 16 (or fewer, `count`) token columns t.. of weight row n; lanes of a warp hold neighbouring rows
template <int EPI, bool ROUNDED>
__device__ __forceinline__ void tc_store(const DenseDev& a, float* y, __nv_bfloat16* yb, const float* aux, float bias, int n, int t, int count,
                                         const float (&acc)[16]) {
    const int lane = threadIdx.x & 31;
    constexpr bool GLU = EPI == EPI_GLU_SILU || EPI == EPI_GLU_GELU || EPI == EPI_GLU_CLAMP;
    if constexpr (GLU) {
        // rows 2i (gate) and 2i + 1 (up) sit in neighbouring lanes: of two columns the even lane finishes the first, the odd one the second
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? acc[j] : acc[j + 1], 1);
            float gate = (lane & 1) ? other : acc[j], up = (lane & 1) ? acc[j + 1] : other;
            const int c = j + (lane & 1);
            if (c >= count || (n | 1) >= a.N) continue;
            if (a.g.row_scale) { const float s = a.g.row_scale[t + c]; gate *= s; up *= s; }
            float v;
            if (EPI == EPI_GLU_CLAMP) {
                const float g = fminf(gate, a.p0), u = fminf(fmaxf(up, -a.p0), a.p0);
                v = g / (1.f + expf(-a.p1 * g)) * (u + 1.f);
            } else v = (EPI == EPI_GLU_SILU ? silu_act(gate) : gelu_tanh_act(gate)) * up;
            const size_t at = (size_t)(t + c) * a.ldy + (n >> 1);
            if constexpr (ROUNDED) yb[at] = __float2bfloat16(v * a.scale);
            else y[at] = v * a.scale;
        }
    } else {
        if (n >= a.N) return;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            if (j >= count) break;
            float v = acc[j] + bias;
            if (EPI == EPI_BIAS_RELU2 || (EPI == EPI_BIAS_PART_RELU2 && n >= a.n_act && n < a.n_act_end)) { v = fmaxf(v, 0.f); v = v * v; }
            if (EPI == EPI_MUL_SIGMOID) v *= 1.f / (1.f + expf(-aux[(size_t)(t + j) * a.ldaux + n * a.aux_ns]));
            if (EPI == EPI_PIECEWISE) v = v > 0.f ? fmaf(a.p0 * v, v, 0.5f * v) : fmaf(a.p1, expm1f(v) - v, 0.5f * v);
            const size_t at = (size_t)(t + j) * a.ldy + n;
            if constexpr (ROUNDED) yb[at] = __float2bfloat16(v * a.scale);
            else y[at] = v * a.scale;
        }
    }
}

}  // namespace b2
