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
    // Values first, stores after, no branches among the values: a test, a load or a store between two of them keeps them from overlapping, and a scheduler
    // has one of these warps. (2048 tokens: gated GELU, 8192 units of 2048, 137 -> 95 us; times a head's gate, 2048 outputs of 512, 127 -> 24.)
    if constexpr (GLU) {
        // rows 2i (gate) and 2i + 1 (up) sit in neighbouring lanes: of two columns the even lane finishes the first, the odd one the second
        float v[8];
        float scale[8];
#pragma unroll
        for (int j = 0; j < 8; j++) scale[j] = a.g.row_scale ? a.g.row_scale[t + min(2 * j + (lane & 1), count - 1)] : 1.f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? acc[2 * j] : acc[2 * j + 1], 1);
            float gate = (lane & 1) ? other : acc[2 * j], up = (lane & 1) ? acc[2 * j + 1] : other;
            gate *= scale[j]; up *= scale[j];
            if (EPI == EPI_GLU_CLAMP) {
                const float g = fminf(gate, a.p0), u = fminf(fmaxf(up, -a.p0), a.p0);
                v[j] = over_one_plus_exp(g, -a.p1 * g) * (u + 1.f);
            } else v[j] = (EPI == EPI_GLU_SILU ? silu_act(gate) : gelu_tanh_act(gate)) * up;
            v[j] *= a.scale;
        }
        const size_t at = (size_t)(t + (lane & 1)) * a.ldy + (n >> 1);
        const int left = (n | 1) < a.N ? count - (lane & 1) : 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (2 * j >= left) break;
            if constexpr (ROUNDED) yb[at + (size_t)(2 * j) * a.ldy] = __float2bfloat16(v[j]);
            else y[at + (size_t)(2 * j) * a.ldy] = v[j];
        }
    } else {
        if (n >= a.N) return;
        float gate[16], v[16];
        if (EPI == EPI_MUL_SIGMOID) {
#pragma unroll
            for (int j = 0; j < 16; j++) gate[j] = aux[(size_t)(t + min(j, count - 1)) * a.ldaux + n * a.aux_ns];
        }
#pragma unroll
        for (int j = 0; j < 16; j++) {
            v[j] = acc[j] + bias;
            if (EPI == EPI_BIAS_RELU2 || (EPI == EPI_BIAS_PART_RELU2 && n >= a.n_act && n < a.n_act_end)) { v[j] = fmaxf(v[j], 0.f); v[j] = v[j] * v[j]; }
            if (EPI == EPI_MUL_SIGMOID) v[j] *= sigmoid_act(gate[j]);
            if (EPI == EPI_PIECEWISE) v[j] = v[j] > 0.f ? fmaf(a.p0 * v[j], v[j], 0.5f * v[j]) : fmaf(a.p1, expm1f(v[j]) - v[j], 0.5f * v[j]);
            v[j] *= a.scale;
        }
        const size_t at = (size_t)t * a.ldy + n;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            if (j >= count) break;
            if constexpr (ROUNDED) yb[at + (size_t)j * a.ldy] = __float2bfloat16(v[j]);
            else y[at + (size_t)j * a.ldy] = v[j];
        }
    }
}

}  // namespace b2
