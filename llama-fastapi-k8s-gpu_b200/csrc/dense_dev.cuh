// What the dense-product kernels share (dense.cu, dense_tc.cu): the description a kernel gets by value and the epilogues.
#pragma once
#include "kernels.h"
#include "layered.h"
#include "ptx.cuh"

namespace b2 {

// what a kernel needs beyond its operands: epilogue, batch strides, grouping (DenseArgs, by value)
struct DenseDev {
    const float* x; int ldx;
    const void* w;
    const float* bias;
    float* y; int ldy;
    int T, N, K, epi;
    int n_act, n_act_end;          // EPI_BIAS_PART_RELU2
    __nv_bfloat16* yb;             // tcgen05 kernel: rounded output instead of y, or null
    float scale, p0, p1;
    const float* aux; int ldaux, aux_ns;      // aux column of output column n: n * aux_ns
    long x_bs, w_bs, y_bs, aux_bs;
    int grouped;                   // 0 plain, 1 one pair per blockIdx.y, 2 tiles
    DenseGroups g;
};

// The rows [t0, t1) this CTA computes and the operands they use. false: nothing to do.
template <typename TW>
__device__ __forceinline__ bool dense_tile(const DenseDev& a, int rows_per_cta, const float*& x, const TW*& w, float*& y, const float*& aux,
                                           int& t0, int& t1, unsigned by, unsigned bz) {
    x = a.x; w = reinterpret_cast<const TW*>(a.w); y = a.y; aux = a.aux;
    if (a.grouped == 0) {
        const long b = bz;
        x += b * a.x_bs; w += b * a.w_bs; y += b * a.y_bs;
        if (aux) aux += b * a.aux_bs;
        t0 = by * rows_per_cta; t1 = a.T;
        return t0 < t1;
    }
    if (a.grouped == 1) {
        const int p = by, g = a.g.group[p];
        if (g < 0 || g >= a.g.n_groups) return false;
        w += (long)g * a.g.w_stride;
        t0 = p; t1 = p + 1;
        return true;
    }
    const int tile = by;
    if (tile >= *a.g.n_tiles) return false;
    w += (long)a.g.tile_group[tile] * a.g.w_stride;
    t0 = a.g.tile_row0[tile]; t1 = t0 + a.g.tile_rows[tile];
    return true;
}
__device__ __forceinline__ int x_row(const DenseDev& a, int t) { return (a.grouped && a.g.x_rows) ? a.g.x_rows[t] : t; }

// gates of the epilogues, without branches (see tc_store)
__device__ __forceinline__ float silu_act(float z) { return over_one_plus_exp(z, -z); }
__device__ __forceinline__ float sigmoid_act(float z) { return over_one_plus_exp(1.f, -z); }
// z (1 + tanh u) / 2 = z / (1 + exp(-2u)), which does not cancel where tanh is near -1
__device__ __forceinline__ float gelu_tanh_act(float z) { return over_one_plus_exp(z, -1.5957691216057308f * fmaf(0.044715f * z * z, z, z)); }
__device__ __forceinline__ float epi_value(const DenseDev& a, const float* aux, int t, int n, float v) {
    const int epi = a.epi;
    if (epi == EPI_BIAS || epi == EPI_BIAS_RELU2 || epi == EPI_BIAS_PART_RELU2) { if (a.bias) v += a.bias[n]; }
    if (epi == EPI_BIAS_RELU2 || (epi == EPI_BIAS_PART_RELU2 && n >= a.n_act && n < a.n_act_end)) { v = fmaxf(v, 0.f); v = v * v; }
    if (epi == EPI_MUL_SIGMOID) v *= sigmoid_act(aux[(size_t)t * a.ldaux + n * a.aux_ns]);
    if (epi == EPI_PIECEWISE) v = v > 0.f ? fmaf(a.p0 * v, v, 0.5f * v) : fmaf(a.p1, expm1f(v) - v, 0.5f * v);
    return v * a.scale;
}
// one output column
__device__ __forceinline__ void epi_store(const DenseDev& a, float* y, const float* aux, int t, int n, float v) {
    y[(size_t)t * a.ldy + n] = epi_value(a, aux, t, n, v);
}
// two neighbouring columns n (even) and n + 1; rs: scales of the product rows (GLU epilogues) or null
__device__ __forceinline__ void epi_store2(const DenseDev& a, float* y, const float* aux, const float* rs, int t, int n, float v0, float v1) {
    const int epi = a.epi;
    if (epi == EPI_GLU_SILU || epi == EPI_GLU_GELU || epi == EPI_GLU_CLAMP) {
        if (n + 1 >= a.N) return;
        if (rs) { v0 *= rs[t]; v1 *= rs[t]; }
        float v;
        if (epi == EPI_GLU_CLAMP) {
            const float g = fminf(v0, a.p0), u = fminf(fmaxf(v1, -a.p0), a.p0);
            v = g / (1.f + expf(-a.p1 * g)) * (u + 1.f);
        } else v = (epi == EPI_GLU_SILU ? silu_act(v0) : gelu_tanh_act(v0)) * v1;
        y[(size_t)t * a.ldy + (n >> 1)] = v * a.scale;
        return;
    }
    float* dst = y + (size_t)t * a.ldy + n;
    if (n < a.N) dst[0] = epi_value(a, aux, t, n, v0);
    if (n + 1 < a.N) dst[1] = epi_value(a, aux, t, n + 1, v1);
}

// tensor cores, more than 8 tokens (dense_tc.cu): operand rows of K % 8 == 0 entries on 16-byte boundaries
cudaError_t dense_tc_launch(const DenseArgs& a, const DenseDev& d, cudaStream_t s);
// the same in 32 bits, inputs in three bf16 parts (dense_split.cu)
bool dense_takes_split(const DenseArgs& a);
cudaError_t dense_split_launch(const DenseArgs& a, const DenseDev& d, cudaStream_t s);

}  // namespace b2
