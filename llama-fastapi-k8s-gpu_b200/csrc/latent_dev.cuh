// What the latent attention kernels share (latent_attn.cu, latent_tc.cu): the queries.
#pragma once
#include "layered.h"

namespace b2 {

// entry i of a vector whose first rot_dims entries are rotated by position `pos`, in pairs (i, i + rot_dims / 2) or (2i, 2i + 1)
__device__ __forceinline__ float rotated_at(const float* v, int i, int pos, const RotaryTable& rot) {
    const int half = rot.rot_dims / 2;
    if (i >= rot.rot_dims) return v[i];
    if (rot.pairs) {
        const float cs = rot.cos[(size_t)pos * half + i / 2], sn = rot.sin[(size_t)pos * half + i / 2];
        return i & 1 ? v[i] * cs + v[i - 1] * sn : v[i] * cs - v[i + 1] * sn;
    }
    const int p = i < half ? i : i - half;
    const float cs = rot.cos[(size_t)pos * half + p], sn = rot.sin[(size_t)pos * half + p];
    return i < half ? v[i] * cs - v[i + half] * sn : v[i] * cs + v[i - half] * sn;
}
// entry i of a head's query in the coordinates of the cached rows
__device__ __forceinline__ float query_at(const LatentAttnArgs& a, int t, int h, int i, int pos) {
    if (a.q_raw && i >= a.rank) return rotated_at(a.q_raw + ((size_t)t * a.H + h) * (a.d + a.dr) + a.d, i - a.rank, pos, a.rot);
    return a.qv[((size_t)t * a.H + h) * (a.rank + a.dr) + i];
}

}  // namespace b2
