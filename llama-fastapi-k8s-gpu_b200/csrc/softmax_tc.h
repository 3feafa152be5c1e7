// Softmax attention of steps of more than 8 tokens on the tensor cores (softmax_tc.cu), shared by the mixers of the layer-list models.
#pragma once
#include "layered.h"

namespace b2 {

// Query i sees key j when j <= i and (window <= 0, i - j < window, or j < keep_first). Grouped query heads over paged bf16 keys and
// values [page][G][block_tokens][d | dv].
struct SoftmaxTcArgs {
    const float* q;                                    // [T][H][d], 16-byte aligned
    const void* k_pool; const void* v_pool; long pool_rows;      // rows of either pool: pages * G * block_tokens
    int* const* block_tables; int block_tokens;
    int H, G, d, dv, window, keep_first;
    float scale, softcap;                              // softcap <= 0: none
    const float* sink;                                 // [H] or null
    const float* gate; int ld_gate; int gate_per_head; // sigmoid output gate or null (as in SinkAttnArgs)
    float* out; __nv_bfloat16* out_bf16; int ld_out;   // out[t][h * dv + i], or rounded
    int skip;                                          // leading tiles of the step that are not this launch's (at most the one-token ones)
};
bool softmax_takes_tc(const SoftmaxTcArgs& a);
cudaError_t softmax_tc_launch(const SoftmaxTcArgs& a, const RaggedDev& r, cudaStream_t s);

}  // namespace b2
