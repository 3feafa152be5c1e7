// Causal attention of a prompt over the paged f16 cache on the 5th-generation tensor cores (the llama graph; attn_prefill_kernel in
// prefill.cu takes short prompts and page sizes that are no multiple of 64). Same precision: f16 queries, keys, values and
// probabilities, f32 scores, sums and output.
//
// A CTA takes 128 consecutive queries of one head; blocks of 128 keys and values come by tensor copies (page rows of 64, parts of 64
// columns in 128-byte-swizzled rows, two stages). Tensor memory holds the output (128 columns), two score tiles (2 x 128) and the
// probabilities (64 columns), which are the second product's A operand; the next block's scores are computed while this one's softmax
// runs. Eight softmax warps, two threads a query row with 64 key columns each. The output is rescaled only when a row's maximum has
// grown by more than 2^8 and leaves in the operand order of the next GEMM.
#include "kernels.h"
#include "ptx.cuh"
#include "tc05.cuh"
#include "tensor_map.h"
#include <cuda_fp16.h>

#include <algorithm>

namespace b2 {

constexpr int PX_Q = 128, PX_K = 128, PX_PART = PX_Q * 128;       // queries, keys of a block; bytes of a part (128 rows x 64 columns)
constexpr int PX_THREADS = 320;                                   // warps 0-7 softmax, 8 copies, 9 matrix instructions

namespace {
__device__ __forceinline__ float px_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ uint32_t px_pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
}  // namespace

// grid (heads, query tiles, latest first)
template <int HD>
__global__ void __launch_bounds__(PX_THREADS, 1) prompt_attn_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                       const __grid_constant__ CUtensorMap map_v, const int* block_table, int T, int T_pad, int pos0,
                                                                       int n_head, int n_kv, int bt, float scale_log2, __half* out, unsigned int* err) {
    griddep_launch();
    griddep_wait();
    constexpr int PARTS = HD / 64;
    extern __shared__ uint8_t px_smem[];
    __shared__ uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], q_full, s_full[2], p_full, pv_done;
    __shared__ uint32_t tmem_at;
    __shared__ float row_max[2][2][PX_Q], row_sum[2][PX_Q];
    const int h = blockIdx.x, g = h / (n_head / n_kv), row0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * PX_Q;
    const int nq = min(PX_Q, T - row0), p0 = pos0 + row0, p_last = p0 + nq - 1, n_blocks = p_last / PX_K + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* qs = reinterpret_cast<uint8_t*>(((uintptr_t)px_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* ks = qs + PARTS * PX_PART;                    // [stage][part]
    uint8_t* vs = ks + 2 * PARTS * PX_PART;
    if (warp == 9) {
        if (lane == 0) {
            for (int i = 0; i < 2; i++) {
                mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); mbar_init(&s_full[i], 1);
            }
            mbar_init(&q_full, 1); mbar_init(&p_full, 256); mbar_init(&pv_done, 1);
            fence_mbar_init();
        }
        __syncwarp();
        tc_alloc(&tmem_at, 512);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t o_at = tmem_at, s_at = tmem_at + 128, p_at = tmem_at + 384;

    if (warp == 8 && lane == 0) {
        // ================= copies
        mbar_arrive_expect_tx(&q_full, (uint32_t)(PARTS * PX_PART));
        for (int c = 0; c < PARTS; c++) tma_load_3d(qs + c * PX_PART, &map_q, c * 64, h, row0, &q_full);
        for (int i = 0; i < n_blocks; i++) {
            const int st = i & 1, j0 = i * PX_K, halves = j0 + 64 <= p_last ? 2 : 1;
            for (int kv = 0; kv < 2; kv++) {
                uint64_t *full = kv ? &v_full[st] : &k_full[st], *empty = kv ? &v_empty[st] : &k_empty[st];
                uint8_t* dst = (kv ? vs : ks) + st * PARTS * PX_PART;
                if (i >= 2) mbar_wait(empty, ((i >> 1) - 1) & 1, err, 0x80001u, (unsigned)i);
                mbar_arrive_expect_tx(full, (uint32_t)(halves * PARTS * (PX_PART / 2)));
                for (int hf = 0; hf < halves; hf++) {
                    const int j = j0 + 64 * hf, row = (block_table[j / bt] * n_kv + g) * bt + j % bt;
                    for (int c = 0; c < PARTS; c++) tma_load_3d(dst + c * PX_PART + hf * (PX_PART / 2), kv ? &map_v : &map_k, c * 64, row, 0, full);
                }
            }
        }
    } else if (warp == 9 && lane == 0) {
        // ================= matrix instructions (f16 operands)
        constexpr uint32_t BF16 = (1u << 7) | (1u << 10);
        const uint32_t id_s = tc_idesc_bf16(PX_Q, PX_K) & ~BF16, id_o = tc_idesc_bf16(PX_Q, HD, true) & ~BF16;
        const uint32_t qa = smem_u32(qs), ka = smem_u32(ks), va = smem_u32(vs);
        auto scores = [&](int i) {
            mbar_wait(&k_full[i & 1], (i >> 1) & 1, err, 0x80002u, (unsigned)i);
            tc_after_sync();
#pragma unroll
            for (int c = 0; c < PARTS; c++) {
                const uint64_t dq = tc_desc(qa + c * PX_PART), dk = tc_desc(ka + ((i & 1) * PARTS + c) * PX_PART);
#pragma unroll
                for (int k = 0; k < 4; k++) tc_mma(s_at + (i & 1) * PX_K, dq + 2 * k, dk + 2 * k, id_s, (c | k) ? 1u : 0u);
            }
            tc_commit(&s_full[i & 1]);
            tc_commit(&k_empty[i & 1]);
        };
        mbar_wait(&q_full, 0, err, 0x80003u);
        tc_after_sync();
        scores(0);
        for (int i = 0; i < n_blocks; i++) {
            if (i + 1 < n_blocks) scores(i + 1);
            mbar_wait(&v_full[i & 1], (i >> 1) & 1, err, 0x80004u, (unsigned)i);
            mbar_wait(&p_full, i & 1, err, 0x80005u, (unsigned)i);
            tc_after_sync();
            const uint32_t v_at = va + (i & 1) * PARTS * PX_PART;
#pragma unroll
            for (int k = 0; k < PX_K / 16; k++) tc_mma_ts(o_at, p_at + k * 8, tc_desc(v_at + k * 2048, PX_PART), id_o, (i | k) ? 1u : 0u);
            tc_commit(&pv_done);
            tc_commit(&v_empty[i & 1]);
        }
    } else if (warp < 8) {
        // ================= softmax: threads t and t + 128 share query row t, key columns 0-63 and 64-127 of a block
        const int row = threadIdx.x & 127, side = threadIdx.x >> 7, pos = p0 + row;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        float m_ref = -INFINITY, l = 0.f;                         // weights are 2^(score - m_ref)
        for (int i = 0; i < n_blocks; i++) {
            const int j0 = i * PX_K, c0 = j0 + side * 64;
            mbar_wait(&s_full[i & 1], (i >> 1) & 1, err, 0x80006u, (unsigned)i);
            tc_after_sync();
            float s[64];
            {
                uint32_t raw[2][32];
                __syncwarp();
                tc_ld32(s_at + (i & 1) * PX_K + side * 64 + lanes, raw[0]);
                tc_ld32(s_at + (i & 1) * PX_K + side * 64 + 32 + lanes, raw[1]);
                tc_wait_ld();
#pragma unroll
                for (int j = 0; j < 64; j++) s[j] = __uint_as_float(raw[j >> 5][j & 31]) * scale_log2;
            }
            if (j0 + PX_K - 1 > p0) {
#pragma unroll
                for (int j = 0; j < 64; j++) if (c0 + j > pos) s[j] = -INFINITY;
            }
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 64; j++) mx = fmaxf(mx, s[j]);
            row_max[i & 1][side][row] = mx;
            named_bar_sync(1, 256);
            mx = fmaxf(mx, row_max[i & 1][side ^ 1][row]);
            const bool grow = mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY);
            // the previous block's product must be in before the output is rescaled and the probabilities are rewritten
            if (i > 0) { mbar_wait(&pv_done, (i - 1) & 1, err, 0x80007u, (unsigned)i); tc_after_sync(); }
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = grow ? mx : m_ref, f = grow ? px_exp2(m_ref - m_new) : 1.f;
                m_ref = m_new;
                l *= f;
                if (i > 0) {                                      // this side's half of the output
#pragma unroll 1
                    for (int c = side * (HD / 2); c < side * (HD / 2) + HD / 2; c += 32) {
                        uint32_t o[32];
                        tc_ld32(o_at + c + lanes, o);
                        tc_wait_ld();
#pragma unroll
                        for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                        tc_st32(o_at + c + lanes, o);
                    }
                }
            }
            const float ref = m_ref > -INFINITY ? m_ref : 0.f;
            uint32_t p[32];
#pragma unroll
            for (int j = 0; j < 64; j += 2) {
                const float e0 = px_exp2(s[j] - ref), e1 = px_exp2(s[j + 1] - ref);
                l += e0 + e1;
                p[j >> 1] = px_pack(e0, e1);
            }
            __syncwarp();
            tc_st32(p_at + side * 32 + lanes, p);
            tc_wait_st();
            if (i == n_blocks - 1 && p_last - j0 + 1 < PX_K) {
                // rows past the sequence: whatever shared memory or the page holds must not meet the zero weights as values
                mbar_wait(&v_full[i & 1], (i >> 1) & 1, err, 0x80008u, (unsigned)i);
                const int r0 = p_last - j0 + 1, n_bad = PX_K - r0;
                for (int e = threadIdx.x; e < PARTS * n_bad * 8; e += 256) {
                    const int c = e / (n_bad * 8), rr = r0 + e / 8 % n_bad;
                    *reinterpret_cast<uint4*>(vs + ((i & 1) * PARTS + c) * PX_PART + rr * 128 + (e & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
            }
            tc_before_sync();
            mbar_arrive(&p_full);
        }
        row_sum[side][row] = l;
        named_bar_sync(1, 256);
        const float inv = 1.f / (l + row_sum[side ^ 1][row]);
        mbar_wait(&pv_done, (n_blocks - 1) & 1, err, 0x80009u);
        tc_after_sync();
        for (int c = side * (HD / 2); c < side * (HD / 2) + HD / 2; c += 32) {
            uint32_t o[32];
            __syncwarp();
            tc_ld32(o_at + c + lanes, o);
            tc_wait_ld();
            if (row < nq) {
#pragma unroll
                for (int e = 0; e < 32; e += 8) {
                    uint32_t u[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) u[k] = px_pack(__uint_as_float(o[e + 2 * k]) * inv, __uint_as_float(o[e + 2 * k + 1]) * inv);
                    // [column / 8][T_pad][8]: neighbouring rows are neighbouring 16-byte pieces
                    *reinterpret_cast<uint4*>(out + ((size_t)((h * HD + c + e) >> 3) * T_pad + row0 + row) * 8) = make_uint4(u[0], u[1], u[2], u[3]);
                }
            }
        }
        tc_before_sync();
    }
    __syncthreads();
    if (warp == 9) tc_dealloc(tmem_at, 512);
}

// Prompts of whole tiles and page sizes that a 64-row copy stays inside of.
bool prompt_attn_takes_tc(int T, int hd, int bt) { return T >= 96 && (hd == 64 || hd == 128) && bt % 64 == 0; }

cudaError_t prompt_attn_tc_launch(const __half* qh, const __half* k_cache, const __half* v_cache, long pool_rows, const int* block_table, int T, int T_pad, int pos0,
                                  int n_head, int n_kv, int hd, int bt, __half* out, cudaStream_t s) {
    if (!prompt_attn_takes_tc(T, hd, bt)) return cudaErrorInvalidValue;
    const size_t smem = (size_t)5 * (hd / 64) * PX_PART + 1024;
    static const bool ready = cudaFuncSetAttribute(prompt_attn_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 5 * PX_PART + 1024) == cudaSuccess &&
                              cudaFuncSetAttribute(prompt_attn_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 10 * PX_PART + 1024) == cudaSuccess;
    CUtensorMap mq, mk, mv;       // 16-bit entries are copied as they are: the maps' element type does not matter
    if (!ready || !bf16_heads_map(&mq, qh, hd, n_head, T, PX_Q) || !bf16_rows_map(&mk, k_cache, hd, pool_rows, hd, 1, 0, 64) ||
        !bf16_rows_map(&mv, v_cache, hd, pool_rows, hd, 1, 0, 64)) return cudaErrorInvalidValue;
    const float scale_log2 = 1.4426950408889634f / sqrtf((float)hd);
    const dim3 grid(n_head, (T + PX_Q - 1) / PX_Q), block(PX_THREADS);
    return hd == 64 ? launch_chain(prompt_attn_tc_kernel<64>, grid, block, smem, s, mq, mk, mv, block_table, T, T_pad, pos0, n_head, n_kv, bt, scale_log2, out, kernel_error_word())
                    : launch_chain(prompt_attn_tc_kernel<128>, grid, block, smem, s, mq, mk, mv, block_table, T, T_pad, pos0, n_head, n_kv, bt, scale_log2, out, kernel_error_word());
}

}  // namespace b2
