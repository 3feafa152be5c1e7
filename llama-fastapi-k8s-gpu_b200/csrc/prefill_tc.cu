// Attention of a prompt's queries over the paged f16 cache on the 5th-generation tensor cores (GGUF models; prefill.cu has the mma.sync form for few keys
// and pages of other sizes). Rounded where that one rounds: queries and cached rows f16 as they are, scores and sums 32-bit, probabilities f16 for the
// weighted sum, the output f16 in the operand order of the next product. (A probability is taken against a maximum that may lag by 2^8, so other
// bits of it are rounded, the same number of them.)
//
// A CTA takes 128 consecutive queries of one head; blocks of 128 keys and values come by tensor copies (64 columns a part in 128-byte-swizzled rows, two
// stages). Tensor memory holds the output (up to 128 columns), two score tiles (2 x 128) and two of probabilities (2 x 64), the A operand of the second
// product. Warps 0-7: softmax, two threads a query with 64 keys of a block each; 8: copies; 9: matrix instructions. The next block's scores are computed
// while this one's softmax runs. Bound by the chain of a block's scores, softmax and sums; 128 CTAs of 1 to 4 blocks for 512 tokens of 32 heads.
// 32 heads of 128 over 8 (B200), us a layer with the wait for the kernel before it: 512 tokens 33 with mma.sync, 13 here. Whole prompts of two layers of 4096:
// 300 tokens 612 -> 572 us, 512 744 -> 672, 30 behind 500 350 -> 317, 8 behind 2000 457 -> 336, 512 behind 2000 954 -> 710.
#include "kernels.h"
#include "ptx.cuh"
#include "tc05.cuh"
#include "tensor_map.h"
#include <cuda_fp16.h>

namespace b2 {

constexpr int PT_Q = 128, PT_K = 128, PT_PART = 128 * 128;        // queries, keys of a block; bytes of a part (128 rows x 64 columns)
constexpr int PT_THREADS = 320;
constexpr int PT_TC_KEYS = 128;                                   // from more keys on

namespace {
__device__ __forceinline__ float pt_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ uint32_t pt_pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// f16 operands, f32 sums (tc_idesc_bf16 without the bits that say bf16)
__device__ __forceinline__ uint32_t pt_idesc(int N, bool b_rows_are_k) { return tc_idesc_bf16(PT_Q, N, b_rows_are_k) & ~((1u << 7) | (1u << 10)); }
}  // namespace

// CTAs: (tile of queries, head), the tiles with the most keys first
template <int HD>
__global__ void __launch_bounds__(PT_THREADS, 1) attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                        const __grid_constant__ CUtensorMap map_v, const int* __restrict__ block_table, int T, int T_pad,
                                                                        int pos0, int n_head, int n_kv, int bt, float scale_log2, __half* __restrict__ out,
                                                                        unsigned int* err) {
    constexpr int PARTS = HD / 64;
    extern __shared__ uint8_t pt_smem[];
    __shared__ uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], pv_done[2], o_full;
    __shared__ uint32_t tmem_at;
    __shared__ float row_max[2][2][PT_Q], row_sum[2][PT_Q];
    const int n_tiles = (T + PT_Q - 1) / PT_Q, q0 = (n_tiles - 1 - (int)blockIdx.x / n_head) * PT_Q, head = blockIdx.x % n_head, kvh = head / (n_head / n_kv);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp: known to be uniform)
    const int nq = min(PT_Q, T - q0), p0 = pos0 + q0, p_last = p0 + nq - 1, n_blocks = p_last / PT_K + 1;
    uint8_t* qs = reinterpret_cast<uint8_t*>(((uintptr_t)pt_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* ks = qs + PARTS * PT_PART;                           // [stage][part]
    uint8_t* vs = ks + 2 * PARTS * PT_PART;
    if (warp == 9) {
        if (lane == 0) {
            mbar_init(&q_full, 1); mbar_init(&o_full, 1);
            for (int i = 0; i < 2; i++) {
                mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
                mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 256); mbar_init(&pv_done[i], 1);
            }
            fence_mbar_init();
        }
        __syncwarp();
        tc_alloc(&tmem_at, 512);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    griddep_launch();                                             // (tensor memory is this CTA's: see softmax_tc.cu)
    griddep_wait();
    const uint32_t o_at = tmem_at, s_at = tmem_at + 128, p_at = tmem_at + 384;

    if (warp == 8) {
        // ================= copies (all lanes run the loop, one issues: see dense_tc.cu)
        const bool one = elect_one();
        if (one) {
            mbar_arrive_expect_tx(&q_full, PARTS * PT_PART);
            for (int c = 0; c < PARTS; c++) tma_load_3d(qs + c * PT_PART, &map_q, head * HD + c * 64, q0, 0, &q_full);
        }
        for (int i = 0; i < n_blocks; i++) {
            const int st = i & 1, j0 = i * PT_K, halves = j0 + 64 <= p_last ? 2 : 1;
            int row[2];
#pragma unroll
            for (int hf = 0; hf < 2; hf++) {
                const int j = min(j0 + 64 * hf, p_last);          // (a page holds whole halves)
                row[hf] = (block_table[j / bt] * n_kv + kvh) * bt + (j0 + 64 * hf) % bt;
            }
            for (int kv = 0; kv < 2; kv++) {
                uint64_t *full = kv ? &v_full[st] : &k_full[st], *empty = kv ? &v_empty[st] : &k_empty[st];
                uint8_t* dst = (kv ? vs : ks) + st * PARTS * PT_PART;
                if (i >= 2) mbar_wait_warp(empty, ((i >> 1) - 1) & 1, err, 0x80001u, (unsigned)i);
                if (!one) continue;
                mbar_arrive_expect_tx(full, (uint32_t)(halves * PARTS * (PT_PART / 2)));
                for (int hf = 0; hf < halves; hf++)
                    for (int c = 0; c < PARTS; c++) tma_load_3d(dst + c * PT_PART + hf * (PT_PART / 2), kv ? &map_v : &map_k, c * 64, row[hf], 0, full);
            }
        }
    } else if (warp == 9) {
        // ================= matrix instructions
        const bool one = elect_one();
        const uint32_t id_s = pt_idesc(PT_K, false), id_o = pt_idesc(HD, true);
        const uint64_t dq = tc_desc(smem_u32(qs));
        const uint32_t ka = smem_u32(ks), va = smem_u32(vs);
        auto scores = [&](int i) {
            mbar_wait_warp(&k_full[i & 1], (i >> 1) & 1, err, 0x80002u, (unsigned)i);
            tc_after_sync();
            if (!one) return;
            const uint64_t dk = tc_desc(ka + (i & 1) * PARTS * PT_PART);
#pragma unroll
            for (int c = 0; c < PARTS; c++)
#pragma unroll
                for (int k = 0; k < 4; k++) tc_mma(s_at + (i & 1) * PT_K, dq + c * (PT_PART >> 4) + 2 * k, dk + c * (PT_PART >> 4) + 2 * k, id_s, (c | k) ? 1u : 0u);
            tc_commit(&s_full[i & 1]);
            tc_commit(&k_empty[i & 1]);
        };
        mbar_wait_warp(&q_full, 0, err, 0x80003u);
        tc_after_sync();
        scores(0);
        for (int i = 0; i < n_blocks; i++) {
            if (i + 1 < n_blocks) scores(i + 1);                  // (the scores they replace have been read: probabilities made of them are in use)
            mbar_wait_warp(&v_full[i & 1], (i >> 1) & 1, err, 0x80004u, (unsigned)i);
            mbar_wait_warp(&p_full[i & 1], (i >> 1) & 1, err, 0x80005u, (unsigned)i);
            tc_after_sync();
            if (!one) continue;
            const uint64_t dv = tc_desc(va + (i & 1) * PARTS * PT_PART, PT_PART);
            // 16 keys a product: queries ahead of all of them take no part (a value that is no number would reach them through a weight of 0)
#pragma unroll
            for (int k = 0; k < PT_K / 16; k++) {
                const int j = i * PT_K + 16 * k;
                if (j <= p_last) tc_mma_ts_from_row(o_at, p_at + (i & 1) * (PT_K / 2) + k * 8, dv + k * (2048 >> 4), id_o, (i | k) ? 1u : 0u, j - p0);
            }
            tc_commit(&pv_done[i & 1]);
            tc_commit(&v_empty[i & 1]);
            if (i == n_blocks - 1) tc_commit(&o_full);
        }
    } else {
        // ================= softmax: threads t and t + 128 share query row t, keys 0-63 and 64-127 of a block
        const int row = threadIdx.x & 127, side = threadIdx.x >> 7, pos = p0 + row;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        float m_ref = -INFINITY, l = 0.f;                         // weights are 2^(score - m_ref)
        for (int i = 0; i < n_blocks; i++) {
            const int st = i & 1, j0 = i * PT_K, c0 = j0 + side * 64;
            const uint32_t phase = (i >> 1) & 1;
            mbar_wait(&s_full[st], phase, err, 0x80006u, (unsigned)i);
            tc_after_sync();
            uint32_t raw[2][32];
            __syncwarp();
            tc_ld32(s_at + st * PT_K + side * 64 + lanes, raw[0]);
            tc_ld32(s_at + st * PT_K + side * 64 + 32 + lanes, raw[1]);
            tc_wait_ld();
            float s[64];
#pragma unroll
            for (int j = 0; j < 64; j++) s[j] = __uint_as_float(raw[j >> 5][j & 31]) * scale_log2;
            if (j0 + PT_K - 1 > p0) {
#pragma unroll
                for (int j = 0; j < 64; j++) if (c0 + j > pos) s[j] = -INFINITY;
            }
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 64; j++) mx = fmaxf(mx, s[j]);
            row_max[st][side][row] = mx;
            named_bar_sync(1 + (warp & 3), 64);                   // (the two warps of these rows)
            mx = fmaxf(mx, row_max[st][side ^ 1][row]);
            const bool grow = mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY);
            const float m_old = m_ref;
            if (grow) { m_ref = mx; l *= pt_exp2(m_old - mx); }
            const float ref = m_ref > -INFINITY ? m_ref : 0.f;
            uint32_t p[32];
#pragma unroll
            for (int j = 0; j < 64; j += 2) {
                const float e0 = pt_exp2(s[j] - ref), e1 = pt_exp2(s[j + 1] - ref);
                l += e0 + e1;
                p[j >> 1] = pt_pack(e0, e1);
            }
            // the sum before last must be in before its probabilities are overwritten, the last one before the output is rescaled
            if (i > 1) { mbar_wait(&pv_done[st], phase ^ 1, err, 0x80007u, (unsigned)i); tc_after_sync(); }
            if (i > 0 && __any_sync(0xffffffffu, grow)) {
                mbar_wait(&pv_done[st ^ 1], ((i - 1) >> 1) & 1, err, 0x80008u, (unsigned)i);
                tc_after_sync();
                const float f = grow ? pt_exp2(m_old - m_ref) : 1.f;
                __syncwarp();
#pragma unroll
                for (int c = 0; c < HD / 2; c += 32) {            // this side's columns
                    uint32_t o[32];
                    tc_ld32(o_at + side * (HD / 2) + c + lanes, o);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                    tc_st32(o_at + side * (HD / 2) + c + lanes, o);
                }
            }
            __syncwarp();
            tc_st32(p_at + st * (PT_K / 2) + side * 32 + lanes, p);
            tc_wait_st();
            if (i == n_blocks - 1 && (p_last + 1) % 16) {
                // rows past the sequence in the last 16 that are multiplied: whatever the page holds must not meet the zero weights as values
                mbar_wait(&v_full[st], phase, err, 0x80009u, (unsigned)i);
                const int r0 = p_last - j0 + 1, n_bad = 16 - r0 % 16;
                for (int e = threadIdx.x; e < PARTS * n_bad * 8; e += 256) {
                    const int c = e / (n_bad * 8), rr = r0 + e / 8 % n_bad;
                    *reinterpret_cast<uint4*>(vs + (st * PARTS + c) * PT_PART + rr * 128 + (e & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
            }
            tc_before_sync();
            mbar_arrive(&p_full[st]);
        }
        row_sum[side][row] = l;
        named_bar_sync(1 + (warp & 3), 64);
        const float inv = 1.f / (l + row_sum[side ^ 1][row]);
        mbar_wait(&o_full, 0, err, 0x8000au);
        tc_after_sync();
#pragma unroll
        for (int c = 0; c < HD / 2; c += 32) {
            uint32_t o[32];
            const int d = side * (HD / 2) + c;
            __syncwarp();
            tc_ld32(o_at + d + lanes, o);
            tc_wait_ld();
            if (row >= nq) continue;
#pragma unroll
            for (int e = 0; e < 32; e += 8) {                     // eight columns of a token are 16 bytes, neighbouring tokens' side by side
                uint32_t u[4];
#pragma unroll
                for (int k = 0; k < 4; k++) u[k] = pt_pack(__uint_as_float(o[e + 2 * k]) * inv, __uint_as_float(o[e + 2 * k + 1]) * inv);
                *reinterpret_cast<uint4*>(out + ((size_t)((head * HD + d + e) >> 3) * T_pad + q0 + row) * 8) = make_uint4(u[0], u[1], u[2], u[3]);
            }
        }
        tc_before_sync();
    }
    __syncthreads();
    if (warp == 9) tc_dealloc(tmem_at, 512);
}

// ---------------------------------------------------------------- host side
// Pages of whole 64-key halves, and more keys than one block: up to 128 keys the other form's one or two tiles of them take 5 to 8 us on four to eight times as
// many CTAs (130 tokens, two layers: 462 us there, 452 here).
bool attn_prefill_takes_tc(int T, int pos0, int hd, int bt) { return (hd == 64 || hd == 128) && bt % 64 == 0 && pos0 + T > PT_TC_KEYS; }

cudaError_t attn_prefill_tc_launch(const __half* qh, const __half* k_cache, const __half* v_cache, long pool_rows, const int* block_table, int T, int T_pad, int pos0,
                                   int n_head, int n_kv, int hd, int bt, __half* out, cudaStream_t s) {
    if (n_kv <= 0 || n_head % n_kv || !attn_prefill_takes_tc(T, pos0, hd, bt)) return cudaErrorInvalidValue;
    const int parts = hd / 64;
    constexpr int most = 10 * PT_PART + 1024;
    if (!allow_smem<attn_prefill_tc_kernel<64>>(most) || !allow_smem<attn_prefill_tc_kernel<128>>(most)) return cudaErrorInvalidValue;
    CUtensorMap mq, mk, mv;                                       // (copies move 16-bit entries whatever their format)
    if (!bf16_rows_map(&mq, qh, (long)n_head * hd, T, (long)n_head * hd, 1, 0, PT_Q) || !bf16_rows_map(&mk, k_cache, hd, pool_rows, hd, 1, 0, 64) ||
        !bf16_rows_map(&mv, v_cache, hd, pool_rows, hd, 1, 0, 64)) return cudaErrorInvalidValue;
    const dim3 grid((T + PT_Q - 1) / PT_Q * n_head), block(PT_THREADS);
    const size_t smem = (size_t)5 * parts * PT_PART + 1024;
    const float scale_log2 = 1.4426950408889634f / sqrtf((float)hd);
    if (hd == 64) return launch_chain(attn_prefill_tc_kernel<64>, grid, block, smem, s, mq, mk, mv, block_table, T, T_pad, pos0, n_head, n_kv, bt, scale_log2, out, kernel_error_word());
    return launch_chain(attn_prefill_tc_kernel<128>, grid, block, smem, s, mq, mk, mv, block_table, T, T_pad, pos0, n_head, n_kv, bt, scale_log2, out, kernel_error_word());
}

}  // namespace b2
