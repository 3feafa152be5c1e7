// Latent attention of steps of more than 8 tokens on the 5th-generation tensor cores (bf16 pages). Rounded where latent_attn_mma_kernel
// (latent_attn.cu) rounds: queries scaled, then rounded to bf16; cached rows as they are; probabilities rounded to bf16 for the weighted
// sum, 32-bit everywhere else. (Here the running maximum that a probability is taken against may lag by 2^8, so other bits are rounded.)
//
// A CTA takes 128 consecutive queries of one head and up to 256 latent columns of the output (tensor memory holds 128 lanes x 512
// columns: 256 for the output, two score tiles of 64, two probability tiles of 32, so a 512-wide latent is two CTAs that both
// compute the scores). The queries stay in shared memory; blocks of 64 cached rows come by tensor copies as parts of 64 columns and
// serve both products: as rows of K for the scores, and, read across (N contiguous), as the values. Probabilities go to tensor
// memory and are the second product's A operand.
// Warps 0-3: softmax, one query a thread; 4: copies; 5: matrix instructions. The parts that are not values of this CTA are reloaded
// while the softmax runs, and their share of the next block's scores is computed under it. The output is rescaled only when a
// row's maximum has grown by more than 2^8 since the last time.
// Bound by the chain of a block's scores, softmax and sums: six warps an SM, tensor pipe busy for 26 to 30 % of the time, issue slots for 18 % (ncu).
// 2048 tokens, 16 heads, rows of 512 + 64 (B200): 1640 us a layer with mma.sync, 207 here (the rotated parts of the queries: below); rows of 512,
// nothing rotated: 170.
#include "kernels.h"
#include "latent_dev.cuh"
#include "layered.h"
#include "ptx.cuh"
#include "tc05.cuh"
#include "tensor_map.h"

#include <algorithm>
#include <stdlib.h>

namespace b2 {

constexpr int LC_Q = 128, LC_K = 64, LC_PART = 64;          // queries, cached rows of a block, columns of a part
constexpr int LC_QPART = LC_Q * LC_PART * 2, LC_KPART = LC_K * LC_PART * 2;
constexpr int LC_V = 256;                                   // latent columns of the output per CTA

namespace {
__device__ __forceinline__ uint32_t lc_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
}  // namespace

// CTAs: (64-query tile, head, column chunk), latest tiles first (odd tiles of a sequence belong to the CTA before them), then (one-token
// sequence, chunk) for the first n_packed tiles: there the rows are the heads, which all read the same keys
__global__ void __launch_bounds__(192, 1) latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q,
                                                                const __grid_constant__ CUtensorMap map_h, const LatentAttnArgs a, const RaggedDev r,
                                                                int n_packed, int n_chunks, __nv_bfloat16* out, unsigned int* err) {
    extern __shared__ uint8_t lc_smem[];
    __shared__ uint64_t rest_full, val_full, rest_empty, val_empty, q_full, s_full[2], p_full[2], pv_done;
    __shared__ uint32_t tmem_at;
    const int whole = (r.n_tiles - n_packed) * a.H, at = blockIdx.x / n_chunks, chunk = blockIdx.x % n_chunks;
    const bool packed = at >= whole;
    const int tile = packed ? at - whole : r.n_tiles - 1 - at / a.H, h = packed ? 0 : at % a.H;
    const int seg = r.tile_seg[tile], row0 = r.tile_row0[tile];
    if (((row0 - r.seg_start[seg]) / 64) & 1) return;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp: known to be uniform)
    const int nq = packed ? a.H : min(LC_Q, r.seg_start[seg] + r.seg_len[seg] - row0);      // rows in use
    const int p0 = r.seg_pos0[seg] + row0 - r.seg_start[seg], p_last = packed ? p0 : p0 + nq - 1;
    const int* table = a.block_tables[r.seg_slot[seg]];
    const int n_parts = (a.rank + a.dr + LC_PART - 1) / LC_PART, v0 = chunk * (LC_V / LC_PART), n_val = min(LC_V, a.rank - chunk * LC_V) / LC_PART;
    uint8_t* qs = reinterpret_cast<uint8_t*>(((uintptr_t)lc_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* ks = qs + (size_t)n_parts * LC_QPART;
    const int b0 = max(0, p0 - a.window + 1) / LC_K, n_blocks = p_last / LC_K + 1 - b0;
    if (warp == 5) {
        if (lane == 0) {
            mbar_init(&rest_full, 1); mbar_init(&val_full, 1); mbar_init(&rest_empty, 1); mbar_init(&val_empty, 1); mbar_init(&q_full, 1 + 128);
            for (int i = 0; i < 2; i++) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 128); }
            mbar_init(&pv_done, 1);
            fence_mbar_init();
        }
        __syncwarp();
        tc_alloc(&tmem_at, 512);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    // The next kernel is let in once tensor memory is this CTA's: had it come first on this SM, it would hold its own and wait for this kernel
    // to end, and this CTA for that memory. (What is read above is the step's description, older than the kernel before this one.)
    griddep_launch();
    griddep_wait();
    const uint32_t tmem = tmem_at, o_at = tmem, s_at = tmem + LC_V, p_at = tmem + LC_V + 2 * LC_K;

    if (warp == 4) {
        // ================= copies: the latent parts of the queries, then blocks of cached rows (all lanes run the loop, one issues: see dense_tc.cu)
        const bool one = elect_one();
        const int q_parts = a.rank / LC_PART, n_rest = n_parts - n_val;
        if (one) mbar_arrive_expect_tx(&q_full, (uint32_t)(q_parts * LC_QPART));
        if (one) for (int c = 0; c < q_parts; c++) tma_load_3d(qs + (size_t)c * LC_QPART, packed ? &map_h : &map_q, c * LC_PART, h, row0, &q_full);
        for (int i = 0; i < n_blocks; i++) {
            const int j0 = (b0 + i) * LC_K, row = table[j0 / a.block_tokens] * a.block_tokens + j0 % a.block_tokens;
            for (int half = 0; half < 2; half++) {
                uint64_t *full = half ? &val_full : &rest_full, *empty = half ? &val_empty : &rest_empty;
                if (half == 0 && n_rest == 0) continue;
                if (i > 0) mbar_wait_warp(empty, (i - 1) & 1, err, 0x60001u, (unsigned)i);
                if (!one) continue;
                mbar_arrive_expect_tx(full, (uint32_t)((half ? n_val : n_rest) * LC_KPART));
                for (int c = 0; c < n_parts; c++)
                    if ((c >= v0 && c < v0 + n_val) == (half == 1)) tma_load_3d(ks + (size_t)c * LC_KPART, &map_k, c * LC_PART, row, 0, full);
            }
        }
    } else if (warp == 5) {
        const bool one = elect_one();
        // ================= matrix instructions
        const uint32_t id_s = tc_idesc_bf16(LC_Q, LC_K), id_o = tc_idesc_bf16(LC_Q, n_val * LC_PART, true);
        const uint32_t qa = smem_u32(qs), ka = smem_u32(ks);
        bool first = true;
        auto scores = [&](int i, bool values) {              // one group of parts of block i's scores
            for (int c = 0; c < n_parts; c++) {
                if ((c >= v0 && c < v0 + n_val) != values) continue;
                const uint64_t dq = tc_desc(qa + c * LC_QPART), dk = tc_desc(ka + c * LC_KPART);
                if (one)
#pragma unroll
                    for (int k = 0; k < LC_PART / 16; k++) tc_mma(s_at + (i & 1) * LC_K, dq + 2 * k, dk + 2 * k, id_s, first && k == 0 ? 0u : 1u);
                first = false;
            }
        };
        const bool any_rest = n_parts > n_val;
        mbar_wait_warp(&q_full, 0, err, 0x60002u);
        tc_after_sync();
        if (any_rest) { mbar_wait_warp(&rest_full, 0, err, 0x60003u); tc_after_sync(); scores(0, false); if (one) tc_commit(&rest_empty); }
        mbar_wait_warp(&val_full, 0, err, 0x60004u);
        tc_after_sync();
        scores(0, true);
        if (one) tc_commit(&s_full[0]);
        for (int i = 0; i < n_blocks; i++) {
            const bool more = i + 1 < n_blocks;
            first = true;
            if (more && any_rest) { mbar_wait_warp(&rest_full, (i + 1) & 1, err, 0x60005u, (unsigned)i); tc_after_sync(); scores(i + 1, false); if (one) tc_commit(&rest_empty); }
            mbar_wait_warp(&p_full[i & 1], (i >> 1) & 1, err, 0x60006u, (unsigned)i);
            tc_after_sync();
            if (one) {
#pragma unroll
                for (int k = 0; k < LC_K / 16; k++)
                    tc_mma_ts(o_at, p_at + (i & 1) * (LC_K / 2) + k * 8, tc_desc(ka + v0 * LC_KPART + k * 2048, LC_KPART), id_o, (i | k) ? 1u : 0u);
                tc_commit(&pv_done);
                tc_commit(&val_empty);
            }
            if (more) {
                mbar_wait_warp(&val_full, (i + 1) & 1, err, 0x60007u, (unsigned)i);
                tc_after_sync();
                scores(i + 1, true);
                if (one) tc_commit(&s_full[(i + 1) & 1]);
            }
        }
    } else if (warp < 4) {
        // ================= softmax: thread = query row
        const int row = threadIdx.x, pos = packed ? p0 : p0 + row;
        const int t = packed ? row0 : row0 + row, hd = packed ? min(row, a.H - 1) : h;      // the row's token and head
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        // the rotated part of the queries (and zeros up to the part's 64 columns), rows past the tile as zeros: a warp's 32 rows, a lane two neighbouring
        // entries, eight rows read ahead of their stores and without a branch between the reads (a thread per row, branches around every entry:
        // 28 us a CTA, 290 us a layer; 207 here)
        // (queries without a latent of their own have been rotated where the rest of them lies)
        const int half = a.q_raw ? a.rot.rot_dims / 2 : 0, ld_q = a.q_raw ? a.d + a.dr : a.rank + a.dr;
        const float* queries = a.q_raw ? a.q_raw + a.d : a.qv + a.rank;
        for (int e = 2 * lane; e < n_parts * LC_PART - a.rank; e += 64) {
            int own[2], other[2], turn[2];
            float sign[2];                                      // entry = own * cos + sign * other * sin; an entry that is not rotated: sign 0
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int i = min(e + k, a.dr - 1);
                const bool rot = i < 2 * half, first = a.rot.pairs ? !(i & 1) : i < half;
                own[k] = i;
                other[k] = !rot ? i : a.rot.pairs ? i ^ 1 : first ? i + half : i - half;
                turn[k] = !rot ? -1 : a.rot.pairs ? i / 2 : first ? i : i - half;
                sign[k] = !rot ? 0.f : first ? -1.f : 1.f;
            }
            for (int q0 = warp * 32; q0 < warp * 32 + 32; q0 += 8) {
                float v[8][2], w[8][2], cs[8][2], sn[8][2];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int q = min(q0 + u, nq - 1), qt = packed ? row0 : row0 + q, qh = packed ? q : h, qp = packed ? p0 : p0 + q;
                    const float* from = queries + ((size_t)qt * a.H + qh) * ld_q;
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const size_t at = turn[k] < 0 ? 0 : (size_t)qp * half + turn[k];
                        v[u][k] = from[own[k]]; w[u][k] = from[other[k]];
                        cs[u][k] = half > 0 ? a.rot.cos[at] : 1.f; sn[u][k] = half > 0 ? a.rot.sin[at] : 0.f;
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    float y[2];
#pragma unroll
                    for (int k = 0; k < 2; k++) y[k] = q0 + u < nq && e + k < a.dr ? (turn[k] < 0 ? v[u][k] : v[u][k] * cs[u][k] + sign[k] * w[u][k] * sn[u][k]) * a.scale : 0.f;
                    *reinterpret_cast<uint32_t*>(qs + (size_t)((a.rank + e) / LC_PART) * LC_QPART + (q0 + u) * 128 + (((e % LC_PART / 8) ^ (u & 7)) << 4) + e % 8 * 2) =
                        lc_pack(y[0], y[1]);
                }
            }
        }
        fence_proxy_async();
        mbar_arrive(&q_full);
        constexpr float LOG2E = 1.4426950408889634f;
        float m_ref = a.sink ? a.sink[hd] * LOG2E : -INFINITY, l = a.sink ? 1.f : 0.f;           // log2 domain: weights are 2^(score - m_ref)
        for (int i = 0; i < n_blocks; i++) {
            const int j0 = (b0 + i) * LC_K;
            mbar_wait(&s_full[i & 1], (i >> 1) & 1, err, 0x60008u, (unsigned)i);
            tc_after_sync();
            uint32_t raw[2][32];
            __syncwarp();
            tc_ld32(s_at + (i & 1) * LC_K + lanes, raw[0]);
            tc_ld32(s_at + (i & 1) * LC_K + 32 + lanes, raw[1]);
            tc_wait_ld();
            float s[LC_K];
#pragma unroll
            for (int j = 0; j < LC_K; j++) s[j] = __uint_as_float(raw[j >> 5][j & 31]) * LOG2E;
            if (j0 + LC_K - 1 > p0 || p_last - j0 >= a.window) {
                const int lo = pos - a.window + 1 - j0, hi = pos - j0;          // visible columns of this row
#pragma unroll
                for (int j = 0; j < LC_K; j++) if (j < lo || j > hi) s[j] = -INFINITY;
            }
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < LC_K; j++) mx = fmaxf(mx, s[j]);
            const bool grow = mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY);
            // the previous block's sum must be in before the output is rescaled, and before the older probability tile is rewritten
            if (i > 0) { mbar_wait(&pv_done, (i - 1) & 1, err, 0x60009u, (unsigned)i); tc_after_sync(); }
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = grow ? mx : m_ref, f = grow ? exp2f(m_ref - m_new) : 1.f;
                m_ref = m_new;
                l *= f;
                if (i > 0) {
                    for (int c = 0; c < n_val * LC_PART; c += 32) {
                        uint32_t o[32];
                        tc_ld32(o_at + c + lanes, o);
                        tc_wait_ld();
#pragma unroll
                        for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                        tc_st32(o_at + c + lanes, o);
                    }
                }
            }
            const float ref = m_ref > -INFINITY ? m_ref : 0.f;                  // a row that has seen no key yet: all weights are 0
            uint32_t p[32];
#pragma unroll
            for (int j = 0; j < LC_K; j += 2) {
                const float e0 = exp2f(s[j] - ref), e1 = exp2f(s[j + 1] - ref);
                l += e0 + e1;
                p[j >> 1] = lc_pack(e0, e1);
            }
            __syncwarp();
            tc_st32(p_at + (i & 1) * (LC_K / 2) + lanes, p);
            tc_wait_st();
            if (i == n_blocks - 1 && p_last - j0 + 1 < LC_K) {
                // rows of the last block past the sequence: whatever the page holds must not meet the zero weights as values
                const int r0 = p_last - j0 + 1, n_bad = LC_K - r0;
                for (int e = threadIdx.x; e < n_val * n_bad * 8; e += 128) {
                    const int c = e / (n_bad * 8), rr = r0 + e / 8 % n_bad;
                    *reinterpret_cast<uint4*>(ks + (size_t)(v0 + c) * LC_KPART + rr * 128 + (e & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
            }
            tc_before_sync();
            mbar_arrive(&p_full[i & 1]);
        }
        mbar_wait(&pv_done, (n_blocks - 1) & 1, err, 0x6000au);
        tc_after_sync();
        const float inv = 1.f / l;
        __nv_bfloat16* dst = out + ((size_t)t * a.H + hd) * a.rank + chunk * LC_V;
        for (int c = 0; c < n_val * LC_PART; c += 32) {
            uint32_t o[32];
            __syncwarp();
            tc_ld32(o_at + c + lanes, o);
            tc_wait_ld();
            if (row < nq) {
#pragma unroll
                for (int e = 0; e < 32; e += 8) {
                    uint32_t u[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) u[q] = lc_pack(__uint_as_float(o[e + 2 * q]) * inv, __uint_as_float(o[e + 2 * q + 1]) * inv);
                    *reinterpret_cast<uint4*>(dst + c + e) = make_uint4(u[0], u[1], u[2], u[3]);
                }
            }
        }
        tc_before_sync();
    }
    __syncthreads();
    if (warp == 5) tc_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- host side
// Rows of 64-column parts that fit shared memory beside the queries (9 of them), whole chunks of output columns, pages of whole blocks; of
// the step only what the few-token kernels do not take (see softmax_tc.cu). 16 heads, rows of 512 + 64, us a layer with the preparation,
// mma.sync / here: a prompt of 9 tokens 52 / 36, of 64 93 / 44, of 255 120 / 63; 32 prompts of 60 568 / 212; one token of each of 32 sequences
// behind 60 208 / 38, behind 1900 2087 / 114; 512 tokens beside 31 sequences that decode behind 500, 869 / 97.
bool latent_attn_takes_tc(const LatentAttnArgs& a, int T) {
    static const bool no_mma = getenv("B2_NO_ATTN_MMA") != nullptr;        // tuning aid: scalar attention for prompts too
    const int parts = (a.rank + a.dr + LC_PART - 1) / LC_PART;
    return !no_mma && !a.cache_f32 && T > 8 && a.rank % LC_PART == 0 && (a.rank <= LC_V || a.rank % LC_V == 0) && parts <= 9 && a.ld_row % 8 == 0 &&
           a.block_tokens % LC_K == 0;
}

cudaError_t latent_attn_tc_launch(const LatentAttnArgs& a, const RaggedDev& r, const __nv_bfloat16* q, long pool_rows, __nv_bfloat16* out, cudaStream_t s) {
    if (!allow_smem<latent_attn_tc_kernel>(9 * (LC_QPART + LC_KPART) + 1024) || !latent_attn_takes_tc(a, r.T)) return cudaErrorInvalidValue;
    const int parts = (a.rank + a.dr + LC_PART - 1) / LC_PART, chunks = (a.rank + LC_V - 1) / LC_V;
    CUtensorMap mk, mq, mh;
    // rows of the pages [pages * block_tokens][ld_row]; columns past rank + dr arrive as zeros
    if (!bf16_rows_map(&mk, a.pool, a.rank + a.dr, pool_rows, a.ld_row, 1, 0, LC_K)) return cudaErrorInvalidValue;
    // queries [T][H][rank]: 128 tokens of one head, or the heads of one token
    if (!bf16_heads_map(&mq, q, a.rank, a.H, r.T, 1, LC_Q) || !bf16_heads_map(&mh, q, a.rank, a.H, r.T, LC_Q, 1)) return cudaErrorInvalidValue;
    const int n_packed = a.H <= LC_Q ? r.n_upto[0] : 0;
    return launch_chain(latent_attn_tc_kernel, dim3(((r.n_tiles - n_packed) * a.H + n_packed) * chunks), dim3(192), (size_t)parts * (LC_QPART + LC_KPART) + 1024, s,
                        mk, mq, mh, a, r, n_packed, chunks, out, kernel_error_word());
}

}  // namespace b2
