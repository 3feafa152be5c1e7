// Latent attention of steps of more than 8 tokens on the 5th-generation tensor cores (bf16 pages). Rounded where latent_attn_mma_kernel
// (latent_attn.cu) rounds: queries scaled, then rounded to bf16; cached rows as they are; probabilities rounded to bf16 for the weighted
// sum, 32-bit everywhere else. (Here the running maximum that a probability is taken against may lag by 2^8, so other bits are rounded.)
//
// A CTA takes 128 consecutive queries of one head and up to 256 latent columns of the output. A 512-wide latent is a PAIR of CTAs, a cluster: each
// forms the part of every score that its own 256 columns (and half of the rotated ones) give, so each reads and multiplies only those, and they
// exchange the parts through distributed shared memory; both then hold the same sums and the same probabilities. Blocks of 64 cached rows come by
// tensor copies as parts of 64 columns and serve both products: as rows of K for the scores, and, read across (N contiguous), as the values. Tensor
// memory (128 lanes x 512 columns) holds the output (256 columns), two score tiles of 64, two of probabilities (32, the second product's A operand) and
// half of the latent part of the queries (64; A operand of its part of the scores): shared memory then has room for a fourth block.
// Warps 0-7: softmax, two threads a query with 32 keys of a block each; 8-11 send this CTA's score parts to the other; 12: copies; 13: matrix instructions.
// As soon as a block's scores have been read, those of the block after next take their place, and their parts are on their way to the other CTA
// while the softmax of two blocks runs. The output is rescaled only when a row's maximum has grown by more than 2^8.
// Bound by shared memory, which holds every operand but the probabilities and a quarter of the queries and passes the score parts on (about 190 KB a block and CTA,
// 1500 of its 2900 cycles), and by what a CTA costs beside its blocks: 9000 cycles, four times in 2048 tokens.
// 2048 tokens, 16 heads (B200), us a layer: rows of 512 + 64 1640 with mma.sync, 207 with both CTAs computing all scores, 149 here; rows of 512, nothing
// rotated, 170 and 130. (Six warps and one thread a query: 180, 165. One barrier a block for all rows of the score parts: 163, 139. Four
// tiles of 32 scores with all of the queries in tensor memory: 182, 140: a product takes 50 to 70 cycles whether 32 or 64 keys wide.)
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
constexpr int LC_QPART = LC_Q * LC_PART * 2, LC_KPART = LC_K * LC_PART * 2, LC_XPART = LC_Q * LC_K * 4;
constexpr int LC_V = 256;                                   // latent columns of the output per CTA
constexpr int LC_NV = 4;                                    // stages of value parts at most
constexpr int LC_THREADS = 448, LC_SMEM = 225 * 1024;

namespace {
__device__ __forceinline__ uint32_t lc_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
}  // namespace

// where piece c of 16 bytes of a row lies in a plane of rows of `pieces` (a multiple of 8), so that neighbouring rows' meet other banks
__device__ __forceinline__ int lc_piece(int row, int c, int pieces) { return (row * pieces + (c ^ (row & 7))) * 16; }

// Stages of the value parts and of the other parts, as many as shared memory holds beside the queries
struct LcPlan { int n_val_stages, n_rest_stages, n_packed, n_even; };

// CTAs: (128-query tile, head, column chunk), the last tiles of longer sequences first, then the short sequences', then (one-token
// sequence, chunk) for the first n_packed tiles: there the rows are the heads, which all read the same keys
template <bool PAIR>
__global__ void __launch_bounds__(LC_THREADS, 1) latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q,
                                                                       const __grid_constant__ CUtensorMap map_h, const LatentAttnArgs a, const RaggedDev r,
                                                                       const LcPlan plan, __nv_bfloat16* out, unsigned int* err) {
    extern __shared__ uint8_t lc_smem[];
    __shared__ uint64_t rest_full[2], val_full[LC_NV], rest_empty[2], val_empty[LC_NV], q_come, q_full, s_full[2], s_read[2], p_full[2], pv_done[2], o_full;
    __shared__ uint64_t x_full[2][4], x_taken[2][4], x_empty[2][4];      // PAIR: [stage][32 rows]
    __shared__ uint32_t tmem_at;
    __shared__ float both[2][LC_Q];                        // what the two threads of a row tell each other (one buffer: shared memory is full)
    constexpr int CHUNKS = PAIR ? 2 : 1;
    const int n_short = r.n_upto[6] - plan.n_packed, at = blockIdx.x / CHUNKS, chunk = blockIdx.x % CHUNKS;      // (chunk: rank in the cluster)
    const bool packed = at >= (plan.n_even + n_short) * a.H;
    const int of_tile = packed ? at - (plan.n_even + n_short) * a.H : at / a.H;
    const int tile = packed ? of_tile : of_tile < plan.n_even ? r.n_tiles - 1 - of_tile : r.n_upto[6] - 1 - (of_tile - plan.n_even), h = packed ? 0 : at % a.H;
    const int seg = r.tile_seg[tile], row0 = r.tile_row0[tile];
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp: known to be uniform)
    const int nq = packed ? a.H : min(LC_Q, r.seg_start[seg] + r.seg_len[seg] - row0);      // rows in use
    const int p0 = r.seg_pos0[seg] + row0 - r.seg_start[seg], p_last = packed ? p0 : p0 + nq - 1;
    const int* table = a.block_tables[r.seg_slot[seg]];
    // this CTA's parts: n_val of the latent, which are values too, and n_rest rotated ones (of a pair's, each CTA takes two of the four steps of 16)
    const int n_val = PAIR ? LC_V / LC_PART : a.rank / LC_PART, v0 = chunk * n_val, n_rest = (a.dr + LC_PART - 1) / LC_PART, rest0 = a.rank / LC_PART;
    const int n_held = n_val / 2, n_qs = n_val - n_held;       // latent parts of the queries in tensor memory, in shared memory
    const int NV = plan.n_val_stages, NR = plan.n_rest_stages;
    uint8_t* qs = reinterpret_cast<uint8_t*>(((uintptr_t)lc_smem + 1023) & ~(uintptr_t)1023);      // [n_qs latent parts, n_rest rotated]
    uint8_t* vs = qs + (size_t)(n_qs + n_rest) * LC_QPART;                                         // [stage][n_val]
    uint8_t* rs = vs + (size_t)NV * n_val * LC_KPART;                                              // [stage][n_rest]
    float4* xs = reinterpret_cast<float4*>(rs + (size_t)NR * n_rest * LC_KPART);                   // PAIR: the other's score parts [2][16][128 rows] of 4
    const int b0 = max(0, p0 - a.window + 1) / LC_K, n_blocks = p_last / LC_K + 1 - b0;
    if (warp == 13) {
        if (lane < LC_NV) { mbar_init(&val_full[lane], 1); mbar_init(&val_empty[lane], 1); }
        else if (lane < LC_NV + 2) {
            const int i = lane - LC_NV;
            mbar_init(&rest_full[i], 1); mbar_init(&rest_empty[i], 1); mbar_init(&s_full[i], 1); mbar_init(&s_read[i], PAIR ? 384 : 256); mbar_init(&p_full[i], 256);
            mbar_init(&pv_done[i], 1);
        } else if (lane == LC_NV + 2) { mbar_init(&q_come, 1); mbar_init(&q_full, 256); mbar_init(&o_full, 1); }
        if (PAIR && lane < 8) { mbar_init(&x_full[0][0] + lane, 1); mbar_init(&x_taken[0][0] + lane, 2); mbar_init(&x_empty[0][0] + lane, 1); }
        fence_mbar_init();
        __syncwarp();
        tc_alloc(&tmem_at, 512);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if constexpr (PAIR) cluster_arrive();                  // (waited for ahead of the first access to the other CTA: its barriers exist)
    // The next kernel is let in once tensor memory is this CTA's: had it come first on this SM, it would hold its own and wait for this kernel
    // to end, and this CTA for that memory. (What is read above is the step's description, older than the kernel before this one.)
    griddep_launch();
    griddep_wait();
    const uint32_t tmem = tmem_at, o_at = tmem, s_at = tmem + LC_V, p_at = s_at + 2 * LC_K, q_at = p_at + LC_K;

    if (warp < 8) {
        // the rotated part of the queries (and zeros up to the part's 64 columns), rows past the tile as zeros: a warp's 16 rows, half a warp a row
        // of 32 entries, eight rows read ahead of their stores and without a branch between the reads (a thread per row, branches around every
        // entry: 28 us a CTA)
        // (queries without a latent of their own have been rotated where the rest of them lies)
        const int half = a.q_raw ? a.rot.rot_dims / 2 : 0, ld_q = a.q_raw ? a.d + a.dr : a.rank + a.dr;
        const float* queries = a.q_raw ? a.q_raw + a.d : a.qv + a.rank;
        for (int e0 = PAIR ? 32 * chunk : 0; e0 < n_rest * LC_PART; e0 += PAIR ? LC_PART : 32) {
            const int e = e0 + 2 * (lane & 15), q0 = warp * 16 + (lane >> 4) * 8;
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
            float v[8][2], w[8][2], cs[8][2], sn[8][2];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int q = min(q0 + u, nq - 1), qt = packed ? row0 : row0 + q, qh = packed ? q : h, qp = packed ? p0 : p0 + q;
                const float* from = queries + ((size_t)qt * a.H + qh) * ld_q;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const size_t turn_at = turn[k] < 0 ? 0 : (size_t)qp * half + turn[k];
                    v[u][k] = from[own[k]]; w[u][k] = from[other[k]];
                    cs[u][k] = half > 0 ? a.rot.cos[turn_at] : 1.f; sn[u][k] = half > 0 ? a.rot.sin[turn_at] : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                float y[2];
#pragma unroll
                for (int k = 0; k < 2; k++) y[k] = q0 + u < nq && e + k < a.dr ? (turn[k] < 0 ? v[u][k] : v[u][k] * cs[u][k] + sign[k] * w[u][k] * sn[u][k]) * a.scale : 0.f;
                *reinterpret_cast<uint32_t*>(qs + (size_t)(n_qs + e / LC_PART) * LC_QPART + (q0 + u) * 128 + (((e % LC_PART / 8) ^ (u & 7)) << 4) + e % 8 * 2) =
                    lc_pack(y[0], y[1]);
            }
        }
        // the latent parts that are held in tensor memory have come into the first stage of values: a row's two threads take half of it each
        mbar_wait(&q_come, 0, err, 0x60001u);
        {
            const int row = threadIdx.x & 127, side = threadIdx.x >> 7, cols = n_held * LC_PART / 4;      // columns of two entries
            for (int c = 0; c < cols; c += 16) {
                uint32_t v[16];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int piece = (side * cols + c) / 4 + k;
                    const uint4 x = *reinterpret_cast<const uint4*>(vs + (size_t)(piece / 8) * LC_QPART + row * 128 + (((piece & 7) ^ (row & 7)) << 4));
                    v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
                }
                __syncwarp();
                tc_st16(q_at + side * cols + c + ((uint32_t)((warp & 3) * 32) << 16), v);
            }
        }
        fence_proxy_async();
        tc_wait_st();
        tc_before_sync();
        mbar_arrive(&q_full);
    }
    if (warp == 12) {
        // ================= copies: the latent parts of the queries, then blocks of cached rows (all lanes run the loop, one issues: see dense_tc.cu)
        if constexpr (PAIR) cluster_wait();
        const bool one = elect_one();
        if (one) {
            mbar_arrive_expect_tx(&q_come, (uint32_t)(n_val * LC_QPART));
            for (int c = 0; c < n_val; c++)                    // (the held ones through the first stage of values)
                tma_load_3d(c < n_held ? vs + (size_t)c * LC_QPART : qs + (size_t)(c - n_held) * LC_QPART, packed ? &map_h : &map_q, (v0 + c) * LC_PART, h, row0, &q_come);
        }
        int sv = 1, sr = 0;                                    // block i in stage (i + 1) % NV
        uint32_t ur = 0;
        for (int i = 0; i < n_blocks; i++) {
            const int j0 = (b0 + i) * LC_K, row = table[j0 / a.block_tokens] * a.block_tokens + j0 % a.block_tokens;
            if (n_rest > 0) {
                if (ur > 0) mbar_wait_warp(&rest_empty[sr], (ur - 1) & 1, err, 0x60011u, (unsigned)i);
                if (one) {
                    mbar_arrive_expect_tx(&rest_full[sr], (uint32_t)(n_rest * LC_KPART));
                    for (int c = 0; c < n_rest; c++) tma_load_3d(rs + (size_t)(sr * n_rest + c) * LC_KPART, &map_k, (rest0 + c) * LC_PART, row, 0, &rest_full[sr]);
                }
                if (++sr == NR) { sr = 0; ur++; }
            }
            if (i >= NV) mbar_wait_warp(&val_empty[sv], (i / NV - 1) & 1, err, 0x60002u, (unsigned)i);
            else if (sv == 0) mbar_wait_warp(&q_full, 0, err, 0x6000eu, (unsigned)i);
            if (one) {
                mbar_arrive_expect_tx(&val_full[sv], (uint32_t)(n_val * LC_KPART));
                for (int c = 0; c < n_val; c++) tma_load_3d(vs + (size_t)(sv * n_val + c) * LC_KPART, &map_k, (v0 + c) * LC_PART, row, 0, &val_full[sv]);
            }
            if (++sv == NV) sv = 0;
        }
    } else if (warp == 13) {
        if constexpr (PAIR) cluster_wait();
        const bool one = elect_one();
        // ================= matrix instructions
        const uint32_t id_s = tc_idesc_bf16(LC_Q, LC_K), id_o = tc_idesc_bf16(LC_Q, n_val * LC_PART, true);
        const uint32_t qa = smem_u32(qs), va = smem_u32(vs), ra = smem_u32(rs);
        const uint64_t dq0 = tc_desc(qa);
        int sv = 1, sr = 0, sp = 1;                            // stages of the next scores, and of the next sum's values
        uint32_t uv = 0, ur = 0;
        auto scores = [&](int i) {
            const uint32_t to = s_at + (i & 1) * LC_K;
            if (i > 1) mbar_wait_warp(&s_read[i & 1], ((i >> 1) - 1) & 1, err, 0x60003u, (unsigned)i);
            if (n_rest > 0) {
                mbar_wait_warp(&rest_full[sr], ur & 1, err, 0x60004u, (unsigned)i);
                tc_after_sync();
                if (one) for (int c = 0; c < n_rest; c++) {
                    const uint64_t dq = tc_desc(qa + (n_qs + c) * LC_QPART), dk = tc_desc(ra + (sr * n_rest + c) * LC_KPART);
#pragma unroll
                    for (int k = 0; k < LC_PART / 16; k++)
                        if (!PAIR || k / 2 == chunk) tc_mma(to, dq + 2 * k, dk + 2 * k, id_s, c == 0 && k == (PAIR ? 2 * chunk : 0) ? 0u : 1u);
                }
                if (one) tc_commit(&rest_empty[sr]);
                if (++sr == NR) { sr = 0; ur++; }
            }
            mbar_wait_warp(&val_full[sv], uv & 1, err, 0x60005u, (unsigned)i);
            tc_after_sync();
            if (one) {
                const uint64_t dk0 = tc_desc(va + sv * n_val * LC_KPART);
#pragma unroll
                for (int c = 0; c < LC_V / LC_PART; c++) {
                    if (!PAIR && c >= n_val) break;
#pragma unroll
                    for (int k = 0; k < LC_PART / 16; k++) {
                        const uint64_t dk = dk0 + c * (LC_KPART >> 4) + 2 * k;
                        if (c < (PAIR ? LC_V / LC_PART / 2 : n_held)) tc_mma_ts(to, q_at + (c * (LC_PART / 16) + k) * 8, dk, id_s, (n_rest | c | k) ? 1u : 0u);
                        else tc_mma(to, dq0 + (c - n_held) * (LC_QPART >> 4) + 2 * k, dk, id_s, (n_rest | c | k) ? 1u : 0u);
                    }
                }
                tc_commit(&s_full[i & 1]);
            }
            if (++sv == NV) sv = 0;
            if (sv == 1) uv++;
        };
        mbar_wait_warp(&q_come, 0, err, 0x60012u);
        mbar_wait_warp(&q_full, 0, err, 0x60006u);
        tc_after_sync();
        scores(0);
        if (n_blocks > 1) scores(1);
        for (int i = 0; i < n_blocks; i++) {
            if (NV > 2 && i + 2 < n_blocks) scores(i + 2);     // (of two stages, its block's is the one that waits for this block's sum)
            mbar_wait_warp(&p_full[i & 1], (i >> 1) & 1, err, 0x60007u, (unsigned)i);
            tc_after_sync();
            if (one) {
                const uint64_t dv = tc_desc(va + sp * n_val * LC_KPART, LC_KPART);
#pragma unroll
                for (int k = 0; k < LC_K / 16; k++) tc_mma_ts(o_at, p_at + (i & 1) * (LC_K / 2) + k * 8, dv + k * (2048 >> 4), id_o, (i | k) ? 1u : 0u);
                tc_commit(&pv_done[i & 1]);
                tc_commit(&val_empty[sp]);
                if (i == n_blocks - 1) tc_commit(&o_full);
            }
            if (++sp == NV) sp = 0;
            if (NV <= 2 && i + 2 < n_blocks) scores(i + 2);
        }
    } else if (warp >= 8) {
        // ================= this CTA's parts of the scores, to the other's shared memory
        if constexpr (PAIR) {
            // (a warp sends 32 rows, which two softmax warps read there; the barriers of other rows are not its own)
            const int row = threadIdx.x & 127, rows = warp & 3;
            const uint32_t lanes = (uint32_t)(rows * 32) << 16;
            const uint32_t to = cluster_address(smem_u32(xs) + row * 16, chunk ^ 1), bar = cluster_address(smem_u32(x_full) + rows * 8, chunk ^ 1);
            const uint32_t x_free = cluster_address(smem_u32(x_empty) + rows * 8, chunk ^ 1);
            cluster_wait();
            for (int i = 0; i < n_blocks; i++) {
                const int st = i & 1;
                mbar_wait(&s_full[st], (i >> 1) & 1, err, 0x60008u, (unsigned)i);
                tc_after_sync();
                uint32_t raw[2][32];
                __syncwarp();
                tc_ld32(s_at + st * LC_K + lanes, raw[0]);
                tc_ld32(s_at + st * LC_K + 32 + lanes, raw[1]);
                tc_wait_ld();
                tc_before_sync();
                mbar_arrive(&s_read[st]);
                if (i > 1) {
                    // each may send this block's parts once the softmax warps over there have read those of the block before last. (The arrival orders for
                    // the cluster and waits for what its warp has under way: by a softmax warp it took 1500 cycles; ahead of the scores 160 and 129 us)
                    const uint32_t phase = ((i >> 1) - 1) & 1;
                    mbar_wait_warp(&x_taken[st][rows], phase, err, 0x60010u, (unsigned)i);
                    if (lane == 0) mbar_arrive_cluster(x_free + st * 32);
                    mbar_wait_cluster(&x_empty[st][rows], phase, err, 0x60009u, (unsigned)i);
                }
#pragma unroll
                for (int j = 0; j < 16; j++) st_async_16(to + st * LC_XPART + j * (LC_Q * 16), &raw[j >> 3][(j & 7) * 4], bar + st * 32);
            }
        }
    } else {
        // ================= softmax: threads t and t + 128 share query row t, keys 0-31 and 32-63 of a block
        constexpr int HALF = LC_K / 2;
        const int row = threadIdx.x & 127, side = threadIdx.x >> 7, pos = packed ? p0 : p0 + row;
        const int t = packed ? row0 : row0 + row, hd = packed ? min(row, a.H - 1) : h;      // the row's token and head
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const int my_cols = n_val * LC_PART / 2, col0 = side * my_cols;                    // of the output
        if constexpr (PAIR) {
            if (warp < 4 && lane == 0) for (int i = 0; i < 2; i++) mbar_arrive_expect_tx(&x_full[i][warp], LC_XPART / 4);
            cluster_wait();
        }
        constexpr float LOG2E = 1.4426950408889634f;
        float m_ref = a.sink ? a.sink[hd] * LOG2E : -INFINITY, l = a.sink && side == 0 ? 1.f : 0.f;      // log2 domain: weights are 2^(score - m_ref)
        for (int i = 0; i < n_blocks; i++) {
            const int st = i & 1, j0 = (b0 + i) * LC_K, c0 = j0 + side * HALF;             // this thread's first key
            const uint32_t phase = (i >> 1) & 1;
            mbar_wait(&s_full[st], phase, err, 0x6000au, (unsigned)i);
            tc_after_sync();
            uint32_t raw[HALF];
            __syncwarp();
            tc_ld32(s_at + st * LC_K + side * HALF + lanes, raw);
            tc_wait_ld();
            tc_before_sync();
            mbar_arrive(&s_read[st]);
            float s[HALF];
#pragma unroll
            for (int j = 0; j < HALF; j++) s[j] = __uint_as_float(raw[j]);
            if constexpr (PAIR) {                              // a sum of two: the same in both CTAs
                mbar_wait_cluster(&x_full[st][warp & 3], phase, err, 0x6000bu, (unsigned)i);
                __syncwarp();
#pragma unroll
                for (int j = 0; j < HALF / 4; j++) {
                    const float4 x = xs[(st * (LC_K / 4) + side * (HALF / 4) + j) * LC_Q + row];
                    s[4 * j] += x.x; s[4 * j + 1] += x.y; s[4 * j + 2] += x.z; s[4 * j + 3] += x.w;
                }
                __syncwarp();
                if (i + 2 < n_blocks && lane == 0) {           // this warp has read its share
                    if (warp < 4) mbar_arrive_expect_tx(&x_full[st][warp], LC_XPART / 4);
                    mbar_arrive(&x_taken[st][warp & 3]);
                }
            }
#pragma unroll
            for (int j = 0; j < HALF; j++) s[j] *= LOG2E;
            if (j0 + LC_K - 1 > p0 || p_last - j0 >= a.window) {
                const int lo = pos - a.window + 1 - c0, hi = pos - c0;          // visible columns of this row
#pragma unroll
                for (int j = 0; j < HALF; j++) if (j < lo || j > hi) s[j] = -INFINITY;
            }
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < HALF; j++) mx = fmaxf(mx, s[j]);
            named_bar_sync(1 + (warp & 3), 64);                   // (the two warps of these rows) the last block's maxima have been read
            both[side][row] = mx;
            named_bar_sync(1 + (warp & 3), 64);
            mx = fmaxf(mx, both[side ^ 1][row]);
            const bool grow = mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY);
            const float m_old = m_ref;
            if (grow) { m_ref = mx; l *= exp2f(m_old - mx); }
            const float ref = m_ref > -INFINITY ? m_ref : 0.f;                  // a row that has seen no key yet: all weights are 0
            uint32_t p[HALF / 2];
#pragma unroll
            for (int j = 0; j < HALF; j += 2) {
                const float e0 = exp2f(s[j] - ref), e1 = exp2f(s[j + 1] - ref);
                l += e0 + e1;
                p[j >> 1] = lc_pack(e0, e1);
            }
            // the sum before last must be in before its probabilities are overwritten, the last one before the output is rescaled
            if (i > 1) { mbar_wait(&pv_done[st], phase ^ 1, err, 0x6000cu, (unsigned)i); tc_after_sync(); }
            if (i > 0 && __any_sync(0xffffffffu, grow)) {
                mbar_wait(&pv_done[st ^ 1], ((i - 1) >> 1) & 1, err, 0x6000du, (unsigned)i);
                tc_after_sync();
                const float f = grow ? exp2f(m_old - m_ref) : 1.f;
                __syncwarp();
                for (int c = col0; c < col0 + my_cols; c += 32) {
                    uint32_t o[32];
                    tc_ld32(o_at + c + lanes, o);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                    tc_st32(o_at + c + lanes, o);
                }
            }
            __syncwarp();
            tc_st16(p_at + st * (LC_K / 2) + side * (HALF / 2) + lanes, p);
            tc_wait_st();
            if (i == n_blocks - 1 && p_last - j0 + 1 < LC_K) {
                // rows of the last block past the sequence: whatever the page holds must not meet the zero weights as values (the scores, which read
                // those rows too, are in)
                const int r0 = p_last - j0 + 1, n_bad = LC_K - r0, sv = (i + 1) % NV;
                for (int e = threadIdx.x; e < n_val * n_bad * 8; e += 256) {
                    const int c = e / (n_bad * 8), rr = r0 + e / 8 % n_bad;
                    *reinterpret_cast<uint4*>(vs + (size_t)(sv * n_val + c) * LC_KPART + rr * 128 + (e & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
            }
            tc_before_sync();
            mbar_arrive(&p_full[st]);
        }
        named_bar_sync(1 + (warp & 3), 64);
        both[side][row] = l;
        named_bar_sync(1 + (warp & 3), 64);
        l = both[0][row] + both[1][row];
        mbar_wait(&o_full, 0, err, 0x6000fu);
        tc_after_sync();
        // rounded, and through the stages of values (nothing reads them any more), so that neighbouring lanes write a row (a thread per row: 4700 cycles)
        const float inv = 1.f / l;
        const int pieces = n_val * LC_PART / 8;
        for (int c = col0; c < col0 + my_cols; c += 32) {
            uint32_t o[32];
            __syncwarp();
            tc_ld32(o_at + c + lanes, o);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
                uint32_t u[4];
#pragma unroll
                for (int q = 0; q < 4; q++) u[q] = lc_pack(__uint_as_float(o[e + 2 * q]) * inv, __uint_as_float(o[e + 2 * q + 1]) * inv);
                *reinterpret_cast<uint4*>(vs + lc_piece(row, (c + e) / 8, pieces)) = make_uint4(u[0], u[1], u[2], u[3]);
            }
        }
        named_bar_sync(5, 256);
#pragma unroll 4
        for (int e = lane; e < 16 * pieces; e += 32) {
            const int q = warp * 16 + e / pieces;
            if (q < nq) *reinterpret_cast<uint4*>(out + ((size_t)(packed ? row0 : row0 + q) * a.H + (packed ? q : h)) * a.rank + chunk * LC_V + e % pieces * 8) =
                *reinterpret_cast<const uint4*>(vs + lc_piece(q, e % pieces, pieces));
        }
        tc_before_sync();
    }
    __syncthreads();
    if (warp == 13) tc_dealloc(tmem, 512);
    if constexpr (PAIR) { cluster_arrive(); cluster_wait(); }      // nobody leaves while the other may still write or arrive here
}

// ---------------------------------------------------------------- host side
// Rows of 64-column parts that fit shared memory beside the queries (9 of them), whole chunks of output columns, pages of whole blocks; of
// the step only what the few-token kernels do not take (see softmax_tc.cu). 16 heads, rows of 512 + 64, us a layer with the preparation,
// mma.sync / here: a prompt of 9 tokens 52 / 25, of 64 93 / 25, of 255 120 / 32; 32 prompts of 60 568 / 93; one token of each of 32 sequences
// behind 60 208 / 26, behind 1900 2087 / 91; 512 tokens beside 31 sequences that decode behind 500, 869 / 56.
bool latent_attn_takes_tc(const LatentAttnArgs& a, int T) {
    static const bool no_mma = getenv("B2_NO_ATTN_MMA") != nullptr;        // tuning aid: scalar attention for prompts too
    const int parts = (a.rank + a.dr + LC_PART - 1) / LC_PART;
    return !no_mma && !a.cache_f32 && T > 8 && a.rank % LC_PART == 0 && (a.rank <= LC_V || a.rank % LC_V == 0) && parts <= 9 && a.ld_row % 8 == 0 &&
           a.block_tokens % LC_K == 0;
}

cudaError_t latent_attn_tc_launch(const LatentAttnArgs& a, const RaggedDev& r, const __nv_bfloat16* q, long pool_rows, __nv_bfloat16* out, cudaStream_t s) {
    if (!allow_smem<latent_attn_tc_kernel<false>>(LC_SMEM) || !allow_smem<latent_attn_tc_kernel<true>>(LC_SMEM) || !latent_attn_takes_tc(a, r.T)) return cudaErrorInvalidValue;
    CUtensorMap mk, mq, mh;
    // rows of the pages [pages * block_tokens][ld_row]; columns past rank + dr arrive as zeros
    if (!bf16_rows_map(&mk, a.pool, a.rank + a.dr, pool_rows, a.ld_row, 1, 0, LC_K)) return cudaErrorInvalidValue;
    // queries [T][H][rank]: 128 tokens of one head, or the heads of one token
    if (!bf16_heads_map(&mq, q, a.rank, a.H, r.T, 1, LC_Q) || !bf16_heads_map(&mh, q, a.rank, a.H, r.T, LC_Q, 1)) return cudaErrorInvalidValue;
    const bool pair = a.rank > LC_V;
    const int n_val = (pair ? LC_V : a.rank) / LC_PART, n_rest = (a.dr + LC_PART - 1) / LC_PART, chunks = pair ? 2 : 1;
    LcPlan plan = {};
    plan.n_packed = a.H <= LC_Q ? r.n_upto[0] : 0;
    plan.n_even = r.n_tiles - r.n_upto[6] - r.n_odd;
    auto bytes = [&] { return (n_val - n_val / 2 + n_rest) * LC_QPART + (plan.n_val_stages * n_val + plan.n_rest_stages * n_rest) * LC_KPART + (pair ? 2 * LC_XPART : 0) + 1024; };
    plan.n_val_stages = LC_NV; plan.n_rest_stages = 2;
    while (bytes() > LC_SMEM && plan.n_val_stages > 2) plan.n_val_stages--;
    if (bytes() > LC_SMEM) plan.n_rest_stages = 1;         // (the sizes that latent_attn_takes_tc lets in fit with two and one)
    const int grid = ((plan.n_even + r.n_upto[6] - plan.n_packed) * a.H + plan.n_packed) * chunks, smem = bytes();
    if (grid == 0) return cudaSuccess;
    if (smem > LC_SMEM) return cudaErrorInvalidValue;
    if (!pair) return launch_chain(latent_attn_tc_kernel<false>, dim3(grid), dim3(LC_THREADS), smem, s, mk, mq, mh, a, r, plan, out, kernel_error_word());
    return launch_chain_cluster(latent_attn_tc_kernel<true>, chunks, dim3(grid), dim3(LC_THREADS), smem, s, mk, mq, mh, a, r, plan, out, kernel_error_word());
}

}  // namespace b2
