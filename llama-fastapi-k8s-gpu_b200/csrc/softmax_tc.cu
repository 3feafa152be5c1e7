// Softmax attention of steps of more than 8 tokens on the 5th-generation tensor cores, for the layer-list models (bf16 pages, key and value
// sizes up to 128). Queries and probabilities enter the products as TWO bf16 each (leading part + remainder), so the only 16-bit rounding is
// that of the cached keys and values; everything else is 32-bit, with ex2.approx for the exponentials. (The mma.sync kernels, which other
// sizes take, split at the same places. They round a probability against the exact running maximum, here it may lag by 2^8, and window
// attention there uses expf on unscaled queries: the two agree to about 1e-5 ahead of the rounding of the output.)
//
// A CTA takes 128 consecutive queries of one head (or, of a short sequence, the queries of several heads that share their keys); blocks of 128 keys and values come by tensor copies (two pages rows of 64 each, parts
// of 64 columns in 128-byte-swizzled rows, two stages). Tensor memory holds the output (128 columns), two score tiles (2 x 128) and the two
// halves of the probabilities (64 + 64), which are the A operand of the second product. The next block's scores are computed while
// this one's softmax runs. Eight softmax warps, two threads a query row with 64 key columns each (capped scores take three special-function
// operations a score; that unit is busy for 35 % of 2048 tokens' time, the tensor pipe for 25 %: what bounds the kernel is the chain of a block, and
// 256 CTAs of unequal length on 148 SMs); they exchange their maxima through shared memory. The output is rescaled only
// when a row's maximum has grown by more than 2^8.
// 2048 tokens (B200): 16 capped heads of 128, 300 us a layer with mma.sync, 65 here; 32 heads of 128 over a window of 1024 keys, 326 and 92.
// (70 and 100 with the wait for the previous block's products ahead of the exponentials and all eight warps at one barrier for the maxima.
// Blocks of 64 keys with one thread a row, of which two CTAs fit on an SM: 80 and 80; there the first product reads its queries from shared
// memory twice as often, and 256 CTAs of unequal length leave an SM two long ones.)
#include "kernels.h"
#include "layered.h"
#include "ptx.cuh"
#include "softmax_tc.h"
#include "tc05.cuh"
#include "tensor_map.h"

#include <algorithm>

namespace b2 {

constexpr int SX_Q = 128, SX_K = 128, SX_PART = SX_Q * 128;       // queries, keys of a block; bytes of a part (128 rows x 64 columns)
constexpr int SX_THREADS = 320;                                   // warps 0-7 softmax, 8 copies, 9 matrix instructions

namespace {
__device__ __forceinline__ float sx_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float sx_rcp(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ void sx_split(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a - __low2float(h), b - __high2float(h));
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
}  // namespace

// A sequence of up to 2^k <= 64 tokens shares a CTA between heads[k] query heads of a key/value head, rows token by token; its tiles start at
// tile0[k], its CTAs at cta0[k]
struct SxShort { int tile0[7], cta0[7], heads[7]; };

// CTAs: (even tile, head) of longer sequences, the last tiles first, then (sequence,
// group of heads) of the others, the longest first. SHORT: there are such (2048 tokens of one sequence take 85 us a layer without that part
// and 89 with it, preparation included)
template <bool CAP, bool SHORT>
__global__ void __launch_bounds__(SX_THREADS, 1) softmax_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                                                                   const SoftmaxTcArgs a, const RaggedDev r, const __grid_constant__ SxShort sh, unsigned int* err) {
    extern __shared__ uint8_t sx_smem[];
    __shared__ uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], q_full, s_full[2], p_full, pv_done;
    __shared__ uint32_t tmem_at;
    __shared__ float row_max[2][2][SX_Q], row_sum[2][SX_Q];
    int tile = r.n_tiles - 1 - (int)blockIdx.x / a.H, h = (int)blockIdx.x % a.H, per_tok = 1;      // per_tok: rows of a token, heads h ..
    if (const int in_short = (int)blockIdx.x - (r.n_tiles - r.n_upto[6] - r.n_odd) * a.H; SHORT && in_short >= 0) {
        int k = 6;
        while (k > 0 && in_short >= sh.cta0[k - 1]) k--;
        per_tok = sh.heads[k];
        tile = sh.tile0[k] + (in_short - sh.cta0[k]) / (a.H / per_tok);
        h = (in_short - sh.cta0[k]) % (a.H / per_tok) * per_tok;
    }
    const int seg = r.tile_seg[tile], row0 = r.tile_row0[tile];
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp: known to be uniform)
    const int n_tok = min(SX_Q, r.seg_start[seg] + r.seg_len[seg] - row0);
    const int nq = n_tok * per_tok, n_thr = SHORT ? (nq + 31) / 32 * 64 : 2 * SX_Q;      // rows in use; softmax threads: two a row, whole warps
    const int p0 = r.seg_pos0[seg] + row0 - r.seg_start[seg], p_last = p0 + n_tok - 1;
    const int* table = a.block_tables[r.seg_slot[seg]];
    const int g = h / (a.H / a.G), bt = a.block_tokens;
    const int k_parts = (a.d + 63) / 64, v_parts = (a.dv + 63) / 64;
    uint8_t* qs = reinterpret_cast<uint8_t*>(((uintptr_t)sx_smem + 1023) & ~(uintptr_t)1023);      // [leading, remainder][part]
    uint8_t* ks = qs + 2 * k_parts * SX_PART;                                                      // [stage][part]
    uint8_t* vs = ks + 2 * k_parts * SX_PART;
    // key blocks: those of the kept prefix, then those of the window
    const int lo_first = a.window > 0 ? max(0, p0 - a.window + 1) : 0;
    const int n_kept = lo_first > 0 ? (min(a.keep_first, lo_first) + SX_K - 1) / SX_K : 0;
    const int w0 = max(lo_first / SX_K, n_kept), n_blocks = n_kept + p_last / SX_K + 1 - w0;
    auto block_at = [&](int i) { return (i < n_kept ? i : w0 + i - n_kept) * SX_K; };
    if (warp == 9) {
        if (lane == 0) {
            for (int i = 0; i < 2; i++) {
                mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); mbar_init(&s_full[i], 1);
            }
            mbar_init(&q_full, n_thr); mbar_init(&p_full, n_thr); mbar_init(&pv_done, 1);
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
    const uint32_t o_at = tmem_at, s_at = tmem_at + 128, p_at = tmem_at + 384;       // probabilities: 64 columns leading, 64 remainder

    if (warp == 8) {
        // ================= copies (all lanes run the loop, one issues: see dense_tc.cu)
        const bool one = elect_one();
        for (int i = 0; i < n_blocks; i++) {
            const int st = i & 1, j0 = block_at(i), halves = j0 + 64 <= p_last ? 2 : 1;
            for (int kv = 0; kv < 2; kv++) {
                uint64_t *full = kv ? &v_full[st] : &k_full[st], *empty = kv ? &v_empty[st] : &k_empty[st];
                const int parts = kv ? v_parts : k_parts;
                uint8_t* dst = (kv ? vs : ks) + (size_t)st * parts * SX_PART;
                if (i >= 2) mbar_wait_warp(empty, ((i >> 1) - 1) & 1, err, 0x70001u, (unsigned)i);
                if (!one) continue;
                mbar_arrive_expect_tx(full, (uint32_t)(halves * parts * (SX_PART / 2)));
                for (int hf = 0; hf < halves; hf++) {
                    const int j = j0 + 64 * hf, row = (table[j / bt] * a.G + g) * bt + j % bt;
                    for (int c = 0; c < parts; c++) tma_load_3d(dst + (size_t)c * SX_PART + hf * (SX_PART / 2), kv ? &map_v : &map_k, c * 64, row, 0, full);
                }
            }
        }
    } else if (warp == 9) {
        const bool one = elect_one();
        // ================= matrix instructions
        const uint32_t id_s = tc_idesc_bf16(SX_Q, SX_K), id_o = tc_idesc_bf16(SX_Q, a.dv, true);
        const uint32_t qa = smem_u32(qs), ka = smem_u32(ks), va = smem_u32(vs);
        auto scores = [&](int i) {
            mbar_wait_warp(&k_full[i & 1], (i >> 1) & 1, err, 0x70002u, (unsigned)i);
            tc_after_sync();
            if (one) for (int part = 0; part < 2 * k_parts; part++) {    // remainders first
                const int c = part % k_parts, lead = part / k_parts;
                const uint64_t dq = tc_desc(qa + ((lead ? 0 : k_parts) + c) * SX_PART), dk = tc_desc(ka + ((i & 1) * k_parts + c) * SX_PART);
#pragma unroll
                for (int k = 0; k < 4; k++) tc_mma(s_at + (i & 1) * SX_K, dq + 2 * k, dk + 2 * k, id_s, (part | k) ? 1u : 0u);
            }
            if (one) { tc_commit(&s_full[i & 1]); tc_commit(&k_empty[i & 1]); }
        };
        mbar_wait_warp(&q_full, 0, err, 0x70003u);
        tc_after_sync();
        scores(0);
        for (int i = 0; i < n_blocks; i++) {
            if (i + 1 < n_blocks) scores(i + 1);
            mbar_wait_warp(&v_full[i & 1], (i >> 1) & 1, err, 0x70004u, (unsigned)i);
            mbar_wait_warp(&p_full, i & 1, err, 0x70005u, (unsigned)i);
            tc_after_sync();
            const uint32_t v_at = va + (i & 1) * v_parts * SX_PART;
            if (!one) continue;
#pragma unroll
            for (int half = 0; half < 2; half++)                         // remainders first
#pragma unroll
                for (int k = 0; k < SX_K / 16; k++)
                    tc_mma_ts(o_at, p_at + (half ? 0 : 64) + k * 8, tc_desc(v_at + k * 2048, SX_PART), id_o, (i | half | k) ? 1u : 0u);
            tc_commit(&pv_done);
            tc_commit(&v_empty[i & 1]);
        }
    } else if (warp < 8 && (warp & 3) * 64 < n_thr) {
        // ================= softmax: threads t and t + 128 share query row t, key columns 0-63 and 64-127 of a block
        const int row = threadIdx.x & 127, side = threadIdx.x >> 7, tok = SHORT ? row / per_tok : row, pos = p0 + tok;
        const int t = row0 + tok, hd = SHORT ? h + row % per_tok : h;      // the row's token and query head
        const int thr = side * (n_thr / 2) + row;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        constexpr float LOG2E = 1.4426950408889634f;
        // scores live in the log2 domain. Capped: cap tanh(s / cap) = cap - 2 cap / (exp(2 s / cap) + 1), the exponential's factor folded
        // into the query as well
        const float q_mul = CAP ? a.scale * (2.f * LOG2E) / a.softcap : a.scale * LOG2E;
        [[maybe_unused]] const float cap2 = CAP ? a.softcap * LOG2E : 0.f;
        {   // queries, 8 columns at a time: neighbouring threads take neighbouring pieces of a row
            const int per = k_parts * 8, d8 = a.d / 8;
            for (int e = thr; e < n_thr / 2 * per; e += n_thr) {
                const int rr = e / per, c8 = e % per;
                float v[8] = {};
                if (rr < nq && c8 < d8) {
                    const float4* src = reinterpret_cast<const float4*>(a.q + (SHORT ? (size_t)(row0 + rr / per_tok) * a.H + h + rr % per_tok : (size_t)(row0 + rr) * a.H + h) * a.d + c8 * 8);
                    const float4 x = src[0], y = src[1];
                    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
                }
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int k = 0; k < 4; k++) sx_split(v[2 * k] * q_mul, v[2 * k + 1] * q_mul, hi[k], lo[k]);
                uint8_t* dst = qs + (size_t)(c8 >> 3) * SX_PART + rr * 128 + (((c8 & 7) ^ (rr & 7)) << 4);
                *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(dst + (size_t)k_parts * SX_PART) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            fence_proxy_async();
            mbar_arrive(&q_full);
        }
        const float sink = a.sink ? a.sink[hd] * LOG2E : -INFINITY;
        float m_ref = sink, l = 0.f;                              // weights are 2^(score - m_ref); the sink's term joins at the end
        const int lo_key = a.window > 0 ? max(0, pos - a.window + 1) : 0;
        for (int i = 0; i < n_blocks; i++) {
            const int j0 = block_at(i), c0 = j0 + side * 64;      // this thread's first key
            mbar_wait(&s_full[i & 1], (i >> 1) & 1, err, 0x70006u, (unsigned)i);
            tc_after_sync();
            float s[64];
            {
                uint32_t raw[2][32];
                __syncwarp();
                tc_ld32(s_at + (i & 1) * SX_K + side * 64 + lanes, raw[0]);
                tc_ld32(s_at + (i & 1) * SX_K + side * 64 + 32 + lanes, raw[1]);
                tc_wait_ld();
#pragma unroll
                for (int j = 0; j < 64; j++) s[j] = __uint_as_float(raw[j >> 5][j & 31]);
            }
            if constexpr (CAP)
#pragma unroll
                for (int j = 0; j < 64; j++) s[j] = fmaf(-2.f * cap2, sx_rcp(sx_exp2(s[j]) + 1.f), cap2);
            if (j0 + SX_K - 1 > p0 || (a.window > 0 && p_last - j0 >= a.window)) {
#pragma unroll
                for (int j = 0; j < 64; j++) if (c0 + j > pos || (c0 + j < lo_key && c0 + j >= a.keep_first)) s[j] = -INFINITY;
            }
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 64; j++) mx = fmaxf(mx, s[j]);
            row_max[i & 1][side][row] = mx;
            named_bar_sync(1 + (warp & 3), 64);                   // (the two warps of these rows)
            mx = fmaxf(mx, row_max[i & 1][side ^ 1][row]);
            const bool grow = mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY);
            float f = 1.f;
            if (grow) { f = sx_exp2(m_ref - mx); m_ref = mx; l *= f; }
            const float ref = m_ref > -INFINITY ? m_ref : 0.f;    // nothing visible yet and no sink: every weight is 0
            uint32_t hi[32], lo[32];
#pragma unroll
            for (int j = 0; j < 64; j += 2) {
                const float e0 = sx_exp2(s[j] - ref), e1 = sx_exp2(s[j + 1] - ref);
                l += e0 + e1;
                sx_split(e0, e1, hi[j >> 1], lo[j >> 1]);
            }
            // the previous block's products run until here; they must be in before the output is rescaled and the probabilities are rewritten
            if (i > 0) {
                mbar_wait(&pv_done, (i - 1) & 1, err, 0x70007u, (unsigned)i);
                tc_after_sync();
                if (__any_sync(0xffffffffu, grow))                // this side's 64 columns of the output
                    for (int c = side * 64; c < min(side * 64 + 64, a.dv); c += 16) {
                        float o[16];
                        tc_ld16(o_at + c + lanes, o);
#pragma unroll
                        for (int e = 0; e < 16; e++) o[e] *= f;
                        tc_st16(o_at + c + lanes, o);
                    }
            }
            __syncwarp();
            tc_st32(p_at + side * 32 + lanes, hi);
            tc_st32(p_at + 64 + side * 32 + lanes, lo);
            tc_wait_st();
            if (i == n_blocks - 1 && p_last - j0 + 1 < SX_K) {
                // rows past the sequence: whatever shared memory or the page holds must not meet the zero weights as values
                mbar_wait(&v_full[i & 1], (i >> 1) & 1, err, 0x70008u, (unsigned)i);
                const int r0 = p_last - j0 + 1, n_bad = SX_K - r0;
                for (int e = thr; e < v_parts * n_bad * 8; e += n_thr) {
                    const int c = e / (n_bad * 8), rr = r0 + e / 8 % n_bad;
                    *reinterpret_cast<uint4*>(vs + (size_t)((i & 1) * v_parts + c) * SX_PART + rr * 128 + (e & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
            }
            tc_before_sync();
            mbar_arrive(&p_full);
        }
        row_sum[side][row] = l;
        named_bar_sync(1 + (warp & 3), 64);
        l += row_sum[side ^ 1][row];
        if (a.sink) l += sx_exp2(sink - m_ref);
        const float inv = l > 0.f ? 1.f / l : 0.f;
        mbar_wait(&pv_done, (n_blocks - 1) & 1, err, 0x70009u);
        tc_after_sync();
        const int dv = a.dv;
        const size_t at = (size_t)t * a.ld_out + (size_t)hd * dv;
        const float* gate = a.gate && row < nq ? a.gate + (size_t)t * a.ld_gate + (a.gate_per_head ? hd : hd * dv) : nullptr;
        const float head_gate = gate && a.gate_per_head ? 1.f / (1.f + expf(-gate[0])) : 1.f;
        for (int c = side * 64; c < min(side * 64 + 64, dv); c += 32) {
            uint32_t o[32];
            __syncwarp();
            tc_ld32(o_at + c + lanes, o);
            tc_wait_ld();
            if (row >= nq) continue;
#pragma unroll
            for (int e = 0; e < 32; e += 8) {                     // dv is a multiple of 16
                if (c + e >= dv) break;
                float v[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    v[k] = __uint_as_float(o[e + k]) * inv;
                    if (gate && !a.gate_per_head) v[k] *= 1.f / (1.f + expf(-gate[c + e + k]));
                    else v[k] *= head_gate;
                }
                if (a.out_bf16) {
                    uint32_t u[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
                        u[k] = *reinterpret_cast<const uint32_t*>(&b);
                    }
                    *reinterpret_cast<uint4*>(a.out_bf16 + at + c + e) = make_uint4(u[0], u[1], u[2], u[3]);
                } else {
                    *reinterpret_cast<float4*>(a.out + at + c + e) = make_float4(v[0], v[1], v[2], v[3]);
                    *reinterpret_cast<float4*>(a.out + at + c + e + 4) = make_float4(v[4], v[5], v[6], v[7]);
                }
            }
        }
        tc_before_sync();
    }
    __syncthreads();
    if (warp == 9) tc_dealloc(tmem_at, 512);
}

// ---------------------------------------------------------------- host side
// Sizes that the tiles and 16-byte stores take, pages of whole 64-key halves; nothing of the step, so that a row goes to the same kernel
// whatever shares its step and wherever its prompt was cut. 16 heads of 128 over 4, us a layer with the preparation, mma.sync / here, capped |
// over a window of 1024: a prompt of 9 tokens 30 / 24 | 24 / 23, of 64 44 / 24 | 33 / 24, of 255 53 / 26 | 54 / 28; 32 prompts of 16 72 / 33 |
// 47 / 27, of 60 110 / 56 | 66 / 49; 512 tokens beside 31 sequences that decode behind 500, 168 / 75 | 148 / 46.
bool softmax_takes_tc(const SoftmaxTcArgs& a) {
    return a.d % 16 == 0 && a.dv % 16 == 0 && a.d <= 128 && a.dv <= 128 && a.block_tokens % 64 == 0 && a.ld_out % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.out_bf16)) & 15) == 0;
}

cudaError_t softmax_tc_launch(const SoftmaxTcArgs& a, const RaggedDev& r, cudaStream_t s) {
    const int k_parts = (a.d + 63) / 64, v_parts = (a.dv + 63) / 64;
    constexpr int most = 12 * SX_PART + 1024;
    if (!allow_smem<softmax_tc_kernel<false, false>>(most) || !allow_smem<softmax_tc_kernel<false, true>>(most) || !allow_smem<softmax_tc_kernel<true, false>>(most) ||
        !allow_smem<softmax_tc_kernel<true, true>>(most) || !softmax_takes_tc(a)) return cudaErrorInvalidValue;
    CUtensorMap mk, mv;
    if (!bf16_rows_map(&mk, a.k_pool, a.d, a.pool_rows, a.d, 1, 0, 64) || !bf16_rows_map(&mv, a.v_pool, a.dv, a.pool_rows, a.dv, 1, 0, 64)) return cudaErrorInvalidValue;
    const size_t smem = (size_t)(4 * k_parts + 2 * v_parts) * SX_PART + 1024;
    // heads a CTA: 32 sequences of 2 tokens, 16 heads over 4, 53 us with one and 24 with four; of 40 tokens, 60 with one and 45 with two
    SxShort sh = {};
    int ctas = 0;
    for (int k = 6; k >= 0; k--) {
        int heads = std::min(a.H / a.G, SX_Q >> k);
        while (a.H / a.G % heads) heads--;
        sh.heads[k] = heads;
        sh.tile0[k] = std::max(k ? r.n_upto[k - 1] : 0, a.skip);
        sh.cta0[k] = ctas;
        ctas += (r.n_upto[k] - sh.tile0[k]) * (a.H / heads);
    }
    const dim3 grid((r.n_tiles - r.n_upto[6] - r.n_odd) * a.H + ctas), block(SX_THREADS);
    if (grid.x == 0) return cudaSuccess;
    const auto kernel = a.softcap > 0.f ? (ctas ? softmax_tc_kernel<true, true> : softmax_tc_kernel<true, false>)
                                        : (ctas ? softmax_tc_kernel<false, true> : softmax_tc_kernel<false, false>);
    return launch_chain(kernel, grid, block, smem, s, mk, mv, a, r, sh, kernel_error_word());
}

}  // namespace b2
