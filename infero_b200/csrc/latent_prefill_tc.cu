// Latent attention for prompt portions on the 5th-generation tensor cores (bf16): keys and values written out per head.
//
// Carrying the up-projections to the query side (latent_attention_mma.cu) makes every (query, key) pair cost 2 C + R
// multiply-adds per head; a portion of many tokens amortises writing its keys and values out, after which a pair costs
// 2 D + R.  A step runs
//     gather: the visible latent rows of every portion, from their pages, side by side: c [keys, C] and the rotated part
//             [keys, 64]; a request's rows start at a multiple of 64 keys of its positions and end in zeros
//     one product (gemm_tc.cu): [Wuk; Wuv] c -> [keys, H D + H D], the keys bf16, the values IEEE halves
//     this file's attention over it, the output gate in its epilogue.
// At 2,048 tokens, 16 heads of 128 + 64 and a latent of 512 a layer's attention with its up-projections took 600 us
// through the latent rows (73 GFLOP of scores and sums, on mma.sync) and takes 71 written out (21.5 GFLOP, of it 38 us in the
// attention kernel).  Weights and values are IEEE halves: bf16 for both left a layer 1 to 6 % further from 64 bits than the latent
// rows do, halves leave it 17 to 23 % nearer (16 to 600 tokens, 8 heads of 64 + 32 and 16 of 128 + 64), in the same time.  A weight is
// 256 at most, and layers whose values could leave the range of halves (their weights bound them: the latent row is normed) keep to
// the latent rows.
//
// One CTA = 128 query rows of one request and one head; it walks the visible keys in tiles of 64.  The tensor memory holds
// two results: tiles of even number (of the absolute position) belong to warps 0..3, odd ones to warps 4..7, each with its
// own running maximum, sum and O, so the softmax of one tile runs under the products of the next; at the end the two are
// added up, every thread for its row and half of the columns.  (A head's keys are its own here, so there is no second head
// that could share them, as attention_prefill_tc.cu has it; 256 rows a CTA would leave too few CTAs: 128 at the size above.)
// Per tile: S = [q | q_rot] [k | k_rot]^T over D / 64 + 1 blocks of 64 columns (tcgen05.mma from shared memory, TMA with
// 128-byte swizzle), P = 2^(S c - m) by one thread a row, back over S as halves, O += P V.  Two S buffers a parity, so the
// products of the next two tiles are issued ahead.  Scores, maxima, sums and O are 32-bit.
//
// Same formula as latent_attention.cu: key j is visible from position p iff lo <= j <= p, lo = max(0, p - window + 1); a learned
// sink is one more term of the sum.  What is computed for a token here depends on its position only: tiles sit at multiples of 64
// of the absolute position.  (Which of the two routes it takes depends on the step: kernels/latent_prefill.py.)  Every wait is
// bounded, as in attention_prefill_tc.cu.
#include "tc_common.cuh"
#include "tc_softmax.cuh"
#include <math_constants.h>

namespace {

using namespace tc;

constexpr int QROWS = 128, KTILE = 64, BLOCK = 64;
constexpr int LP_K_WARP = 8, LP_V_WARP = 9, LP_MMA_WARP = 10, LP_THREADS = 352;       // warps 0..7: softmax
constexpr float RESCALE_STEP = 8.0f;

template <int D>
struct LpPlan {
    static constexpr int DB = D / 64;                        // 64-column blocks of a plain part or a value
    static constexpr int STAGES = D == 128 ? 4 : 6;
    static constexpr int QBLOCK_BYTES = QROWS * 128, KBLOCK_BYTES = KTILE * 128;
    static constexpr int Q_BYTES = (DB + 1) * QBLOCK_BYTES;
    static constexpr int K_BYTES = (DB + 1) * KBLOCK_BYTES, V_BYTES = DB * KBLOCK_BYTES;
    static constexpr int K_OFF = Q_BYTES, V_OFF = K_OFF + STAGES * K_BYTES, STAT_OFF = V_OFF + STAGES * V_BYTES;
    static constexpr int BAR_OFFSET = STAT_OFF + 2 * QROWS * 8;
    static constexpr int N_BARS = 1 + 4 * STAGES + 2 * 5;
    static constexpr int TOTAL = BAR_OFFSET + 8 * N_BARS + 64 + 1024;
    static constexpr uint32_t SIDE_COLS = 256, O_COL = 2 * KTILE, TMEM_COLS = 512;    // per parity: S, S, O
    static_assert(2 * KTILE + D <= 256 && TOTAL <= 227 * 1024 && TOTAL > 114 * 1024, "tensor memory, shared memory; one CTA per SM");
};

// First key that is kept for a portion: the lowest one its first token sees, down to a whole tile.
__device__ __forceinline__ int keys_from(int pos0, int window) { return window > 0 ? max(0, pos0 - window + 1) / KTILE * KTILE : 0; }
__device__ __forceinline__ int key_tiles(int pos0, int q_len, int window) {
    return (pos0 + q_len - keys_from(pos0, window) + KTILE - 1) / KTILE;
}

// One block per tile of 64 gathered keys; rows behind a request's last key are zeros (they are multiplied by weights of 0).
__global__ void __launch_bounds__(256)
latent_gather_kernel(const bf16* __restrict__ cache, const int* __restrict__ block_table, int max_blocks, int page_size,
                     const int* __restrict__ entry_q_len, const int* __restrict__ entry_pos0, int first_entry, int n_entries,
                     int window, int C, int R, bf16* __restrict__ lat, bf16* __restrict__ rot) {
    pdl_launch_dependents();
    pdl_wait();
    int e = first_entry, tile = (int)blockIdx.x;
    for (; e < n_entries; ++e) {
        const int n = key_tiles(entry_pos0[e], entry_q_len[e], window);
        if (tile < n) break;
        tile -= n;
    }
    const int end = e < n_entries ? entry_pos0[e] + entry_q_len[e] : 0;
    const int key0 = e < n_entries ? keys_from(entry_pos0[e], window) + tile * KTILE : 0;
    const int* table = block_table + (size_t)(e < n_entries ? e : 0) * max_blocks;
    const int W = C + R, cl = C / 8, per_row = cl + BLOCK / 8;           // 16-byte pieces
    for (int i = threadIdx.x; i < KTILE * per_row; i += blockDim.x) {
        const int r = i / per_row, p = i % per_row, key = key0 + r;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (key < end && (p < cl || (p - cl) * 8 < R)) {
            const int page = table[key / page_size];
            if (page >= 0) v = __ldg(reinterpret_cast<const uint4*>(cache + ((size_t)page * page_size + key % page_size) * W) + p);
        }
        const size_t row = (size_t)blockIdx.x * KTILE + r;
        if (p < cl) reinterpret_cast<uint4*>(lat + row * C)[p] = v;
        else reinterpret_cast<uint4*>(rot + row * BLOCK)[p - cl] = v;
    }
}

template <int D>
__global__ void __launch_bounds__(LP_THREADS)
latent_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                         const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_kr,
                         bf16* __restrict__ out, int out_stride, const float* __restrict__ gate, int gate_stride,
                         const int* __restrict__ entry_q_start, const int* __restrict__ entry_q_len,
                         const int* __restrict__ entry_pos0, int first_entry, int n_entries, int first_token, int n_tiles,
                         int n_heads, int head_rows, int rot_blocks, int window, float scale_log2,
                         const float* __restrict__ sinks_log2, int* __restrict__ err_flag) {
    using Plan = LpPlan<D>;
    constexpr int DB = Plan::DB, ST = Plan::STAGES;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    float2* stats = reinterpret_cast<float2*>(smem + Plan::STAT_OFF);         // [parity][row]: reference point, sum
    uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + Plan::BAR_OFFSET);  // 1
    uint64_t* k_full = q_full + 1;           // ST
    uint64_t* v_full = k_full + ST;          // ST
    uint64_t* k_empty = v_full + ST;         // ST
    uint64_t* v_empty = k_empty + ST;        // ST
    uint64_t* s_full = v_empty + ST;         // [parity][2]
    uint64_t* p_full = s_full + 4;           // [parity][2] (128 arrivals)
    uint64_t* o_done = p_full + 4;           // [parity]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* never_flag = abort_flag + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_qr);
        prefetch_tensormap(&map_kv);
        prefetch_tensormap(&map_kr);
        mbar_init(q_full, 1);
        for (int i = 0; i < 4 * ST; ++i) mbar_init(&k_full[i], 1);            // k_full, v_full, k_empty, v_empty
        for (int i = 0; i < 4; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], QROWS);
        }
        mbar_init(&o_done[0], 1);
        mbar_init(&o_done[1], 1);
        *abort_flag = 0;
        *never_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == LP_MMA_WARP) {
        tmem_alloc(tmem_slot, Plan::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();

    // ---- which head, which request and which block of 128 query rows? (longest first) ------------------
    const int h = (int)blockIdx.x;
    int e = -1, tile_in_e = 0, key_base = 0;
    {
        int left = n_tiles - 1 - (int)blockIdx.y;
        for (int i = first_entry; i < n_entries; ++i) {
            const int nt = (entry_q_len[i] + QROWS - 1) / QROWS;
            if (left < nt) { e = i; tile_in_e = left; break; }
            left -= nt;
            key_base += key_tiles(entry_pos0[i], entry_q_len[i], window) * KTILE;
        }
    }
    int n_kt = 0, kt_begin = 0, key_row = 0, q_row = 0, rows_here = 0, first_pos = 0;
    if (e >= 0) {
        const int q_len = entry_q_len[e], pos0 = entry_pos0[e], row_first = tile_in_e * QROWS;
        q_row = entry_q_start[e] - first_token + row_first;
        rows_here = min(QROWS, q_len - row_first);
        first_pos = pos0 + row_first;
        kt_begin = (window > 0 ? max(0, first_pos - window + 1) : 0) / KTILE;
        n_kt = (first_pos + rows_here - 1) / KTILE - kt_begin + 1;
        key_row = key_base + kt_begin * KTILE - keys_from(pos0, window);       // the first tile's row among the gathered keys
    }

    if (warp == LP_K_WARP || warp == LP_V_WARP) {
        // ---- loaders: one thread for the keys (and the queries), one for the values ------------------------
        const bool is_k = warp == LP_K_WARP;
        if (n_kt > 0 && elect_one()) {
            uint64_t* full = is_k ? k_full : v_full;
            uint64_t* empty = is_k ? k_empty : v_empty;
            const int bytes = is_k ? (DB + rot_blocks) * Plan::KBLOCK_BYTES : Plan::V_BYTES;
            uint8_t* ring = smem + (is_k ? Plan::K_OFF : Plan::V_OFF);
            if (is_k) {
                mbar_expect_tx(q_full, (DB + rot_blocks) * Plan::QBLOCK_BYTES);
                const int row = h * head_rows + q_row;
#pragma unroll
                for (int b = 0; b < DB; ++b) tma_load_2d(smem + b * Plan::QBLOCK_BYTES, &map_q, b * BLOCK, row, q_full);
                if (rot_blocks) tma_load_2d(smem + DB * Plan::QBLOCK_BYTES, &map_qr, 0, row, q_full);
            }
            const int col = (is_k ? h : n_heads + h) * D;
            bool ok = true;
            int issued = 0;
            for (int j = 0; j < n_kt; ++j) {
                const int s = j % ST, row = key_row + j * KTILE;
                if (!mbar_wait(&empty[s], ((uint32_t)(j / ST) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                mbar_expect_tx(&full[s], bytes);
                uint8_t* dst = ring + s * (is_k ? Plan::K_BYTES : Plan::V_BYTES);
#pragma unroll
                for (int b = 0; b < DB; ++b) tma_load_2d(dst + b * Plan::KBLOCK_BYTES, &map_kv, col + b * BLOCK, row, &full[s]);
                if (is_k && rot_blocks) tma_load_2d(dst + DB * Plan::KBLOCK_BYTES, &map_kr, 0, row, &full[s]);
                issued = j + 1;
            }
            if (!ok) {
                *abort_flag = 1;
                atomicExch(err_flag, 5);
            }
            if (*abort_flag) {
                // let copies that are still in flight land before the block goes away
                if (is_k) mbar_wait(q_full, 0, never_flag);
                for (int j = max(0, issued - ST); j < issued; ++j) mbar_wait(&full[j % ST], (uint32_t)(j / ST) & 1u, never_flag);
            }
        }
    } else if (warp == LP_MMA_WARP) {
        // ---- MMA issue: tile j belongs to parity (kt_begin + j) & 1 and is its (j >> 1)-th ----------------------
        if (n_kt > 0 && elect_one()) {
            constexpr uint32_t idesc_qk = idesc_bf16_f32(QROWS, KTILE);
            constexpr uint32_t idesc_pv = idesc_f16_f32_b_mn(QROWS, D);
            const uint32_t q_addr = smem_u32(smem);
            const int k_steps = (DB + rot_blocks) * (BLOCK / 16);
            bool ok = true;
            auto issue_qk = [&](int j) {
                if (!mbar_wait(&k_full[j % ST], (uint32_t)(j / ST) & 1u, abort_flag)) { ok = false; return; }
                tc_fence_after_sync();
                const uint32_t side = (uint32_t)(kt_begin + j) & 1u, buf = (uint32_t)(j >> 1) & 1u;
                const uint32_t k_addr = smem_u32(smem + Plan::K_OFF + (j % ST) * Plan::K_BYTES);
                const uint32_t s_tmem = tmem_base + side * Plan::SIDE_COLS + buf * KTILE;
                for (int ks = 0; ks < k_steps; ++ks) {
                    const uint32_t in_block = (uint32_t)(ks & 3) * 32u, blk = (uint32_t)(ks >> 2);
                    umma_bf16(s_tmem, smem_desc_k_sw128(q_addr + blk * Plan::QBLOCK_BYTES + in_block),
                              smem_desc_k_sw128(k_addr + blk * Plan::KBLOCK_BYTES + in_block), idesc_qk, ks > 0 ? 1u : 0u);
                }
                umma_commit(&s_full[side * 2 + buf]);
                umma_commit(&k_empty[j % ST]);
            };
            if (!mbar_wait(q_full, 0, abort_flag)) ok = false;
            for (int j = 0; j < 2 && j < n_kt && ok; ++j) issue_qk(j);
            for (int j = 0; j < n_kt && ok; ++j) {
                if (j + 2 < n_kt) {
                    issue_qk(j + 2);            // into the S buffer whose P the product issued two tiles ago has read
                    if (!ok) break;
                }
                const uint32_t side = (uint32_t)(kt_begin + j) & 1u, buf = (uint32_t)(j >> 1) & 1u;
                if (!mbar_wait(&v_full[j % ST], (uint32_t)(j / ST) & 1u, abort_flag)) { ok = false; break; }
                if (!mbar_wait(&p_full[side * 2 + buf], (uint32_t)(j >> 2) & 1u, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t v_addr = smem_u32(smem + Plan::V_OFF + (j % ST) * Plan::V_BYTES);
                const uint32_t o_tmem = tmem_base + side * Plan::SIDE_COLS + Plan::O_COL;
                const uint32_t p_tmem = tmem_base + side * Plan::SIDE_COLS + buf * KTILE;
#pragma unroll
                for (int ks = 0; ks < KTILE / 16; ++ks)
                    // 16 keys: 8 columns of P (two halves each), 16 rows of V (2048 bytes)
                    umma_bf16_ts(o_tmem, p_tmem + (uint32_t)ks * 8u, smem_desc_mn_sw128(v_addr + (uint32_t)ks * 2048u, Plan::KBLOCK_BYTES, 1024u),
                                 idesc_pv, (j > 1 || ks > 0) ? 1u : 0u);
                umma_commit(&o_done[side]);
                umma_commit(&v_empty[j % ST]);
            }
            if (!ok) {
                *abort_flag = 1;
                atomicExch(err_flag, 6);
            }
        }
    } else if (n_kt > 0) {
        // ---- softmax, correction of O, epilogue: one query row per thread and parity ----------------------------
        const int side = warp >> 2, r = (warp & 3) * 32 + lane;
        const bool valid = r < rows_here;
        const int pos_r = first_pos + r;
        const int hi_r = valid ? pos_r : -1, lo_r = window > 0 ? max(0, pos_r - window + 1) : 0;
        const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t my_tmem = tmem_base + (uint32_t)side * Plan::SIDE_COLS + lane_sel;
        const int j_first = side ^ (kt_begin & 1);
        float m = -CUDART_INF_F, l = 0.f;
        bool ok = true;
        int done = 0;                                        // tiles of this parity so far
        for (int j = j_first; j < n_kt; j += 2, ++done) {
            const int b = done & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&s_full[side * 2 + b], (uint32_t)(done >> 1) & 1u, abort_flag))) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t s_addr = my_tmem + (uint32_t)b * KTILE;
            const int kb = (kt_begin + j) * KTILE;
            // every key of the tile visible from every row of the block?
            const bool open_tile = (kb + KTILE - 1 <= first_pos) && (window <= 0 || kb >= first_pos + rows_here - 1 - window + 1);
            uint32_t sv[KTILE];
#pragma unroll
            for (int c = 0; c < KTILE / 32; ++c) tmem_ld32_nowait(s_addr + (uint32_t)c * 32u, sv + c * 32);
            tmem_wait_ld();
            float mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
            if (open_tile) {
#pragma unroll
                for (int i = 0; i < KTILE; i += 2)
                    mx4[(i >> 1) & 3] = fmax3(mx4[(i >> 1) & 3], __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
            } else {
#pragma unroll
                for (int i = 0; i < KTILE; ++i) {
                    const int key = kb + i;
                    if (!(key >= lo_r && key <= hi_r)) sv[i] = 0xff800000u;      // -inf: contributes 2^-inf = 0
                    mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[i]));
                }
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            // the reference point moves only when the maximum has grown by more than 2^RESCALE_STEP (see attention_prefill_tc.cu)
            const float m_seen = fmaxf(m, mx * scale_log2);
            const float m_new = (m_seen - m > RESCALE_STEP) ? m_seen : m;
            const float sub = m_new == -CUDART_INF_F ? 0.f : m_new;
            const float corr = ex2(m - sub);
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t pk[KTILE / 2];
#pragma unroll
            for (int i = 0; i < KTILE; i += 2) {
                float x0, x1;
                fma2(x0, x1, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]), scale_log2, -sub);
                const float p0 = ex2(x0), p1 = ex2(x1);
                sum4[(i >> 1) & 3] += p0 + p1;
                pk[i >> 1] = pack2_half(p0, p1);
            }
#pragma unroll
            for (int c = 0; c < KTILE / 32; ++c) tmem_st16(s_addr + (uint32_t)c * 16u, pk + c * 16);
            l = l * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
            m = m_new;
            if (done > 0) {
                // this parity's product before this one (waited for at every tile: a parity wait must not fall two phases behind)
                if (!__all_sync(0xffffffffu, mbar_wait(&o_done[side], (uint32_t)(done - 1) & 1u, abort_flag))) { ok = false; break; }
                if (__any_sync(0xffffffffu, corr != 1.0f)) {
                    tc_fence_after_sync();
                    const uint32_t o_addr = my_tmem + Plan::O_COL;
#pragma unroll 1
                    for (int c = 0; c < D / 32; ++c) {
                        uint32_t v[32];
                        tmem_ld32_nowait(o_addr + (uint32_t)c * 32u, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
                        tmem_st32(o_addr + (uint32_t)c * 32u, v);
                    }
                }
            }
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(&p_full[side * 2 + b]);
        }
        if (ok && done > 0 && !__all_sync(0xffffffffu, mbar_wait(&o_done[side], (uint32_t)(done - 1) & 1u, abort_flag))) ok = false;
        if (!ok) *abort_flag = 1;
        // both parities' results are complete and both know the other's reference point and sum
        stats[side * QROWS + r] = make_float2(m, l);
        tc_fence_before_sync();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        tc_fence_after_sync();
        if (!*abort_flag) {
            const float2 s0 = stats[r], s1 = stats[QROWS + r];
            const float top = fmaxf(s0.x, s1.x), ref = top == -CUDART_INF_F ? 0.f : top;
            const float a0 = ex2(s0.x - ref), a1 = ex2(s1.x - ref);          // (a parity without a tile: 2^-inf = 0)
            float sum = s0.y * a0 + s1.y * a1;
            if (sinks_log2) sum += ex2(sinks_log2[h] - ref);
            const int row = q_row + (valid ? r : 0);
            const float inv = 1.0f / sum;
            const float f0 = a0 * inv, f1 = a1 * inv;
            const float g = gate ? 1.0f / (1.0f + expf(-gate[(size_t)row * gate_stride + h])) : 1.0f;
            const bool two = n_kt > 1;
            const uint32_t base = tmem_base + lane_sel + Plan::O_COL;
            const uint32_t first = (uint32_t)(kt_begin & 1) * Plan::SIDE_COLS, second = Plan::SIDE_COLS - first;
            const float ff = kt_begin & 1 ? f1 : f0, fs = kt_begin & 1 ? f0 : f1;
            bf16* orow = out + (size_t)row * out_stride + (size_t)h * D;
#pragma unroll 1
            for (int c = side * (D / 2); c < (side + 1) * (D / 2); c += 32) {
                uint32_t v[32], w[32];
                tmem_ld32_nowait(base + first + (uint32_t)c, v);
                if (two) tmem_ld32_nowait(base + second + (uint32_t)c, w);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    float x = __uint_as_float(v[i]) * ff;
                    if (two) x = fmaf(__uint_as_float(w[i]), fs, x);
                    v[i] = __float_as_uint(x * g);
                }
                if (valid) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8)
                        *reinterpret_cast<uint4*>(orow + c + i) =
                            make_uint4(pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), pack2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])),
                                       pack2(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5])), pack2(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7])));
                }
                __syncwarp();
            }
        } else if (lane == 0) {
            atomicExch(err_flag, 7);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == LP_MMA_WARP) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, Plan::TMEM_COLS);
    }
}

template <int D>
int launch(const CUtensorMap& mq, const CUtensorMap& mqr, const CUtensorMap& mkv, const CUtensorMap& mkr, void* out, int out_stride,
           const float* gate, int gate_stride, const int* entry_q_start, const int* entry_q_len, const int* entry_pos0,
           int first_entry, int n_entries, int first_token, int n_tiles, int n_heads, int head_rows, int rot_blocks, int window,
           float scale_log2, const float* sinks_log2, int* err, cudaStream_t stream) {
    using Plan = LpPlan<D>;
    auto kern = latent_prefill_tc_kernel<D>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Plan::TOTAL);
        if (e != cudaSuccess) {
            infero_set_error("latent_prefill_tc: cannot get %d bytes of shared memory: %s", Plan::TOTAL, cudaGetErrorString(e));
            return 1;
        }
        configured = true;
    }
    launch_pdl(kern, dim3(n_heads, n_tiles), dim3(LP_THREADS), Plan::TOTAL, stream, mq, mqr, mkv, mkr, (bf16*)out, out_stride, gate,
               gate_stride, entry_q_start, entry_q_len, entry_pos0, first_entry, n_entries, first_token, n_tiles, n_heads, head_rows,
               rot_blocks, window, scale_log2, sinks_log2, err);
    return infero_check_launch("latent_prefill_tc");
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

extern "C" {

// D plain = D value columns a head, R rotated ones (at most one block of 64), latent width C.
int infero_latent_prefill_tc_supported(int D, int V, int R, int C) {
    return (D == 64 || D == 128) && V == D && R >= 0 && R <= BLOCK && R % 8 == 0 && C >= 8 && C % 8 == 0;
}

// The visible latent rows of the portions first_entry .. n_entries - 1, side by side: lat [64 * n_key_tiles, C] and
// rot [64 * n_key_tiles, 64]; n_key_tiles = the sum over them of ceil((pos0 + q_len - from) / 64) with from = 0, or
// max(0, pos0 - window + 1) down to a multiple of 64.
int infero_latent_gather(const void* cache, const int* block_table, int max_blocks, int page_size, const int* entry_q_len,
                         const int* entry_pos0, int first_entry, int n_entries, int n_key_tiles, int window, int C, int R,
                         void* lat, void* rot, cudaStream_t stream) {
    if (n_key_tiles == 0) return 0;
    INFERO_REQUIRE(C % 8 == 0 && R % 8 == 0 && R <= BLOCK && aligned16(cache) && aligned16(lat) && aligned16(rot),
                   "latent_gather: widths %d + %d, or an address, not in units of 16 bytes", C, R);
    launch_pdl(latent_gather_kernel, dim3(n_key_tiles), dim3(256), 0, stream, (const bf16*)cache, block_table, max_blocks, page_size,
               entry_q_len, entry_pos0, first_entry, n_entries, window, C, R, (bf16*)lat, (bf16*)rot);
    return infero_check_launch("latent_gather");
}

// q [H, head_rows, D] and q_rot [H, head_rows, 64] (bf16; row t is token first_token + t), kv [64 * n_key_tiles, 2 H D] = head
// by head the plain keys (bf16), then the values (IEEE halves), of the gathered rows, k_rot their rotated parts; out [tokens, >= H D] bf16;
// gate float32 [tokens, H] (row stride gate_stride) or null; n_tiles = the sum of ceil(q_len / 128) over the portions.
int infero_latent_prefill_tc(const void* q, const void* q_rot, int head_rows, const void* kv, const void* k_rot, int n_key_tiles,
                             void* out, int out_stride, const float* gate, int gate_stride, const int* entry_q_start,
                             const int* entry_q_len, const int* entry_pos0, int first_entry, int n_entries, int first_token,
                             int n_tiles, int H, int D, int V, int R, int C, float scale, int window, const float* sinks_log2,
                             cudaStream_t stream) {
    if (n_tiles == 0) return 0;
    INFERO_REQUIRE(infero_latent_prefill_tc_supported(D, V, R, C), "latent_prefill_tc: sizes D=%d V=%d R=%d C=%d not supported", D, V, R, C);
    INFERO_REQUIRE(n_tiles <= 65535 && H >= 1 && out_stride % 8 == 0 && aligned16(out) && aligned16(q) && aligned16(q_rot) && aligned16(kv) &&
                       aligned16(k_rot),
                   "latent_prefill_tc: %d tiles, %d heads, row stride %d, or an address, not supported", n_tiles, H, out_stride);
    INFERO_REQUIRE((long long)H * head_rows < (1ll << 31) && (long long)n_key_tiles * KTILE < (1ll << 31), "latent_prefill_tc: too many rows");
    CUtensorMap mq, mqr, mkv, mkr;
    const int keys = n_key_tiles * KTILE;
    if (infero_tensor_map_bf16(q, H * head_rows, D, D, QROWS, &mq)) return 1;
    if (infero_tensor_map_bf16(q_rot, H * head_rows, BLOCK, BLOCK, QROWS, &mqr)) return 1;
    if (infero_tensor_map_bf16(kv, keys, 2 * H * D, 2 * H * D, KTILE, &mkv)) return 1;
    if (infero_tensor_map_bf16(k_rot, keys, BLOCK, BLOCK, KTILE, &mkr)) return 1;
    int* err;
    if (infero_tc_err_flag(&err)) return 1;
    const float sl2 = scale * 1.4426950408889634f;
#define GO(D_) return launch<D_>(mq, mqr, mkv, mkr, out, out_stride, gate, gate_stride, entry_q_start, entry_q_len, entry_pos0, first_entry, \
                                 n_entries, first_token, n_tiles, H, head_rows, R > 0 ? 1 : 0, window, sl2, sinks_log2, err, stream)
    if (D == 128) GO(128);
    GO(64);
#undef GO
}

}  // extern "C"
