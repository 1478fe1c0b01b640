// Attention whose keys and values are made from one small cached vector per token ("latent attention").
//
// Per token the layer's input product gives a query of H heads, each [D plain | R rotated] wide, and one row of
// C + R numbers: the first C, RMS-normed with a weight, are the latent c; the last R are a rotated key part shared by
// all heads.  Head n's key is [Wuk_n c | rotated part], its value Wuv_n c.  Only the row [c | rotated part] is cached
// (one "kv head" of width C + R; the value of a key is the first C columns of the same row), and the two
// up-projections move to the query side:
//     q_n . k_n = (Wuk_n^T q_n,plain) . c + q_n,rot . k_rot        out_n = Wuv_n (sum_j p_j c_j)
// so a step runs  prepare -> per-head product with Wuk^T -> attention over the latent rows -> per-head product with
// Wuv -> finish (optional sigmoid gate per head, heads side by side).  The per-head products are the engine's
// matrix-product kernels; queries and results are kept head-major, [H, rows, width], for them.
//
// prepare: per token one block for the latent row and one per group of heads.  c = row[:C] / sqrt(mean(row[:C]^2) + eps) * w (32-bit); the first `rot` of the R
//   rotated coordinates of the key part and of every head's query turn by position * freq[i], cos and sin times
//   `amp` (a 64-bit frequency table and the amplitude come from the host, so any scaling of the frequencies is the host's);
//   pairing 0: coordinate i with i + rot/2, pairing 1: 2i with 2i + 1.  The row [c | key part] goes to the token's
//   page, the plain query parts to q_plain (the element type of the step) and the rotated ones to q_rot (float32).
// attention (this file: the any-type kernel, one warp per (token, head); keys in ascending chunks of 32 aligned to
//   absolute positions, running maximum and sum in 32-bit, so a token's arithmetic depends on its own position only).
//   With a window W a query at position p sees the keys p - W + 1 .. p; with sinks (one number per head) the softmax's
//   denominator has one more term exp(sink) without a value.
// finish: out[t, n * V + v] = val[n, t, v] * sigmoid(gate[t, n]).
#include "attn_common.cuh"
#include "outer_memory.cuh"
#include <math_constants.h>

namespace {

constexpr int PREP_THREADS = 128;

// The angle is position times frequency in 64-bit, brought into [-pi, pi] there and only then rounded: a 32-bit product
// is off by its own size times 2^-24, which at position 1,000 is already 6e-5 of a turn's worth of radians.
__device__ __forceinline__ float2 turn(double ang, float amp) {
    const double two_pi = 6.283185307179586476925286766559;
    ang -= two_pi * rint(ang / two_pi);
    float s, c;
    sincosf((float)ang, &s, &c);
    return make_float2(c * amp, s * amp);
}

// element i of a rotated part: what it becomes with the token's cosines and sines, cs(pair)
template <typename CS>
__device__ __forceinline__ float rotated(const float* __restrict__ part, int i, int rot, int pairing, CS cs) {
    if (i >= rot) return part[i];
    int ia, ib;
    if (pairing) ia = i & ~1, ib = ia + 1;
    else ia = i < rot / 2 ? i : i - rot / 2, ib = ia + rot / 2;
    const float2 t = cs(pairing ? i >> 1 : ia);
    const float a = part[ia], b = part[ib];
    return i == ia ? a * t.x - b * t.y : b * t.x + a * t.y;
}

// The rotated part's width where the kernel that reads it takes blocks of 64 columns (zeros behind the R-th).
constexpr int ROT_BLOCK = 64;

// A token's cosines and sines are the same for all its heads and for the key part, and their 64-bit angles are most of the
// work, so a block makes them once, into shared memory (2,048 tokens of 16 heads of 128 + 64: 30 us an element at a time, 24 from the
// table).  TABLE off: more of them than fit there, made where they are used.
constexpr int MAX_TABLE = 4096;
template <typename T, bool TABLE>
__global__ void __launch_bounds__(PREP_THREADS)
latent_prepare_kernel(const float* __restrict__ proj, int proj_stride, const float* __restrict__ q_src, int q_stride,
                      int q_off, int kv_off,
                      const float* __restrict__ norm_w, float eps, const double* __restrict__ freq, int rot, int pairing,
                      float amp, const int* __restrict__ positions, const int* __restrict__ tok_entry,
                      const int* __restrict__ block_table, int max_blocks, int page_size, T* __restrict__ cache,
                      int write_cache, T* __restrict__ q_plain, float* __restrict__ q_rot, T* __restrict__ q_rot_block,
                      long long head_rows, int H, int D, int R, int C, int heads_per_block) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float2 table[];                    // [rot / 2]: amp * (cos, sin)
    __shared__ float red[32];
    const int t = blockIdx.x;
    const float* row = proj + (size_t)t * proj_stride;
    const int pos = positions[t];
    if (blockIdx.y == 0 && !write_cache) return;
    if (TABLE) {
        for (int i = threadIdx.x; i < rot / 2; i += blockDim.x) table[i] = turn((double)pos * freq[i], amp);
        __syncthreads();
    }
    auto cs = [&](int pair) { return TABLE ? table[pair] : turn((double)pos * freq[pair], amp); };
    if (blockIdx.y == 0) {
        // the latent row
        const float* kv = row + kv_off;
        float sq = 0.f;
        for (int i = threadIdx.x; i < C; i += blockDim.x) sq = fmaf(kv[i], kv[i], sq);
        const float rstd = 1.0f / sqrtf(block_sum(sq, red) / (float)C + eps);
        const int page = block_table[(size_t)tok_entry[t] * max_blocks + pos / page_size];
        T* dst = cache + ((size_t)page * page_size + (pos % page_size)) * (C + R);
        for (int i = threadIdx.x; i < C; i += blockDim.x) dst[i] = from_f32<T>(kv[i] * rstd * norm_w[i]);
        for (int i = threadIdx.x; i < R; i += blockDim.x) dst[C + i] = from_f32<T>(rotated(kv + C, i, rot, pairing, cs));
        return;
    }
    // the queries of heads [n0, n1)
    const int n0 = (blockIdx.y - 1) * heads_per_block, n1 = min(H, n0 + heads_per_block);
    const float* q = q_src + (size_t)t * q_stride + q_off;
    for (int i = n0 * D + threadIdx.x; i < n1 * D; i += blockDim.x) {
        const int n = i / D, c = i % D;
        q_plain[((size_t)n * head_rows + t) * D + c] = from_f32<T>(q[(size_t)n * (D + R) + c]);
    }
    if (q_rot_block) {
        for (int i = n0 * ROT_BLOCK + threadIdx.x; i < n1 * ROT_BLOCK; i += blockDim.x) {
            const int n = i / ROT_BLOCK, c = i % ROT_BLOCK;
            const float v = c < R ? rotated(q + (size_t)n * (D + R) + D, c, rot, pairing, cs) : 0.f;
            q_rot_block[((size_t)n * head_rows + t) * ROT_BLOCK + c] = from_f32<T>(v);
        }
        return;
    }
    for (int i = n0 * R + threadIdx.x; i < n1 * R; i += blockDim.x) {
        const int n = i / R, c = i % R;
        q_rot[((size_t)n * head_rows + t) * R + c] = rotated(q + (size_t)n * (D + R) + D, c, rot, pairing, cs);
    }
}

constexpr int WARPS = 4;
constexpr int MAX_C = 1024;           // widest latent the any-type kernel keeps in registers (32 per lane)

template <typename T>
__global__ void __launch_bounds__(WARPS * 32)
latent_attention_generic_kernel(const float* __restrict__ q_lat, const float* __restrict__ q_rot, long long head_rows,
                                T* __restrict__ out, const T* __restrict__ cache, const int* __restrict__ block_table,
                                int max_blocks, const int* __restrict__ tok_entry, const int* __restrict__ positions,
                                int tok_first, int n_tokens, int H, int C, int R, int page_size, float scale, int window,
                                const float* __restrict__ sinks) {
    extern __shared__ float q_s[];                       // [WARPS][C + R]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * WARPS + warp;
    if (item >= (long long)n_tokens * H) return;
    const int t = tok_first + (int)(item / H), n = (int)(item % H);
    const int W = C + R;
    float* qs = q_s + (size_t)warp * W;
    const size_t qrow = (size_t)n * head_rows + t;
    for (int i = lane; i < C; i += 32) qs[i] = q_lat[qrow * C + i];
    for (int i = lane; i < R; i += 32) qs[C + i] = q_rot[qrow * R + i];
    __syncwarp();
    const int pos = positions[t];
    const int* table = block_table + (size_t)tok_entry[t] * max_blocks;

    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    float m = sinks ? sinks[n] : -CUDART_INF_F, l = sinks ? 1.f : 0.f;       // a sink counts as a key seen before all others
    float acc[MAX_C / 32];
#pragma unroll
    for (int i = 0; i < MAX_C / 32; ++i) acc[i] = 0.f;
    for (int j0 = lo / 32 * 32; j0 <= pos; j0 += 32) {
        const int j = j0 + lane;
        long long row = -1;
        float s = -CUDART_INF_F;
        if (j >= lo && j <= pos) {
            const int page = table[j / page_size];
            if (page >= 0) {
                row = ((long long)page * page_size + (j % page_size)) * W;
                const T* kr = cache + row;
                float d = 0.f;
                for (int i = 0; i < W; ++i) d = fmaf(qs[i], to_f32(kr[i]), d);
                s = d * scale;
            }
        }
        const float m_new = fmaxf(m, warp_max(s));
        if (m_new == -CUDART_INF_F) continue;
        const float p = (row >= 0) ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < MAX_C / 32; ++i) acc[i] *= corr;
        for (int jj = 0; jj < 32; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const long long rj = __shfl_sync(0xffffffffu, row, jj);
            if (rj < 0) continue;
            const T* vr = cache + rj;
#pragma unroll
            for (int i = 0; i < MAX_C / 32; ++i) {
                const int dd = i * 32 + lane;
                if (dd < C) acc[i] = fmaf(pj, to_f32(vr[dd]), acc[i]);
            }
        }
        m = m_new;
    }
    T* orow = out + qrow * C;
    const float inv = 1.0f / l;
#pragma unroll
    for (int i = 0; i < MAX_C / 32; ++i) {
        const int dd = i * 32 + lane;
        if (dd < C) orow[dd] = from_f32<T>(acc[i] * inv);
    }
}

template <typename T>
__global__ void latent_finish_kernel(const float* __restrict__ val, long long head_rows, const float* __restrict__ gate,
                                     int gate_stride, T* __restrict__ out, int out_stride, int H, int V) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    for (int i = threadIdx.x; i < H * V; i += blockDim.x) {
        const int n = i / V, v = i % V;
        float x = val[((size_t)n * head_rows + t) * V + v];
        if (gate) x *= 1.0f / (1.0f + expf(-gate[t * gate_stride + n]));
        out[t * out_stride + i] = from_f32<T>(x);
    }
}

// ---- steps of few single tokens (bf16) ---------------------------------------------------------------------------------
// What is around the attention of up to FEW_TOKENS tokens in two launches instead of five: every launch costs more than its
// work here, and the tiles of 128 rows of the grouped products were mostly padding.  Both kernels ask for their weights before they
// wait for the kernel in front.  A layer of 16 heads of 128 + 64, latent 512, eight tokens: the launches around the attention
// 27 us (in five, one after the other), 15 in two; a step of four such layers with experts 462 us before, 404 now.
constexpr int FEW_TOKENS = 16, FEW_COLS = 64, FEW_MAX_D = 128;

// Blocks 0 .. T - 1: a token's latent row.  Then for every head the blocks of FEW_COLS latent columns, a warp 16 of them, and
// one block that turns the rotated parts.  q_lat = bf16(q plain) Wuk^T on mma.sync with the columns as rows of the tile and the
// tokens as its eight columns; a lane's 16 bytes of a row serve two steps of k (the order of k is the same on both sides).
template <int OCT>
__global__ void __launch_bounds__(128)
latent_query_few_kernel(const float* __restrict__ proj, int proj_stride, const float* __restrict__ q_src, int q_stride, int q_off,
                        int kv_off, const float* __restrict__ norm_w, float eps, const double* __restrict__ freq, int rot, int pairing,
                        float amp, const int* __restrict__ positions, const int* __restrict__ tok_entry,
                        const int* __restrict__ block_table, int max_blocks, int page_size, bf16* __restrict__ cache, int write_cache,
                        const bf16* __restrict__ w_k, float* __restrict__ q_lat, float* __restrict__ q_rot, long long head_rows,
                        int T, int H, int D, int R, int C) {
    extern __shared__ float2 table[];                    // a latent row: [rot / 2]
    __shared__ __align__(16) bf16 qs[8 * OCT][FEW_MAX_D + 8];
    __shared__ float red[32];
    pdl_launch_dependents();
    const int tid = threadIdx.x;
    if ((int)blockIdx.x < T) {
        pdl_wait();
        if (!write_cache) return;
        const int t = blockIdx.x, pos = positions[t];
        for (int i = tid; i < rot / 2; i += blockDim.x) table[i] = turn((double)pos * freq[i], amp);
        __syncthreads();
        auto cs = [&](int pair) { return table[pair]; };
        const float* kv = proj + (size_t)t * proj_stride + kv_off;
        float sq = 0.f;
        for (int i = tid; i < C; i += blockDim.x) sq = fmaf(kv[i], kv[i], sq);
        const float rstd = 1.0f / sqrtf(block_sum(sq, red) / (float)C + eps);
        const int page = block_table[(size_t)tok_entry[t] * max_blocks + pos / page_size];
        bf16* dst = cache + ((size_t)page * page_size + (pos % page_size)) * (C + R);
        for (int i = tid; i < C; i += blockDim.x) dst[i] = from_f32<bf16>(kv[i] * rstd * norm_w[i]);
        for (int i = tid; i < R; i += blockDim.x) dst[C + i] = from_f32<bf16>(rotated(kv + C, i, rot, pairing, cs));
        return;
    }
    const int chunks = C / FEW_COLS, n = ((int)blockIdx.x - T) / (chunks + 1), ch = ((int)blockIdx.x - T) % (chunks + 1);
    const float* q0 = q_src + q_off + (size_t)n * (D + R);
    if (ch == chunks) {
        pdl_wait();
        for (int i = tid; i < T * R; i += blockDim.x) {
            const int t = i / R, c = i % R;
            const float* part = q0 + (size_t)t * q_stride + D;
            float v = part[c];
            if (c < rot) {
                const int ia = pairing ? c & ~1 : c < rot / 2 ? c : c - rot / 2, ib = pairing ? ia + 1 : ia + rot / 2;
                const float2 f = turn((double)positions[t] * freq[pairing ? c >> 1 : ia], amp);
                v = c == ia ? part[ia] * f.x - part[ib] * f.y : part[ib] * f.x + part[ia] * f.y;
            }
            q_rot[((size_t)n * head_rows + t) * R + c] = v;
        }
        return;
    }
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, c4 = lane & 3, col0 = ch * FEW_COLS + warp * 16;
    const bf16* wr = w_k + ((size_t)n * C + col0 + g) * D + c4 * 8;
    uint4 wa[FEW_MAX_D / 32], wb[FEW_MAX_D / 32];
#pragma unroll
    for (int k = 0; k < FEW_MAX_D / 32; ++k)
        if (k * 32 < D) {
            wa[k] = __ldg(reinterpret_cast<const uint4*>(wr + k * 32));
            wb[k] = __ldg(reinterpret_cast<const uint4*>(wr + (size_t)8 * D + k * 32));
        }
    pdl_wait();
    for (int i = tid; i < 8 * OCT * D; i += blockDim.x) {
        const int t = i / D, c = i % D;
        qs[t][c] = from_f32<bf16>(t < T ? q0[(size_t)t * q_stride + c] : 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < OCT; ++o) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < FEW_MAX_D / 32; ++k)
            if (k * 32 < D) {
                const uint4 qb = *reinterpret_cast<const uint4*>(&qs[o * 8 + g][k * 32 + c4 * 8]);
                const uint32_t a0[4] = {wa[k].x, wb[k].x, wa[k].y, wb[k].y}, a1[4] = {wa[k].z, wb[k].z, wa[k].w, wb[k].w};
                attn::mma16816(acc, a0, qb.x, qb.y);
                attn::mma16816(acc, a1, qb.z, qb.w);
            }
        const int t = o * 8 + c4 * 2;
#pragma unroll
        for (int x = 0; x < 2; ++x)
            if (t + x < T) {
                float* dst = q_lat + ((size_t)n * head_rows + t + x) * C + col0 + g;
                dst[0] = acc[x];
                dst[8] = acc[2 + x];
            }
    }
}

// A block per (head, token): the ranges' results merged (or the finished one read), rounded to bf16 as the product's operand, then
// out[t, n V + v] = (Wuv row v . that) * sigmoid(gate): a warp eight rows at a time, a lane eight neighbouring columns of each 256.
constexpr int FEW_ROWS = 8, FEW_MAX_C = 512, FEW_MAX_SPLITS = 64;
__global__ void __launch_bounds__(256)
latent_result_few_kernel(const bf16* __restrict__ o_lat, long long head_rows, const float* __restrict__ part_o,
                         const float* __restrict__ part_ml, int splits, const float* __restrict__ sinks_log2, const bf16* __restrict__ w_v,
                         const float* __restrict__ gate, int gate_stride, bf16* __restrict__ out, int out_stride, int H, int C, int V) {
    __shared__ float w_s[FEW_MAX_SPLITS];
    __shared__ float inv_s;
    __shared__ __align__(16) bf16 o_s[FEW_MAX_C];
    pdl_launch_dependents();
    const int n = blockIdx.x, t = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int NJ = FEW_MAX_C / 256;
    uint4 w[FEW_ROWS][NJ];
    auto fetch = [&](int v0) {
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int k = j * 256 + lane * 8;
                w[r][j] = make_uint4(0, 0, 0, 0);
                if (v0 + r < V && k < C) w[r][j] = __ldg(reinterpret_cast<const uint4*>(w_v + ((size_t)n * V + v0 + r) * C + k));
            }
    };
    fetch(warp * FEW_ROWS);
    pdl_wait();
    if (splits > 1) {
        const size_t item0 = ((size_t)t * H + n) * splits;
        if (warp == 0) {
            const float2* ml = reinterpret_cast<const float2*>(part_ml) + item0;
            const float2 none = make_float2(-CUDART_INF_F, 0.f);
            const float2 a = lane < splits ? ml[lane] : none, b = lane + 32 < splits ? ml[lane + 32] : none;
            const float M = warp_max(fmaxf(a.x, b.x));
            const float w0 = a.x == -CUDART_INF_F ? 0.f : exp2f(a.x - M), w1 = b.x == -CUDART_INF_F ? 0.f : exp2f(b.x - M);
            w_s[lane] = w0, w_s[lane + 32] = w1;
            float L = warp_sum(w0 * a.y + w1 * b.y);
            if (sinks_log2) L += exp2f(sinks_log2[n] - M);
            if (lane == 0) inv_s = 1.0f / L;
        }
        __syncthreads();
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            const float* src = part_o + item0 * C + c;
            float acc = 0.f;
            for (int s0 = 0; s0 < splits; s0 += 8) {
                float v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = s0 + k < splits ? src[(size_t)(s0 + k) * C] : 0.f;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (s0 + k < splits) acc = fmaf(w_s[s0 + k], v[k], acc);
            }
            o_s[c] = from_f32<bf16>(acc * inv_s);
        }
    } else {
        for (int c = threadIdx.x; c < C; c += blockDim.x) o_s[c] = o_lat[((size_t)n * head_rows + t) * C + c];
    }
    __syncthreads();
    float o[NJ][8];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) o[j][i] = j * 256 + lane * 8 + i < C ? to_f32(o_s[j * 256 + lane * 8 + i]) : 0.f;
    const float sg = gate ? 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + n])) : 1.0f;
    for (int v0 = warp * FEW_ROWS; v0 < V; v0 += 8 * FEW_ROWS) {
        float dot[FEW_ROWS];
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r) {
            dot[r] = 0.f;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&w[r][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(p[i]);
                    dot[r] = fmaf(f.x, o[j][2 * i], dot[r]);
                    dot[r] = fmaf(f.y, o[j][2 * i + 1], dot[r]);
                }
            }
        }
        if (v0 + 8 * FEW_ROWS < V) fetch(v0 + 8 * FEW_ROWS);
        memory::scatter_sum<FEW_ROWS, 32>(dot, lane);        // row r's in lane 4 r
        const int v = v0 + (lane >> 2);
        if (!(lane & 3) && v < V) out[(size_t)t * out_stride + (size_t)n * V + v] = from_f32<bf16>(dot[0] * sg);
    }
}

}  // namespace

extern "C" {

// proj float32 [T, proj_stride]: the C + R columns of the latent row from kv_off.  q_src float32 [T, q_stride]: the
// query's H * (D + R) columns from q_off (the same array as proj where one product gives both, another where the queries
// come from a product of their own).  cache [pages, 1, page, C + R]; q_plain [H, head_rows, D] of the cache's type; q_rot
// float32 [H, head_rows, R] (R may be 0: no rotated part), or, where q_rot_block is given, [H, head_rows, 64] of the cache's
// type there instead, zeros behind the R-th column.
int infero_latent_prepare_from(const float* proj, int proj_stride, const float* q_src, int q_stride, int q_off, int kv_off,
                               const float* norm_w, float eps,
                          const double* freq, int rot, int pairing, float amp, const int* positions, const int* tok_entry,
                          const int* block_table, int max_blocks, int page_size, void* cache, int dtype, int write_cache,
                          void* q_plain, float* q_rot, void* q_rot_block, long long head_rows, int n_tokens, int H, int D,
                          int R, int C, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    INFERO_REQUIRE(!q_rot_block || R <= ROT_BLOCK, "latent attention: a rotated part of %d in one block of %d", R, ROT_BLOCK);
    INFERO_REQUIRE(rot >= 0 && rot <= R && rot % 2 == 0, "latent attention: %d rotated coordinates of %d", rot, R);
    INFERO_REQUIRE(head_rows >= n_tokens, "latent attention: %lld rows per head for %d tokens", head_rows, n_tokens);
    // one block for a token's latent row, and one per group of heads (all heads in one block where tokens alone fill
    // the multiprocessors)
    const int heads_per_block = n_tokens >= 512 ? H : max(1, H / 8);
    const dim3 grid(n_tokens, 1 + (H + heads_per_block - 1) / heads_per_block);
    const bool table = rot / 2 <= MAX_TABLE;
#define PREPARE(T_, TABLE_)                                                                                                              \
    launch_pdl(latent_prepare_kernel<T_, TABLE_>, grid, dim3(PREP_THREADS), TABLE_ ? rot / 2 * sizeof(float2) : 0, stream, proj, proj_stride, \
               q_src, q_stride, q_off, kv_off, norm_w, eps, freq, rot, pairing, amp, positions, tok_entry, block_table, max_blocks, page_size,  \
               (T_*)cache, write_cache, (T_*)q_plain, q_rot, (T_*)q_rot_block, head_rows, H, D, R, C, heads_per_block)
    if (dtype == INFERO_F32) {
        if (table) PREPARE(float, true);
        else PREPARE(float, false);
    } else {
        if (table) PREPARE(bf16, true);
        else PREPARE(bf16, false);
    }
#undef PREPARE
    return infero_check_launch("latent_prepare");
}

int infero_latent_prepare(const float* proj, int proj_stride, int q_off, int kv_off, const float* norm_w, float eps,
                          const double* freq, int rot, int pairing, float amp, const int* positions, const int* tok_entry,
                          const int* block_table, int max_blocks, int page_size, void* cache, int dtype, int write_cache,
                          void* q_plain, float* q_rot, long long head_rows, int n_tokens, int H, int D, int R, int C,
                          cudaStream_t stream) {
    return infero_latent_prepare_from(proj, proj_stride, proj, proj_stride, q_off, kv_off, norm_w, eps, freq, rot, pairing, amp,
                                      positions, tok_entry, block_table, max_blocks, page_size, cache, dtype, write_cache,
                                      q_plain, q_rot, nullptr, head_rows, n_tokens, H, D, R, C, stream);
}

// q_lat float32 [H, head_rows, C] (the plain query parts carried through Wuk^T), q_rot float32 [H, head_rows, R];
// out [H, head_rows, C] of the cache's type: softmax-weighted sums of the latent rows.  Tokens tok_first .. + n_tokens.
// window > 0: only that many keys up to the token's own; sinks float32 [H] or null.
int infero_latent_attention_generic(const float* q_lat, const float* q_rot, long long head_rows, void* out, const void* cache,
                                    int dtype, const int* block_table, int max_blocks, const int* tok_entry,
                                    const int* positions, int tok_first, int n_tokens, int H, int C, int R, int page_size,
                                    float scale, int window, const float* sinks, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    INFERO_REQUIRE(C >= 1 && C <= MAX_C, "latent attention: latent width %d outside 1..%d", C, MAX_C);
    const size_t sh = (size_t)WARPS * (C + R) * sizeof(float);
    INFERO_REQUIRE(sh <= 48 * 1024, "latent attention: key width %d too large", C + R);
    const long long items = (long long)n_tokens * H;
    const unsigned blocks = (unsigned)((items + WARPS - 1) / WARPS);
    if (dtype == INFERO_F32)
        latent_attention_generic_kernel<float><<<blocks, WARPS * 32, sh, stream>>>(q_lat, q_rot, head_rows, (float*)out,
            (const float*)cache, block_table, max_blocks, tok_entry, positions, tok_first, n_tokens, H, C, R, page_size, scale, window, sinks);
    else
        latent_attention_generic_kernel<bf16><<<blocks, WARPS * 32, sh, stream>>>(q_lat, q_rot, head_rows, (bf16*)out,
            (const bf16*)cache, block_table, max_blocks, tok_entry, positions, tok_first, n_tokens, H, C, R, page_size, scale, window, sinks);
    return infero_check_launch("latent_attention_generic");
}

// val float32 [H, head_rows, V]; gate float32 (row stride gate_stride, one column per head) or null; out [T, H * V].
int infero_latent_finish(const float* val, long long head_rows, const float* gate, int gate_stride, void* out,
                         int out_stride, int dtype, int n_tokens, int H, int V, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    if (dtype == INFERO_F32)
        launch_pdl(latent_finish_kernel<float>, dim3(n_tokens), dim3(256), 0, stream, val, head_rows, gate, gate_stride, (float*)out, out_stride, H, V);
    else
        launch_pdl(latent_finish_kernel<bf16>, dim3(n_tokens), dim3(256), 0, stream, val, head_rows, gate, gate_stride, (bf16*)out, out_stride, H, V);
    return infero_check_launch("latent_finish");
}

// Steps of up to 16 single tokens in bf16 (every token's request brings it alone).
int infero_latent_few_supported(int n_tokens, int D, int C) {
    return n_tokens >= 1 && n_tokens <= FEW_TOKENS && D >= 32 && D <= FEW_MAX_D && D % 32 == 0 && C >= FEW_COLS && C % FEW_COLS == 0 && C <= FEW_MAX_C;
}

// infero_latent_prepare_from and the product with Wuk^T [H, C, D] in one: q_lat float32 [H, head_rows, C], q_rot float32
// [H, head_rows, R]; the tokens' latent rows go to the cache.
int infero_latent_query_few(const float* proj, int proj_stride, const float* q_src, int q_stride, int q_off, int kv_off,
                            const float* norm_w, float eps, const double* freq, int rot, int pairing, float amp, const int* positions,
                            const int* tok_entry, const int* block_table, int max_blocks, int page_size, void* cache, int write_cache,
                            const void* w_k, float* q_lat, float* q_rot, long long head_rows, int n_tokens, int H, int D, int R, int C,
                            cudaStream_t stream) {
    INFERO_REQUIRE(infero_latent_few_supported(n_tokens, D, C) && (reinterpret_cast<uintptr_t>(w_k) & 15u) == 0,
                   "latent_query_few: %d tokens, %d x %d, not supported", n_tokens, D, C);
    INFERO_REQUIRE(rot >= 0 && rot <= R && rot % 2 == 0 && rot / 2 <= MAX_TABLE && head_rows >= n_tokens, "latent attention: %d rotated coordinates of %d", rot, R);
    const dim3 grid(n_tokens + H * (C / FEW_COLS + 1));
#define GO(O_)                                                                                                                      \
    launch_pdl(latent_query_few_kernel<O_>, grid, dim3(128), rot / 2 * sizeof(float2), stream, proj, proj_stride, q_src, q_stride, q_off, \
               kv_off, norm_w, eps, freq, rot, pairing, amp, positions, tok_entry, block_table, max_blocks, page_size, (bf16*)cache, \
               write_cache, (const bf16*)w_k, q_lat, q_rot, head_rows, n_tokens, H, D, R, C)
    if (n_tokens <= 8) GO(1);
    else GO(2);
#undef GO
    return infero_check_launch("latent_query_few");
}

// From the attention's ranges (splits > 1: part_o, part_ml as infero_latent_attention_mma leaves them) or its finished result o_lat
// (splits = 1) to out [tokens, H V]: merge, product with Wuv [H, V, C], gate.
int infero_latent_result_few(const void* o_lat, long long head_rows, const float* part_o, const float* part_ml, int splits,
                             const float* sinks_log2, const void* w_v, const float* gate, int gate_stride, void* out, int out_stride,
                             int n_tokens, int H, int D, int C, int V, cudaStream_t stream) {
    INFERO_REQUIRE(infero_latent_few_supported(n_tokens, D, C) && V >= 1 && splits >= 1 && splits <= FEW_MAX_SPLITS &&
                       (reinterpret_cast<uintptr_t>(w_v) & 15u) == 0 && (splits == 1 ? o_lat != nullptr : part_o && part_ml),
                   "latent_result_few: %d tokens, latent %d, %d ranges, not supported", n_tokens, C, splits);
    launch_pdl(latent_result_few_kernel, dim3(H, n_tokens), dim3(256), 0, stream, (const bf16*)o_lat, head_rows, part_o, part_ml, splits,
               sinks_log2, (const bf16*)w_v, gate, gate_stride, (bf16*)out, out_stride, H, C, V);
    return infero_check_launch("latent_result_few");
}

}  // extern "C"
