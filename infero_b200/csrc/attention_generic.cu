// Attention over the paged cache for any batch of tokens: a row per (token, query head).
//
// For token t of request entry e at position p, head h (kv head h / group):
//   s_j = (q . K[j]) * scale - slope_h * (p - j)   for lo <= j <= p,  lo = window ? max(0, p - window + 1) : 0
//   (slope_h: a per-head distance bias, zero where the caller gives no slopes; or a table by distance,
//   s_j + rel[h][min(p - j, rel_len - 1)]; with a soft cap the scaled product becomes cap tanh(. / cap) before any bias)
//   out = sum_j softmax(s)_j V[j]
// With `cross` head h's weights meet the values of every kv head c, not only its own: out has G * H rows per token, row
// c * H + h, in 32-bit (what a mixing of the heads' weights needs, see head_mix.cu).
// (crates/kernels/src/cu/ops.cu:709-811 is the reference's three-kernel statement; its
// fused decode kernel is ops.cu:1773-2075.  Contiguous head groups: kv head = h / group.)
//
// Keys are visited in ascending order in chunks of 32 aligned to absolute positions, with a
// running maximum and sum (all 32-bit, accurate expf).  The arithmetic done for a token
// depends only on its own position and window, never on how the step was cut or on what
// else is in the batch.  It takes every head size up to 256 and every group size; it is the
// whole of attention on the 32-bit path and the fallback of the bf16 path.
//
// A block has a few neighbouring tokens and the query heads of one kv head: their rows (token, head), R a warp, share the
// chunks, which are fetched into shared memory a chunk ahead of the arithmetic; a lane looks up its own key's page a chunk before
// that.  In the scores a lane has a key, in the sum over values it has every 32nd column.  Tokens of different requests in one
// block take turns, so single tokens and short portions get a block per token, with warps that only fetch where a kv head has
// fewer query heads than a block wants warps.
// What bounds it: long prompts the multiply-adds and what feeds them from shared memory, single tokens the chain over the
// chunks.  A warp per row reading keys where they lie, and now, in us.  32-bit, 14 heads of 64 over 2: 301 tokens 265 and 43, one token
// at 300 keys 127 and 24, 64 at 1,000 518 and 68; 16 heads of 64 over 16: 250 single tokens at 1,000 keys 1,248 and 426, 10 of them at
// 2,000 beside 250 prompt tokens 1,412 and 208; 16 of 128 over 16: 1,500 tokens 9,560 and 742.  bf16, 16 of 36 over 16: 250 single
// tokens 523 and 308.  (A chunk ahead is enough: two or three ahead made blocks too large, 707 instead of 428 for the 250 of 64.)
#include "common.cuh"
#include <math_constants.h>

extern "C" int infero_sm_count();

namespace {

constexpr int WARPS = 8;
constexpr int MAX_D = 256;
constexpr int CHUNK = 32, STAGES = 2;
constexpr int FEW_TOKENS = 256;         // portions of up to so many tokens: a block per token, one row a warp; beyond, 32 or 16 rows a block
constexpr int WIDE_ROWS = WARPS * 4;

struct GenericArgs {
    const void* q;
    void* out;
    const void* k_cache;
    const void* v_cache;
    const int* block_table;
    const int* tok_entry;
    const int* positions;
    const float* slopes;
    const float* rel;
    const float* sinks;
    int q_stride, out_stride, max_blocks, n_tokens, n_heads, n_kv, head_dim, value_dim, page_size, window, sink, rel_len, cross;
    int tokens_per_block, head_chunks, tiles, singles;   // tiles: blocks of one kv head; singles: tokens in front with a block each
    float scale, softcap;
};

// Elements between rows of keys (an odd multiple of four: lanes read four elements of neighbouring rows each without bank conflicts)
// and of values.
__host__ __device__ inline int key_stride(int head_dim) { return (((head_dim + 3) / 4) | 1) * 4; }
__host__ __device__ inline int value_stride(int value_dim) { return (value_dim + 3) / 4 * 4; }

// VEC: rows of whole pieces of four elements, 16 bytes of 32-bit or 8 of bf16, stay in their type in shared memory; other rows are
// widened to 32-bit element by element.
template <typename T, bool VEC> struct Stored { using type = float; };
template <> struct Stored<bf16, true> { using type = bf16; };

template <typename S>
inline size_t generic_smem(int head_dim, int value_dim, int rows) {
    return (size_t)STAGES * CHUNK * (key_stride(head_dim) + value_stride(value_dim)) * sizeof(S) +
           (STAGES + (size_t)rows * ((head_dim + 3) / 4 * 4 + CHUNK)) * sizeof(float);
}

__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four(const bf16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// The pieces (VEC: four elements; else one) of a row, and what divides by their number.
struct Pieces { int per; unsigned int inverse; };
template <bool VEC> __device__ __forceinline__ Pieces pieces_of(int width) {
    const int per = VEC ? width / 4 : (width + 3) / 4 * 4;
    return {per, 0xffffffffu / per + 1};                 // (exact for numbers below 2^32 / per; 0 for one piece a row)
}

// A chunk's rows of one array into shared memory, zeros where there is none; lane r brings the place of row r (or -1).  Neighbouring
// lanes take neighbouring pieces, whichever row they are of, and a warp every n_warps-th 32 of them.  (A row at a time left half of the
// lanes of a 256-byte row idle and took 240 cycles a row in one chain: all of the time of a block with one warp.)
template <typename T, bool VEC, typename S>
__device__ __forceinline__ void fetch(S* dst, int stride, const T* cache, int width, const Pieces p, long long row, int warp, int n_warps, int lane) {
#pragma unroll 4
    for (int i = warp; i < p.per; i += n_warps) {
        const int e = i * 32 + lane, r = p.per == 1 ? e : (int)__umulhi((unsigned)e, p.inverse), c = (e - r * p.per) * (VEC ? 4 : 1);
        const long long at = __shfl_sync(0xffffffffu, row, r);
        if constexpr (VEC) {
            const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst + r * stride + c);
            const T* src = at < 0 ? cache : cache + at * width + c;
            if constexpr (sizeof(T) == 4)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(at < 0 ? 0 : 16) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(at < 0 ? 0 : 8) : "memory");
        } else {
            dst[r * stride + c] = at >= 0 && c < width ? to_f32(__ldg(cache + at * width + c)) : 0.f;
        }
    }
}

template <typename T, typename TO, int R, int COLS, bool VEC>
__global__ void __launch_bounds__(WARPS * 32)
attention_generic_kernel(const GenericArgs a) {
    using S = typename Stored<T, VEC>::type;
    extern __shared__ float4 smem4[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const int D = a.head_dim, V = a.value_dim, D4 = (D + 3) / 4 * 4, ks = key_stride(D), vs = value_stride(V);
    S* k_s = reinterpret_cast<S*>(smem4);                // [STAGES][CHUNK][ks]
    S* v_s = k_s + STAGES * CHUNK * ks;                  // [STAGES][CHUNK][vs]
    float* rows_s = reinterpret_cast<float*>(v_s + STAGES * CHUNK * vs);
    float* q_s = rows_s + warp * R * D4;                 // this warp's [R][D4]
    float* p_s = rows_s + n_warps * R * D4 + warp * R * CHUNK;
    unsigned int* here = reinterpret_cast<unsigned int*>(rows_s + n_warps * R * (D4 + CHUNK));   // a bit per key
    const Pieces k_pieces = pieces_of<VEC>(D), v_pieces = pieces_of<VEC>(V);
    const int group = a.n_heads / a.n_kv;
    const int side = blockIdx.x / a.tiles, tile = blockIdx.x % a.tiles;
    const int kvh = a.cross ? side / a.n_kv : side, vh = a.cross ? side % a.n_kv : kvh;
    const int at = tile / a.head_chunks, g0 = tile % a.head_chunks * (n_warps * R);
    const int t0 = at < a.singles ? at : a.singles + (at - a.singles) * a.tokens_per_block;
    const int t1 = at < a.singles ? t0 + 1 : min(a.n_tokens, t0 + a.tokens_per_block);
    const int heads = a.head_chunks > 1 ? min(group - g0, n_warps * R) : group;

    int tok[R], head[R], pos[R], lo[R];
    float m[R], l[R], slope[R], acc[R][COLS];
    const T* q = (const T*)a.q;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = warp * R + r;
        tok[r] = t0 + i / heads;
        head[r] = kvh * group + g0 + i % heads;
        const bool mine = tok[r] < t1;
        pos[r] = mine ? a.positions[tok[r]] : -1;
        lo[r] = a.window > 0 ? max(0, pos[r] - a.window + 1) : 0;
        if (!mine) tok[r] = -1;
        slope[r] = mine && a.slopes ? a.slopes[head[r]] : 0.f;
        // a sink is one more term of the softmax's sum, with score 0 and no value: the running maximum and sum start
        // as if that key had been seen (with learned sinks its score is the head's own number)
        m[r] = a.sink ? 0.f : mine && a.sinks ? a.sinks[head[r]] : -CUDART_INF_F;
        l[r] = a.sink || a.sinks ? 1.f : 0.f;
#pragma unroll
        for (int i2 = 0; i2 < COLS; ++i2) acc[r][i2] = 0.f;
        for (int d = lane; d < D4; d += 32)
            q_s[r * D4 + d] = mine && d < D ? to_f32(q[(size_t)tok[r] * a.q_stride + (size_t)head[r] * D + d]) : 0.f;
    }
    __syncwarp();

    for (int first = t0; first < t1;) {                  // the tokens of one request after the other
        const int entry = a.tok_entry[first];
        const int* table = a.block_table + (size_t)entry * a.max_blocks;
        int end = first, start = 0x7fffffff, last = -1;
        for (; end < t1 && a.tok_entry[end] == entry; ++end) {
            const int p = a.positions[end];
            last = max(last, p);
            start = min(start, a.window > 0 ? max(0, p - a.window + 1) : 0);
        }
        auto page_of = [&](int j0) {                     // of this lane's key in a chunk, -1 if there is none
            const int j = j0 + lane;
            return j <= last ? table[j / a.page_size] : -1;
        };
        auto load = [&](int j0, int page, int stage) {
            if (j0 <= last) {
                const long long row = page < 0 ? -1 : ((long long)page * a.n_kv + kvh) * a.page_size + (j0 + lane) % a.page_size;
                const unsigned int there = __ballot_sync(0xffffffffu, page >= 0);
                if (threadIdx.x == 0) here[stage] = there;
                fetch<T, VEC>(k_s + stage * CHUNK * ks, ks, (const T*)a.k_cache, D, k_pieces, row, warp, n_warps, lane);
                fetch<T, VEC>(v_s + stage * CHUNK * vs, vs, (const T*)a.v_cache, V, v_pieces,
                              page < 0 ? -1 : row + (long long)(vh - kvh) * a.page_size, warp, n_warps, lane);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        start = start / CHUNK * CHUNK;
        load(start, page_of(start), 0);
        int page = page_of(start + CHUNK), stage = 0;
        for (int j0 = start; j0 <= last; j0 += CHUNK, stage ^= 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();                             // this chunk is here, and everyone is done with the one before,
            load(j0 + CHUNK, page, stage ^ 1);           // whose place this takes
            page = page_of(j0 + 2 * CHUNK);
            const int j = j0 + lane;
            const bool there = here[stage] >> lane & 1;
            bool sees[R];                                // does the row have keys in this chunk?
            bool any = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                sees[r] = tok[r] >= first && tok[r] < end && j0 <= pos[r] && j0 + CHUNK > lo[r];
                any |= sees[r];
            }
            if (any) {
                float d[R];
#pragma unroll
                for (int r = 0; r < R; ++r) d[r] = 0.f;
                const S* kr = k_s + (stage * CHUNK + lane) * ks;
#pragma unroll 8
                for (int i = 0; i < D4; i += 4) {        // (columns beyond D are zeros on both sides)
                    const float4 k = four(kr + i);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 x = *reinterpret_cast<const float4*>(q_s + r * D4 + i);
                        d[r] = fmaf(x.x, k.x, d[r]);
                        d[r] = fmaf(x.y, k.y, d[r]);
                        d[r] = fmaf(x.z, k.z, d[r]);
                        d[r] = fmaf(x.w, k.w, d[r]);
                    }
                }
                int from = CHUNK, to = -1;               // the values some row of this warp takes
                bool whole = true;                       // every row takes all of them
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool valid = sees[r] && there && j >= lo[r] && j <= pos[r];
                    float s = -CUDART_INF_F;
                    if (valid) {
                        s = d[r] * a.scale;
                        if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
                        s -= slope[r] * (float)(pos[r] - j);
                        if (a.rel) s += a.rel[(size_t)head[r] * a.rel_len + min(pos[r] - j, a.rel_len - 1)];
                    }
                    const float m_new = fmaxf(m[r], warp_max(s));
                    if (m_new == -CUDART_INF_F) sees[r] = false;      // no readable key in this chunk
                    float p = 0.f;
                    if (sees[r]) {
                        p = valid ? expf(s - m_new) : 0.f;
                        const float corr = expf(m[r] - m_new);        // first chunk: exp(-inf) = 0
                        l[r] = l[r] * corr + warp_sum(p);
#pragma unroll
                        for (int i = 0; i < COLS; ++i) acc[r][i] *= corr;
                        m[r] = m_new;
                        from = min(from, max(lo[r] - j0, 0)), to = max(to, min(pos[r] - j0, CHUNK - 1));
                    }
                    whole &= sees[r] && j0 >= lo[r] && j0 + CHUNK - 1 <= pos[r];
                    p_s[r * CHUNK + lane] = p;
                }
                __syncwarp();
                const S* vr = v_s + stage * CHUNK * vs + lane;
                if (whole) {
#pragma unroll
                    for (int jj = 0; jj < CHUNK; jj += 4) {
                        float4 p4[R];
#pragma unroll
                        for (int r = 0; r < R; ++r) p4[r] = *reinterpret_cast<const float4*>(p_s + r * CHUNK + jj);
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
#pragma unroll
                            for (int i = 0; i < COLS; ++i) {
                                const float v = i * 32 + lane < V ? to_f32(vr[(jj + u) * vs + i * 32]) : 0.f;
#pragma unroll
                                for (int r = 0; r < R; ++r) acc[r][i] = fmaf(reinterpret_cast<const float*>(&p4[r])[u], v, acc[r][i]);
                            }
                        }
                    }
                } else {
                    for (int jj = from; jj <= to; ++jj) {
                        float v[COLS];
#pragma unroll
                        for (int i = 0; i < COLS; ++i) v[i] = i * 32 + lane < V ? to_f32(vr[jj * vs + i * 32]) : 0.f;
#pragma unroll
                        for (int r = 0; r < R; ++r) {    // (a key that a row must not see is not even multiplied by zero)
                            if (!sees[r] || j0 + jj < lo[r] || j0 + jj > pos[r]) continue;
                            const float p = p_s[r * CHUNK + jj];
#pragma unroll
                            for (int i = 0; i < COLS; ++i) acc[r][i] = fmaf(p, v[i], acc[r][i]);
                        }
                    }
                }
                __syncwarp();
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                 // the next request's chunks take the same places
        first = end;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (tok[r] < 0) continue;
        const int at = a.cross ? vh * a.n_heads + head[r] : head[r];
        TO* orow = (TO*)a.out + (size_t)tok[r] * a.out_stride + (size_t)at * V;
        const float inv = 1.0f / l[r];
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
            const int dd = i * 32 + lane;
            if (dd < V) orow[dd] = from_f32<TO>(acc[r][i] * inv);
        }
    }
}

template <typename T, typename TO, int R, int COLS, bool VEC>
int launch(GenericArgs& a, int warps, cudaStream_t stream) {
    auto* kernel = attention_generic_kernel<T, TO, R, COLS, VEC>;
    const size_t smem = generic_smem<typename Stored<T, VEC>::type>(a.head_dim, a.value_dim, warps * R);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        INFERO_REQUIRE(e == cudaSuccess, "attention: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    }
    const long long tiles = (a.singles + (long long)(a.n_tokens - a.singles + a.tokens_per_block - 1) / a.tokens_per_block) * a.head_chunks;
    const long long blocks = tiles * a.n_kv * (a.cross ? a.n_kv : 1);
    INFERO_REQUIRE(blocks < (1ll << 31), "attention: %d tokens of %d kv heads are too many for one launch", a.n_tokens, a.n_kv);
    a.tiles = (int)tiles;
    kernel<<<(unsigned)blocks, warps * 32, smem, stream>>>(a);
    return infero_check_launch("attention_generic");
}

// Tokens a block of 32 rows takes at a time (launch_rows may halve them), 0 for a block per token.  A block's tokens of different requests take turns and all but
// one request's rows idle meanwhile, so what counts is the portions' tokens (the single ones in front have blocks of their own
// either way) and that a portion has about a block's tokens and more.
int block_tokens(int n_tokens, int singles, int portions, int group) {
    const int rest = n_tokens - singles, tokens = group > WIDE_ROWS ? 1 : WIDE_ROWS / group;
    return rest <= FEW_TOKENS || 2 * rest < (long long)portions * tokens ? 0 : tokens;
}

// Blocks of 16 rows that a multiprocessor holds.
template <typename T, typename TO, bool VEC>
int resident_half(int head_dim, int value_dim) {
    const size_t smem = generic_smem<typename Stored<T, VEC>::type>(head_dim, value_dim, WIDE_ROWS / 2);
    auto ask = [&](auto* kernel) {
        int n = 0;
        if ((smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, WARPS * 32, smem) != cudaSuccess)
            n = 0, cudaGetLastError();
        return n;
    };
    return head_dim > 128 || value_dim > 128 ? ask(attention_generic_kernel<T, TO, 2, 8, VEC>) : value_dim > 64 ? ask(attention_generic_kernel<T, TO, 2, 4, VEC>)
                                                                                              : ask(attention_generic_kernel<T, TO, 2, 2, VEC>);
}

template <typename T, typename TO, bool VEC>
int launch_rows(GenericArgs& a, int portions, cudaStream_t stream) {
    const int group = a.n_heads / a.n_kv, tokens = block_tokens(a.n_tokens, a.singles, portions, group);
    const bool few = tokens == 0;
    // (warps without a row help to fetch: four suffice for narrow rows)
    const int least = a.head_dim > 64 || a.value_dim > 64 ? WARPS : WARPS / 2;
    const int warps = few ? (group < least ? least : group < WARPS ? group : WARPS) : WARPS;
    // Where blocks of 32 rows are fewer than two a multiprocessor, half as many rows a warp: what a chunk costs a warp is latency, and
    // twice the warps cover it, as long as all the blocks run at once: they fetch a key up to three times as often, and a second wave takes
    // as long as the first.  (us in blocks of 32 rows and of 16, 32-bit, 301 tokens: 14 heads of 64 over 2, 302 blocks of 16, 62 and 43,
    // behind 1,500 cached ones 385 and 244; 16 of 64 over 1, 301 blocks of the 444 that fit, 289 and 252; 18 of 64 over 2, 602 blocks, 400 and 446,
    // without cached ones 69 and 61; 9 of 128 over 1, 301 of 296, 455 and 546, without 82 and 60, 270 tokens behind 2,000 570 and 396.)
    const long long sides = (long long)a.n_kv * (a.cross ? a.n_kv : 1), rest = a.n_tokens - a.singles;
    auto blocks = [&](int rows) {
        const int each = group > rows ? 1 : rows / group;
        return (a.singles + (rest + each - 1) / each) * ((group + rows - 1) / rows) * sides;
    };
    const int sms = infero_sm_count(), half_rows = WIDE_ROWS / 2;
    bool half = !few && blocks(WIDE_ROWS) < 2 * sms;
    if (half) half = blocks(half_rows) <= (long long)sms * resident_half<T, TO, VEC>(a.head_dim, a.value_dim);
    const int rows = few ? warps : half ? half_rows : WIDE_ROWS;
    a.tokens_per_block = few ? 1 : half ? (group > rows ? 1 : rows / group) : tokens;
    a.head_chunks = (group + rows - 1) / rows;
#define COLUMNS(R)                                                                                      \
    do {                                                                                                \
        if (a.head_dim > 128 || a.value_dim > 128) return launch<T, TO, R, 8, VEC>(a, warps, stream);   \
        if (a.value_dim > 64) return launch<T, TO, R, 4, VEC>(a, warps, stream);                        \
        return launch<T, TO, R, 2, VEC>(a, warps, stream);                                              \
    } while (0)
    if (few) COLUMNS(1);
    if (half) COLUMNS(2);
    COLUMNS(4);
#undef COLUMNS
}

}  // namespace

extern "C" {

int infero_attention_generic_block_tokens(int n_tokens, int singles, int portions, int group) {
    return block_tokens(n_tokens, singles, portions, group);
}

// Keys of width head_dim, values of width value_dim (the cache's two arrays have their own row widths); ``sink``:
// the softmax's denominator has one more term exp(0), which carries no value; ``slopes``: float32 [n_heads] or null,
// head h's score loses slopes[h] times the distance between the query and the key; ``rel``: float32 [n_heads, rel_len] or
// null, what a score gains at every distance (the last entry also beyond it); ``cross``: every head meets the values of
// every kv head, out float32 [n_tokens, n_heads * n_kv * value_dim]; ``sinks``: float32 [n_heads] or null, one more term
// exp(sinks[h]) of the denominator; ``softcap`` > 0: scaled scores are soft-capped; ``singles`` tokens in front are their requests'
// only ones and ``portions`` requests bring the others (they choose the blocks and change no result).
int infero_attention_generic_rel(const void* q, int q_stride, void* out, int out_stride, const void* k_cache,
                                 const void* v_cache, int dtype, const int* block_table, int max_blocks,
                                 const int* tok_entry, const int* positions, int n_tokens, int n_heads,
                                 int n_kv, int head_dim, int value_dim, int page_size, int window, float scale,
                                 int sink, const float* slopes, const float* rel, int rel_len, int cross,
                                 const float* sinks, float softcap, int singles, int portions, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    INFERO_REQUIRE(singles >= 0 && singles <= n_tokens && portions >= 0, "attention: %d single tokens and %d portions of %d tokens", singles,
                   portions, n_tokens);
    INFERO_REQUIRE(head_dim >= 1 && head_dim <= MAX_D, "attention: head_dim %d outside 1..%d", head_dim, MAX_D);
    INFERO_REQUIRE(value_dim >= 1 && value_dim <= MAX_D, "attention: value width %d outside 1..%d", value_dim, MAX_D);
    INFERO_REQUIRE(n_kv > 0 && n_heads % n_kv == 0, "attention: %d heads not a multiple of %d kv heads", n_heads, n_kv);
    INFERO_REQUIRE(!rel || rel_len >= 1, "attention: an empty table of distances");
    GenericArgs a;
    a.q = q, a.out = out, a.k_cache = k_cache, a.v_cache = v_cache, a.block_table = block_table, a.tok_entry = tok_entry;
    a.positions = positions, a.slopes = slopes, a.rel = rel, a.sinks = sinks, a.q_stride = q_stride, a.out_stride = out_stride;
    a.max_blocks = max_blocks, a.n_tokens = n_tokens, a.n_heads = n_heads, a.n_kv = n_kv, a.head_dim = head_dim;
    a.value_dim = value_dim, a.page_size = page_size, a.window = window, a.sink = sink, a.rel_len = rel_len, a.cross = cross;
    a.scale = scale, a.softcap = softcap, a.singles = singles;
    const size_t piece = dtype == INFERO_F32 ? 16 : 8;
    const bool vec = head_dim % 4 == 0 && value_dim % 4 == 0 && (uintptr_t)k_cache % piece == 0 && (uintptr_t)v_cache % piece == 0;
    if (dtype == INFERO_F32) return vec ? launch_rows<float, float, true>(a, portions, stream) : launch_rows<float, float, false>(a, portions, stream);
    if (cross) return vec ? launch_rows<bf16, float, true>(a, portions, stream) : launch_rows<bf16, float, false>(a, portions, stream);
    return vec ? launch_rows<bf16, bf16, true>(a, portions, stream) : launch_rows<bf16, bf16, false>(a, portions, stream);
}

int infero_attention_generic_bias(const void* q, int q_stride, void* out, int out_stride, const void* k_cache,
                                  const void* v_cache, int dtype, const int* block_table, int max_blocks,
                                  const int* tok_entry, const int* positions, int n_tokens, int n_heads,
                                  int n_kv, int head_dim, int value_dim, int page_size, int window, float scale,
                                  int sink, const float* slopes, cudaStream_t stream) {
    return infero_attention_generic_rel(q, q_stride, out, out_stride, k_cache, v_cache, dtype, block_table, max_blocks,
                                        tok_entry, positions, n_tokens, n_heads, n_kv, head_dim, value_dim, page_size,
                                        window, scale, sink, slopes, nullptr, 0, 0, nullptr, 0.f, 0, 1, stream);
}

int infero_attention_generic_ex(const void* q, int q_stride, void* out, int out_stride, const void* k_cache,
                                const void* v_cache, int dtype, const int* block_table, int max_blocks,
                                const int* tok_entry, const int* positions, int n_tokens, int n_heads,
                                int n_kv, int head_dim, int value_dim, int page_size, int window, float scale,
                                int sink, cudaStream_t stream) {
    return infero_attention_generic_bias(q, q_stride, out, out_stride, k_cache, v_cache, dtype, block_table, max_blocks,
                                         tok_entry, positions, n_tokens, n_heads, n_kv, head_dim, value_dim, page_size,
                                         window, scale, sink, nullptr, stream);
}

int infero_attention_generic(const void* q, int q_stride, void* out, int out_stride, const void* k_cache,
                             const void* v_cache, int dtype, const int* block_table, int max_blocks,
                             const int* tok_entry, const int* positions, int n_tokens, int n_heads,
                             int n_kv, int head_dim, int page_size, int window, float scale,
                             cudaStream_t stream) {
    return infero_attention_generic_ex(q, q_stride, out, out_stride, k_cache, v_cache, dtype, block_table, max_blocks,
                                       tok_entry, positions, n_tokens, n_heads, n_kv, head_dim, head_dim, page_size,
                                       window, scale, 0, stream);
}

}  // extern "C"
