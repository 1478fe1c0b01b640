// All layers of a decode step of few tokens in one resident kernel.
//
// A step of a handful of single tokens is bound by reading the weights once, but as a chain of launches (five to eight a layer)
// every kernel starts its stream of weights anew: about 3.5 us of a launch, a wait and an empty ring each, during which the
// memory system idles.  Here one block per multiprocessor stays for the whole step.  One warp of it (the loader) knows the
// order in which the block will want its bytes, for all products and all attention of all layers, and keeps a ring of shared
// memory filled with them through the bulk-copy engine, ahead of everything that the other warps wait for.  What the phases of a
// layer (q/k/v, attention, output, gate/up, down) hand to one another goes through tagged words in global memory (below), without
// a barrier; meanwhile the ring fills with the weights of the phases behind it.
//
//   products   Every block has an equal share of a matrix's rows, and all of K: no partial sums leave a block.  Rows come eight
//              at a time (a unit), K in pieces of 896 columns; a unit's piece is one slot of the ring, a bulk
//              copy a row.  The seven consumer
//              warps share a slot's columns, 32 at a time in turns, on mma.sync m16n8k16 (rows of A: two units, columns of B: the
//              tokens); their sums meet in shared memory, in warp order.  A lane reads 16 bytes of a weight row and 16 of
//              an activation row and takes them for two k-steps (k is permuted alike on both sides, so no ldmatrix is needed).
//              tcgen05 would want 128 rows of one block; a block's share here is 6 to 256 rows, and the bound is memory.
//   attention  The keys of all (token, kv head) pairs lie on one line, in slices of 16, and every block takes an equal piece of
//              it, so requests of any lengths keep all blocks busy; pieces are whole multiples of 112 keys while there are
//              few.  Slices come through the same ring (TMA, 128-byte swizzle), a slot to a warp.  A block adds up its warps'
//              results, and the block that arrives last for a pair merges the blocks'.
//   norms      The block that owns a column of the residual stream keeps it in shared memory in 32 bits; it hands on
//              bf16(x * w) and its columns' sum of squares, and the product behind applies 1 / rms to its 32-bit results.
//
// A step of one token at 300 keys, 24 layers of Qwen2.5-0.5B sizes, as one pass of a runner: 694 us as 195 launches, 584 so (0.15 ms of
// bytes; infero_resident_worth has more lengths and sizes, as replays of the captured step alone).  What bounds it are five phases a
// layer that each wait for the one before, a store and a load through L2 and a few rows of work a block.
// Every wait has a time limit: a wait that runs out raises the error flag and every block runs to its end without waiting.
// The reference's counterpart of the step: crates/model/src/lib.rs:3423-4243.
#include "attn_common.cuh"
#include "tc_common.cuh"
#include "decode_resident.h"

#include <algorithm>
#include <mutex>

extern "C" int infero_sm_count();

namespace {

using namespace attn;

constexpr int CW = 7, CT = CW * 32, THREADS = CT + 32;          // consumer warps, their threads, all threads (eight warps: 255 registers)
constexpr int TOKENS = 2;                                       // tokens a step may have (a product has room for eight columns)
constexpr int PIECE = 896;                                      // columns of a weight piece: four steps of 32 for each warp
constexpr int ROW_BYTES = PIECE * 2 + 64;                       // rows in a slot start 64 bytes apart mod 128: no bank conflicts
constexpr int SLOT = 15360, SLOTS = 10;                         // bytes and number of ring slots
constexpr int STEPS = (PIECE / 32 + CW - 1) / CW;               // k-steps of 32 columns a warp has in a piece, at most
constexpr int UNITS = 8;                                        // units a warp accumulates at a time
constexpr int RED_BYTES = CW * 8 * 68 * 4;                      // the warps' sums, or 64 columns of their attention results
constexpr int ACT_BYTES = 44 * 1024;                            // a product's activations in shared memory
constexpr int MAX_ROWS = 64;                                    // columns of the residual stream one block owns, at most
constexpr int GROUP = 8;                                        // query heads of a kv head, at most
static_assert(8 * ROW_BYTES <= SLOT && SLOT % 1024 == 0 && CW * UNITS * 8 * 8 * 4 <= RED_BYTES && GROUP == 8, "");

struct Smem {                                                   // offsets behind the ring (from a 1,024-byte boundary)
    static constexpr int RED = SLOT * SLOTS;
    static constexpr int ACT = RED + RED_BYTES;                 // [tokens][K] bf16
    static constexpr int X = ACT + ACT_BYTES;                   // [TOKENS][MAX_ROWS] float
    static constexpr int ANGLES = X + TOKENS * MAX_ROWS * 4;    // [64] float2
    static constexpr int Q = ANGLES + 64 * 8;                   // [GROUP][D + 8] bf16
    static constexpr int KV = Q + GROUP * 136 * 2;              // the token's own key and value [2][D] bf16
    static constexpr int ML = KV + 2 * 128 * 2;                 // [CW][GROUP] float2
    static constexpr int MISC = ML + CW * GROUP * 8;            // rms, positions, entries [8] each; abort; [28] last to arrive
    static constexpr int BARS = MISC + 32 * 4;                  // full[SLOTS], empty[SLOTS]
    static constexpr int TOTAL = BARS + 2 * SLOTS * 8 + 1024;
};
static_assert(Smem::TOTAL <= 232448, "");
static_assert(Smem::BARS % 8 == 0 && Smem::X % 16 == 0 && Smem::Q % 16 == 0 && Smem::KV % 16 == 0, "");

struct alignas(64) Params {
    CUtensorMap k_map[RESIDENT_LAYERS], v_map[RESIDENT_LAYERS];
    ResidentLayer layer[RESIDENT_LAYERS];
    ResidentStep s;
    int* err_flag;
};

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CT) : "memory"); }
__device__ __forceinline__ int share(int i, int n, int parts) { return (int)((long long)i * n / parts); }
__device__ __forceinline__ uint4 ld_l2_16(const void* p) {      // written by other blocks a moment ago: not through L1
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(tc::smem_u32(bar)), "l"(policy) : "memory");
}
// (a read where it stands, behind the wait for its slot; 32-bit addresses)
__device__ __forceinline__ uint4 lds16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}

// ---- values that carry a tag --------------------------------------------------------------------------------------------------
// What one block hands to the others needs no meeting.  Every value lies in a word of its own beside a tag (bf16 with 16 bits of
// tag, 32-bit values with 32), the number of the layer that will read it, and a reader looks at the word until the tag is there: a
// store and a load on the way, instead of a fence, a counter (4 to 6 thousand cycles a phase, measured) and then the load.
// The step's first kernel clears all tags.  No word is written again before all have read it: a block writes its
// words of a phase after it has read everything of the phase before, and every block has words of gate/up in every layer.
__device__ __forceinline__ uint4 look16(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// (a 32-bit value and its tag are one access of 64 bits: a vector of two would be two accesses in no order)
__device__ __forceinline__ uint2 look8(const uint2* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return make_uint2((unsigned)v, (unsigned)(v >> 32));
}
__device__ __forceinline__ uint32_t tagged(float v, uint32_t tag) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v)) | tag << 16;
}
__device__ __forceinline__ void tell(uint32_t* p, uint32_t word) { asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(word) : "memory"); }
__device__ __forceinline__ void tell(uint2* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((unsigned long long)tag << 32 | __float_as_uint(v)) : "memory");
}

// ---- who takes which keys ------------------------------------------------------------------------------------------------
// Token t's keys are `slices(t)` slices of 16 from slice `first(t)` on.  On the line every (token, kv head) pair has its slices
// rounded up to a multiple of `unit`; block b takes [b * per, (b + 1) * per).  While every seven slices (112 keys, one for each
// warp) can have a block of their own, unit = per = 7: a block then has one piece of one pair.
struct Line {
    int unit, per;
};
struct Keys {
    const int* pos;
    int n_tok, window;
    __device__ __forceinline__ int first(int t) const { return window > 0 ? max(0, pos[t] - window + 1) / KEYS16 : 0; }
    __device__ __forceinline__ int slices(int t) const { return pos[t] < 0 ? 0 : pos[t] / KEYS16 - first(t) + 1; }
    __device__ __forceinline__ Line line(int n_kv, int blocks) const {
        int rounds = 0, all = 0;
        for (int t = 0; t < n_tok; ++t) {
            const int n = slices(t);
            rounds += (n + CW - 1) / CW, all += n;
        }
        return rounds * n_kv <= blocks ? Line{CW, CW} : Line{1, (all * n_kv + blocks - 1) / blocks};
    }
};
struct Segment {
    int token, kvh, pair;           // pair: token * n_kv + kv head
    int s0, s1;                     // slices of the token
    int first, last;                // the blocks that have pieces of this pair
};
// f(segment) for each of block b's pieces, in order
template <typename F>
__device__ __forceinline__ void for_segments(const Keys& keys, const Line line, int n_kv, int b, F f) {
    const int c0 = b * line.per, c1 = c0 + line.per;
    for (int t = 0, off = 0; t < keys.n_tok; ++t) {
        const int n = keys.slices(t), len = (n + line.unit - 1) / line.unit * line.unit;
        if (len > 0 && off < c1 && off + len * n_kv > c0) {
            for (int h = max(0, c0 - off) / len; h < n_kv && off + h * len < c1; ++h) {
                const int base = off + h * len, s0 = max(0, c0 - base), s1 = min(n, c1 - base);
                if (s0 < s1) f(Segment{t, h, t * n_kv + h, s0, s1, base / line.per, (base + n - 1) / line.per});
            }
        }
        off += len * n_kv;
    }
}
// Slices a slot takes: one for each warp before any gets a second, then what fits.
template <int D>
__device__ __forceinline__ int slices_per_slot(int n) {
    constexpr int MOST = SLOT / (64 * D) < 4 ? SLOT / (64 * D) : 4;     // a slice is 16 keys and values of D bf16
    return min(MOST, max(1, (n + CW - 1) / CW));
}

// The blocks' results of a pair, merged in their order.
template <int D>
__device__ __forceinline__ void merge(const ResidentStep& s, const Segment g, uint32_t tag) {
    const int group = s.n_heads / s.n_kv, h0 = g.kvh * group, t = g.token, n = g.last - g.first + 1;
    const float* po0 = s.part_o + (size_t)(g.first + g.pair) * (GROUP * D);
    const float* ml0 = s.part_ml + (size_t)(g.first + g.pair) * (GROUP * 2);
    for (int e = threadIdx.x; e < group * (D / 4); e += CT) {
        const int r = e / (D / 4), d = (e - r * (D / 4)) * 4;
        float M = -CUDART_INF_F, sum = 0.f, v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < n; k0 += 8) {                     // eight blocks' loads in flight at a time
            float2 x[8];
            uint4 y[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k0 + k < n) {
                    x[k] = __ldcg(reinterpret_cast<const float2*>(ml0 + (size_t)(k0 + k) * (GROUP * 2)) + r);
                    y[k] = ld_l2_16(po0 + (size_t)(k0 + k) * (GROUP * D) + r * D + d);
                }
            float Mn = M;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k0 + k < n) Mn = fmaxf(Mn, x[k].x);
            const float fix = M == -CUDART_INF_F ? 0.f : exp2f(M - Mn);
            M = Mn, sum *= fix, v[0] *= fix, v[1] *= fix, v[2] *= fix, v[3] *= fix;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k0 + k < n && x[k].x != -CUDART_INF_F) {
                    const float w = exp2f(x[k].x - M);
                    sum = fmaf(x[k].y, w, sum);
                    v[0] = fmaf(__uint_as_float(y[k].x), w, v[0]), v[1] = fmaf(__uint_as_float(y[k].y), w, v[1]);
                    v[2] = fmaf(__uint_as_float(y[k].z), w, v[2]), v[3] = fmaf(__uint_as_float(y[k].w), w, v[3]);
                }
        }
        const float inv = 1.0f / sum;
        const size_t to = ((size_t)t * s.n_heads + h0 + r) * D + d;
#pragma unroll
        for (int k = 0; k < 4; ++k) tell(s.attn + to + k, tagged(v[k] * inv, tag));
    }
}

template <int D>
struct Block {
    const Params& p;
    uint8_t* smem;
    uint64_t *full, *empty;
    int *pos, *entries;             // of the step's tokens
    volatile int* abort_flag;       // a wait ran out
    float* red;
    float* x_s;
    float* rms;
    int warp, lane;
    uint32_t seq;                   // slots of the ring passed so far

    __device__ __forceinline__ Block(const Params& params, uint8_t* at, uint32_t passed = 0)
        : p(params), smem(at), full(reinterpret_cast<uint64_t*>(at + Smem::BARS)), empty(full + SLOTS),
          pos(reinterpret_cast<int*>(at + Smem::MISC) + 8), entries(pos + 8), abort_flag(pos + 16),
          red(reinterpret_cast<float*>(at + Smem::RED)), x_s(reinterpret_cast<float*>(at + Smem::X)), rms(reinterpret_cast<float*>(at + Smem::MISC)),
          warp(threadIdx.x >> 5), lane(threadIdx.x & 31), seq(passed) {}
    __device__ __forceinline__ const ResidentStep& s() const { return p.s; }

    // A wait that looks at the clock late: reading it takes about as long as a slot's work.
    __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) {
        unsigned long long t0 = 0;
        for (unsigned int i = 1;; ++i) {
            if (tc::mbar_try_wait(bar, parity)) return true;
            if ((i & 255u) == 0) {
                if (*abort_flag) return false;
                const unsigned long long now = tc::global_ns();
                if (!t0) t0 = now;
                if (now - t0 > tc::WAIT_LIMIT_NS) return false;
            }
        }
    }
    // Nobody waits any more: the block runs through the rest of the step with whatever is there, as the other blocks do.
    __device__ __forceinline__ void give_up() {
        *abort_flag = 1;
        *(volatile unsigned int*)s().stop = 1;
        atomicExch(p.err_flag, 10);
    }
    // The bytes of the ring's q-th slot are here.
    __device__ __forceinline__ void arrived(uint32_t q) {
        if (!wait(&full[q % SLOTS], (q / SLOTS) & 1u)) give_up();
    }
    // look() until it is true or the time is up
    template <typename F>
    __device__ __forceinline__ void until(F look) {
        unsigned long long t0 = 0;
        for (unsigned int i = 1; !look(); ++i) {
            if (*abort_flag) return;
            if ((i & 63u) == 0) {
                if (!t0) t0 = tc::global_ns();
                if (tc::global_ns() - t0 > tc::WAIT_LIMIT_NS || *(volatile unsigned int*)s().stop) give_up();
            }
        }
    }

    // ---- the loader ------------------------------------------------------------------------------------------------------
    __device__ __forceinline__ bool acquire() {                 // the slot `seq` is free
        return seq < SLOTS || wait(&empty[seq % SLOTS], (seq / SLOTS - 1) & 1u);
    }
    __device__ __forceinline__ bool load_matrix(const bf16* w, int r0, int r1, int K, uint64_t policy) {
        const int units = (r1 - r0 + 7) / 8, groups = (units + UNITS - 1) / UNITS, per = groups ? (units + groups - 1) / groups : 0;
        for (int u0 = 0; u0 < units; u0 += per)
            for (int k0 = 0; k0 < K; k0 += PIECE) {
                const int bytes = min(PIECE, K - k0) * 2;
                for (int u = u0; u < min(units, u0 + per); ++u, ++seq) {
                    if (!acquire()) return false;
                    const int rows = min(8, r1 - r0 - u * 8);
                    uint64_t* bar = &full[seq % SLOTS];
                    if (lane == 0) tc::mbar_expect_tx(bar, rows * bytes);
                    __syncwarp();
                    if (lane < rows)
                        bulk_load(tc::smem_u32(smem) + (seq % SLOTS) * SLOT + lane * ROW_BYTES, w + (size_t)(r0 + u * 8 + lane) * K + k0, bytes, bar, policy);
                }
            }
        return true;
    }
    __device__ __forceinline__ bool load_keys(int layer, const Keys& keys, uint64_t policy) {
        const ResidentLayer& L = p.layer[layer];
        bool ok = true;
        for_segments(keys, keys.line(s().n_kv, gridDim.x), s().n_kv, blockIdx.x, [&](const Segment g) {
            const int per = slices_per_slot<D>(g.s1 - g.s0), first = keys.first(g.token);
            const int* table = L.table + (size_t)entries[g.token] * s().max_blocks;
            for (int b0 = g.s0; ok && b0 < g.s1; b0 += 32) {    // the pages of 32 slices in one round of loads
                const int mine = b0 + lane < g.s1 ? table[(first + b0 + lane) * KEYS16 / s().page_size] : -1;
                const int b1 = min(g.s1, b0 + 32);
                for (int i = b0; i < b1; ++seq) {
                    if (!acquire()) { ok = false; break; }
                    const int n = min(per, b1 - i);
                    uint64_t* bar = &full[seq % SLOTS];
                    if (lane == 0) tc::mbar_expect_tx(bar, n * 64 * D);
                    for (int j = 0; j < n; ++j, ++i) {
                        const int page = __shfl_sync(0xffffffffu, mine, i - b0), key = (first + i) * KEYS16;
                        const int row = (max(page, 0) * s().n_kv + g.kvh) * s().page_size + key % s().page_size;
                        if (lane == 0) {
                            uint8_t* dst = smem + (seq % SLOTS) * SLOT + j * 64 * D;
#pragma unroll
                            for (int c = 0; c < D / 64; ++c) {
                                tc::tma_load_2d_hint(dst + c * 2048, &p.k_map[layer], c * 64, row, bar, policy);
                                tc::tma_load_2d_hint(dst + 32 * D + c * 2048, &p.v_map[layer], c * 64, row, bar, policy);
                            }
                        }
                    }
                }
            }
        });
        return ok;
    }
    __device__ __forceinline__ void loader() {
        const uint64_t policy = tc::policy_evict_first();       // weights and cache are read once per step
        const int G = gridDim.x, b = blockIdx.x, H = s().hidden, da = s().n_heads * D, nqkv = (s().n_heads + 2 * s().n_kv) * D;
        bool ok = true;
        for (int l = 0; ok && l < s().n_layers; ++l) {
            const ResidentLayer& L = p.layer[l];
            ok = load_matrix(L.w_qkv, share(b, nqkv, G), share(b + 1, nqkv, G), H, policy) &&
                 load_keys(l, Keys{pos, s().n_tok, L.window}, policy) &&
                 load_matrix(L.w_o, share(b, H, G), share(b + 1, H, G), da, policy) &&
                 load_matrix(L.w_gate_up, 2 * share(b, s().ff, G), 2 * share(b + 1, s().ff, G), H, policy) &&
                 load_matrix(L.w_down, share(b, H, G), share(b + 1, H, G), s().ff, policy);
        }
        if (!ok && lane == 0) *abort_flag = 1;
        // whatever is still on its way lands before the block (and its shared memory) goes away
        volatile int never = 0;
        for (uint32_t q = seq > SLOTS ? seq - SLOTS : 0; q < seq; ++q) tc::mbar_wait(&full[q % SLOTS], (q / SLOTS) & 1u, &never);
    }

    // ---- a product -----------------------------------------------------------------------------------------------------------
    // n tagged words of all blocks to shared memory, as bf16 (n is a multiple of 64)
    __device__ __forceinline__ void gather(const uint32_t* words, int n, uint32_t tag) {
        uint2* act = reinterpret_cast<uint2*>(smem + Smem::ACT);
        const uint32_t T = tag << 16;
        for (int v0 = threadIdx.x; v0 < n / 4; v0 += 8 * CT) {
            uint4 w[8];
            until([&] {
                uint32_t off = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (v0 + k * CT < n / 4) w[k] = look16(words + (v0 + k * CT) * 4);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (v0 + k * CT < n / 4) off |= (w[k].x ^ T) | (w[k].y ^ T) | (w[k].z ^ T) | (w[k].w ^ T);
                return off >> 16 == 0;
            });
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (v0 + k * CT < n / 4) act[v0 + k * CT] = make_uint2(__byte_perm(w[k].x, w[k].y, 0x5410), __byte_perm(w[k].z, w[k].w, 0x5410));
        }
        consumers_sync();
    }

    // The gathered [tokens, K] times the next `rows` weight rows of the ring; each(first, n) when the sums of n rows from `first` on
    // are in shared memory (total).
    template <typename F>
    __device__ __forceinline__ void product(int K, int rows, F each) {
        const int units = (rows + 7) / 8, groups = (units + UNITS - 1) / UNITS, per = groups ? (units + groups - 1) / groups : 0;
        const int g = lane >> 2, c = lane & 3, M = s().n_tok;
        const uint32_t act = tc::smem_u32(smem) + Smem::ACT + (g * K + warp * 32 + c * 8) * 2;
        const uint32_t mine_at = tc::smem_u32(smem) + g * ROW_BYTES + warp * 64 + c * 16;
#pragma unroll 1
        for (int u0 = 0; u0 < units; u0 += per) {
            const int n = min(per, units - u0);
            float acc[UNITS / 2][2][4];                         // pairs of units, in two chains
#pragma unroll
            for (int u = 0; u < UNITS / 2; ++u)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[u][0][i] = acc[u][1][i] = 0.f;
#pragma unroll 1
            for (int k0 = 0; k0 < K; k0 += PIECE) {
                const int steps = min(PIECE, K - k0) / 32;
                uint4 x[STEPS];                                 // this lane's activations of the piece
#pragma unroll
                for (int i = 0; i < STEPS; ++i)
                    x[i] = g < M && i * CW + warp < steps ? lds16(act + (k0 + i * (CW * 32)) * 2) : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int u = 0; u < UNITS / 2; ++u) {
                    if (2 * u < n) {
                        const bool two = 2 * u + 1 < n;
                        const uint32_t w0 = mine_at + (seq % SLOTS) * SLOT, w1 = mine_at + ((seq + 1) % SLOTS) * SLOT;
                        uint4 a0[STEPS], a1[STEPS];
                        arrived(seq);
#pragma unroll
                        for (int i = 0; i < STEPS; ++i)
                            if (i * CW + warp < steps) a0[i] = lds16(w0 + i * (CW * 64));
                        if (two) {
                            arrived(seq + 1);
#pragma unroll
                            for (int i = 0; i < STEPS; ++i)
                                if (i * CW + warp < steps) a1[i] = lds16(w1 + i * (CW * 64));
                        } else {
#pragma unroll
                            for (int i = 0; i < STEPS; ++i) a1[i] = make_uint4(0, 0, 0, 0);
                        }
#pragma unroll
                        for (int i = 0; i < STEPS; ++i)
                            if (i * CW + warp < steps) {
                                const uint32_t lo[4] = {a0[i].x, a1[i].x, a0[i].y, a1[i].y}, hi[4] = {a0[i].z, a1[i].z, a0[i].w, a1[i].w};
                                mma16816(acc[u][0], lo, x[i].x, x[i].y);
                                mma16816(acc[u][1], hi, x[i].z, x[i].w);
                            }
                        __syncwarp();
                        if (lane == 0) {
                            tc::mbar_arrive(&empty[seq % SLOTS]);
                            if (two) tc::mbar_arrive(&empty[(seq + 1) % SLOTS]);
                        }
                        seq += two ? 2 : 1;
                    }
                }
            }
            // the warps' sums: [warp][unit][token][8 rows]; a lane has rows g of both units, tokens 2 c and 2 c + 1
#pragma unroll
            for (int u = 0; u < UNITS / 2; ++u)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    red[((warp * UNITS + 2 * u + i / 2) * 8 + 2 * c + i % 2) * 8 + g] = acc[u][0][i] + acc[u][1][i];
            consumers_sync();
            each(u0 * 8, min(rows - u0 * 8, n * 8));
            consumers_sync();                                   // (the sums' place is free again)
        }
    }
    // the sum of all warps for row `row` of the group and token t
    __device__ __forceinline__ float total(int row, int t) const {
        const float* at = red + ((row >> 3) * 8 + t) * 8 + (row & 7);
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CW; ++w) v += at[w * UNITS * 64];
        return v;
    }

    // 1 / rms of every token from the blocks' sums of squares [parts][tokens]: a warp per token
    __device__ __forceinline__ void load_rms(const uint2* sums, int parts, float eps, uint32_t tag) {
        for (int t = warp; t < s().n_tok; t += CW) {
            float v = 0.f;
            uint2 w[8];                                         // (parts is at most 256)
            until([&] {
                bool all = true;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k * 32 + lane < parts) w[k] = look8(sums + (k * 32 + lane) * TOKENS + t);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k * 32 + lane < parts) all &= w[k].y == tag;
                return all;
            });
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k * 32 + lane < parts) v += __uint_as_float(w[k].x);
            v = warp_sum(v);
            if (lane == 0) rms[t] = 1.0f / sqrtf(v * s().inv_hidden + eps);
        }
    }

    // ---- attention -------------------------------------------------------------------------------------------------------------
    __device__ __forceinline__ void angles(int token, const float* inv_freq) {
        float2* at = reinterpret_cast<float2*>(smem + Smem::ANGLES);
        for (int i = threadIdx.x; i < s().rotary_dim / 2; i += CT) {
            float sn, cs;
            sincosf((float)pos[token] * inv_freq[i], &sn, &cs);
            at[i] = make_float2(sn, cs);
        }
    }
    __device__ __forceinline__ void segment(int layer, const Segment g, bool turned) {
        const ResidentLayer& L = p.layer[layer];
        const int group = s().n_heads / s().n_kv, rot = s().rotary_dim, half = rot / 2, t = g.token, at_pos = pos[t];
        const Keys keys{pos, s().n_tok, L.window};
        const int first = keys.first(t), lo = L.window > 0 ? max(0, at_pos - L.window + 1) : 0;
        const int nqkv = (s().n_heads + 2 * s().n_kv) * D, h0 = g.kvh * group;
        const uint32_t tag = layer + 1;
        bf16* q_rows = reinterpret_cast<bf16*>(smem + Smem::Q);
        bf16* own_kv = reinterpret_cast<bf16*>(smem + Smem::KV);
        const float2* at = reinterpret_cast<const float2*>(smem + Smem::ANGLES);
        if (!turned) {                                          // (the angles of the block's first token are there already)
            angles(t, L.inv_freq);
            consumers_sync();
        }
        // q of the group's heads, and the token's own key and value where they are this block's: rotated, in bf16
        const bool own = g.s1 == keys.slices(t);
        const uint2* row = s().qkv + (size_t)t * nqkv;
        const int n_q = group * (D / 2), n_all = n_q + (own ? D : 0);
        const int page = own ? L.table[(size_t)entries[t] * s().max_blocks + at_pos / s().page_size] : -1;
        const size_t cache_row = (((size_t)max(page, 0) * s().n_kv + g.kvh) * s().page_size + at_pos % s().page_size) * D;
        for (int e = threadIdx.x; e < n_all; e += CT) {         // a pair of columns each
            const bool is_q = e < n_q, is_v = e >= n_q + D / 2;
            const int r = is_q ? e / (D / 2) : 0, i = is_q ? e - r * (D / 2) : (e - n_q) % (D / 2);
            // the pair: (i, i + half) where it rotates, else neighbouring columns (behind the rotated ones)
            const bool turns = !is_v && i < half;
            const int c0 = turns ? i : is_v ? 2 * i : rot + 2 * (i - half), c1 = turns ? i + half : c0 + 1;
            const uint2* src = row + (size_t)(is_q ? h0 + r : is_v ? s().n_heads + s().n_kv + g.kvh : s().n_heads + g.kvh) * D;
            uint2 wa, wb;
            until([&] {
                wa = look8(src + c0), wb = look8(src + c1);
                return wa.y == tag && wb.y == tag;
            });
            float a = __uint_as_float(wa.x), b = __uint_as_float(wb.x);
            if (turns) {
                const float2 w = at[i];
                const float ra = a * w.y - b * w.x, rb = a * w.x + b * w.y;
                a = ra, b = rb;
            }
            bf16* dst = is_q ? q_rows + r * (D + 8) : own_kv + (is_v ? D : 0);
            dst[c0] = __float2bfloat16_rn(a);
            dst[c1] = __float2bfloat16_rn(b);
            if (!is_q && page >= 0) {
                bf16* cache = (is_v ? L.v_cache : L.k_cache) + cache_row;
                cache[c0] = __float2bfloat16_rn(a);
                cache[c1] = __float2bfloat16_rn(b);
            }
        }
        consumers_sync();
        uint32_t qf[D / 16][4];
        load_q<D>(qf, q_rows, (size_t)(D + 8), group, lane);
        float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f}, o[D / 8][4];
#pragma unroll
        for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
        const int per = slices_per_slot<D>(g.s1 - g.s0);
        int turn = 0;
        for (int b0 = g.s0; b0 < g.s1; b0 += 32)
            for (int i = b0; i < min(g.s1, b0 + 32); i += per, ++seq, turn = turn + 1 == CW ? 0 : turn + 1) {
                if (turn != warp) {
                    // Another warp's slot, watched all the same: a parity wait tells a phase from the next only, so a warp has to have
                    // seen the barrier's phase before the one it waits for, and the slot is not filled again before all have.
                    if (lane == 0) {
                        arrived(seq);
                        tc::mbar_arrive(&empty[seq % SLOTS]);
                    }
                    continue;
                }
                __syncwarp();                                   // (lane 0 has seen the slots in between)
                arrived(seq);
                const int n = min(per, min(g.s1, b0 + 32) - i);
                for (int j = 0; j < n; ++j) {
                    bf16* kt = reinterpret_cast<bf16*>(smem + (seq % SLOTS) * SLOT + j * 64 * D);
                    bf16* vt = kt + 16 * D;
                    const int kb = (first + i + j) * KEYS16;
                    if (at_pos >= kb && at_pos < kb + KEYS16) {
                        // the slice came from the cache before the token's own key and value were there
                        if (lane < D / 8) {
                            const int chunk = Swizzled128<D, 16>::chunk(at_pos - kb, lane) * 8;
                            *reinterpret_cast<uint4*>(kt + chunk) = *reinterpret_cast<const uint4*>(own_kv + lane * 8);
                            *reinterpret_cast<uint4*>(vt + chunk) = *reinterpret_cast<const uint4*>(own_kv + D + lane * 8);
                        }
                        tc::fence_proxy_async();                // (the slot's next load comes behind this write)
                        __syncwarp();
                    }
                    slice16<D, Swizzled128<D, 16>>(qf, kt, vt, 0, kb, lo, at_pos, lo, at_pos, L.scale_log2, m, l, o, lane);
                }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&empty[seq % SLOTS]);
            }
        // ---- the warps' results, 64 columns at a time
        const int gr = lane >> 2, c = lane & 3;
        float2* ml = reinterpret_cast<float2*>(smem + Smem::ML);
        float l0 = l[0];
        l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
        l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
        if (c == 0) ml[warp * GROUP + gr] = make_float2(m[0], l0);
        const bool alone = g.first == g.last;
        const size_t seg = blockIdx.x + g.pair;                 // pieces in order: every next one is of the next block or pair
        float* po = s().part_o + seg * (GROUP * D);
        float2* pml = reinterpret_cast<float2*>(s().part_ml) + seg * GROUP;
        constexpr int RS = 68;                                  // floats between rows of a warp's results
#pragma unroll
        for (int hcol = 0; hcol < D / 64; ++hcol) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float2*>(red + (warp * GROUP + gr) * RS + i * 8 + c * 2) = make_float2(o[hcol * 8 + i][0], o[hcol * 8 + i][1]);
            consumers_sync();
            for (int e = threadIdx.x; e < group * 32; e += CT) {
                const int r = e >> 5, d = (e & 31) * 2;
                float M = -CUDART_INF_F, sum = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll
                for (int w = 0; w < CW; ++w) M = fmaxf(M, ml[w * GROUP + r].x);
#pragma unroll
                for (int w = 0; w < CW; ++w) {
                    const float2 x = ml[w * GROUP + r];
                    const float k = x.x == -CUDART_INF_F ? 0.f : exp2f(x.x - M);
                    if (k != 0.f) {                             // (a warp without keys is left out)
                        const float2 y = *reinterpret_cast<const float2*>(red + (w * GROUP + r) * RS + d);
                        sum = fmaf(x.y, k, sum), v0 = fmaf(y.x, k, v0), v1 = fmaf(y.y, k, v1);
                    }
                }
                const int col = hcol * 64 + d;
                if (alone) {
                    const float inv = 1.0f / sum;
                    const size_t to = ((size_t)t * s().n_heads + h0 + r) * D + col;
                    tell(s().attn + to, tagged(v0 * inv, tag));
                    tell(s().attn + to + 1, tagged(v1 * inv, tag));
                } else {
                    *reinterpret_cast<float2*>(po + r * D + col) = make_float2(v0, v1);
                    if (col == 0) pml[r] = make_float2(M, sum);
                }
            }
            consumers_sync();
        }
        if (alone) return;
        // ---- the block that arrives last merges the blocks' results (a counter of the layer's own: one that was set back for the
        // next layer would have nothing that orders the reset before that layer's arrivals)
        int* s_last = reinterpret_cast<int*>(smem + Smem::MISC) + 28;
        if (threadIdx.x == 0) {
            int old;
            asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(old) : "l"(s().counters + (size_t)layer * TOKENS * s().n_kv + g.pair) : "memory");
            *s_last = old == g.last - g.first;
        }
        consumers_sync();
        if (*s_last) merge<D>(s(), g, tag);
        consumers_sync();
    }

    // ---- the consumers' step ---------------------------------------------------------------------------------------------------
    __device__ __forceinline__ void attention(int l) {
        const Keys keys{pos, s().n_tok, p.layer[l].window};
        const Line line = keys.line(s().n_kv, gridDim.x);
        int turned = -1;                                        // the token whose angles are there
        for_segments(keys, line, s().n_kv, blockIdx.x, [&](const Segment g) {
            if (turned < 0) angles(g.token, p.layer[l].inv_freq), turned = g.token;
        });
        consumers_sync();
        for_segments(keys, line, s().n_kv, blockIdx.x, [&](const Segment g) {
            segment(l, g, turned == g.token);
            turned = g.token;
        });
    }
    // One of the four products of a layer: q/k/v, output, gate/up, down.
    __device__ __forceinline__ void multiply(int l, int which) {
        const int G = gridDim.x, b = blockIdx.x, H = s().hidden, M = s().n_tok, da = s().n_heads * D, nqkv = (s().n_heads + 2 * s().n_kv) * D;
        const ResidentLayer& L = p.layer[l];
        const uint32_t tag = l + 1, next_tag = which == 3 ? l + 2 : l + 1;      // of what this product reads and of h behind it
        const bool last = which == 3 && l + 1 == s().n_layers, residual = which == 1 || which == 3;
        const int n = which == 0 ? nqkv : which == 2 ? s().ff : H, pairs = which == 2 ? 2 : 1;
        const int r0 = share(b, n, G) * pairs, rows = share(b + 1, n, G) * pairs - r0;
        const uint32_t* in = which == 0 ? s().h[0] : which == 1 ? s().attn : which == 2 ? s().h[1] : s().act;
        gather(in, M * (which == 1 ? da : which == 3 ? s().ff : H), tag);
        if (!residual) load_rms(s().sums[which / 2], l + which == 0 ? 1 : G, which == 0 ? L.eps_mixer : L.eps_ffn, tag);
        const void* bias = which == 0 ? L.b_qkv : which == 1 ? L.b_o : nullptr;
        const void* norm_w = which == 1 ? L.norm_ffn : which == 3 && !last ? p.layer[l + 1].norm_mixer : nullptr;
        const int next = which == 1;                            // whose h and sums a residual product hands on
        product(which == 1 ? da : which == 3 ? s().ff : H, rows, [&](int first, int here) {
            const int mine = here / pairs;                      // results of this block (a gate and its up row make one)
#pragma unroll 1
            for (int e = threadIdx.x; e < mine * M; e += CT) {
                const int t = e / mine, i = e - t * mine, col = (r0 + first) / pairs + i;
                if (which == 2) {
                    const float v = glu_act(total(2 * i, t) * rms[t], total(2 * i + 1, t) * rms[t], GLU_SILU, 0.f, 0.f);
                    const size_t to = (size_t)t * s().ff + col;
                    tell(s().act + to, tagged(v, tag));
                    continue;
                }
                float v = total(i, t);
                if (which == 0) v *= rms[t];
                if (bias) v += load_any(bias, which == 0 ? s().qkv_bias_dtype : s().o_bias_dtype, col);
                if (which == 0) {
                    const size_t to = (size_t)t * nqkv + col;
                    tell(s().qkv + to, v, tag);
                    continue;
                }
                float* x = x_s + t * MAX_ROWS + first + i;
                *x = v += *x;
                const size_t to = (size_t)t * H + col;
                if (last) {
                    s().x[to] = v;
                    continue;
                }
                v *= load_any(norm_w, s().norm_dtype, col);
                tell(s().h[next] + to, tagged(v, next_tag));
            }
        });
        if (residual && !last)
            for (int t = warp; t < M; t += CW) {
                float v = 0.f;
                for (int i = lane; i < rows; i += 32) v += x_s[t * MAX_ROWS + i] * x_s[t * MAX_ROWS + i];
                v = warp_sum(v);
                if (lane == 0) tell(s().sums[next] + b * TOKENS + t, v, next_tag);
            }
    }
    __device__ __forceinline__ void consume() {
        const int G = gridDim.x, H = s().hidden, x0 = share(blockIdx.x, H, G), x_rows = share(blockIdx.x + 1, H, G) - x0;
        for (int e = threadIdx.x; e < x_rows * s().n_tok; e += CT) x_s[e / x_rows * MAX_ROWS + e % x_rows] = s().x[(size_t)(e / x_rows) * H + x0 + e % x_rows];
        consumers_sync();
#pragma unroll 1
        for (int step = 0; step < 4 * s().n_layers; ++step) {   // (one body for the four products)
            if (step % 4 == 1) attention(step / 4);
            multiply(step / 4, step % 4);
        }
    }
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1) decode_resident_kernel(const __grid_constant__ Params p) {
    extern __shared__ uint8_t smem_raw[];
    Block<D> block(p, smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u));
    if (threadIdx.x < p.s.n_tok) {
        block.pos[threadIdx.x] = p.s.positions[threadIdx.x];
        block.entries[threadIdx.x] = p.s.tok_entry[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < SLOTS; ++i) tc::mbar_init(&block.full[i], 1), tc::mbar_init(&block.empty[i], CW);
        *block.abort_flag = 0;
        tc::fence_barrier_init();
        tc::fence_proxy_async();
    }
    __syncthreads();
    if (block.warp == CW) block.loader();
    else block.consume();
}

// The step's first kernel: a token's embedding, bf16(x * w) for the first product and the sum of squares behind its norm; no other
// word has a tag, and the pairs' arrival counters start at zero.
constexpr int BEGIN_BLOCKS = 64;
template <typename TE>
__global__ void __launch_bounds__(256) resident_begin_kernel(const TE* __restrict__ table, const int* __restrict__ ids,
                                                              const int* __restrict__ device_tokens, int vocab, float scale,
                                                              const void* __restrict__ w, const ResidentStep s, int head_dim, int blocks) {
    __shared__ float red[32];
    const int at = blockIdx.x * 256 + threadIdx.x, all = gridDim.x * 256;
    auto clear = [&](void* p, long long words) {
        for (long long i = at; i < words; i += all) reinterpret_cast<uint32_t*>(p)[i] = 0;
    };
    clear(s.h[1], (long long)s.n_tok * s.hidden);
    clear(s.attn, (long long)s.n_tok * s.n_heads * head_dim);
    clear(s.act, (long long)s.n_tok * s.ff);
    clear(s.qkv, 2ll * s.n_tok * (s.n_heads + 2 * s.n_kv) * head_dim);
    clear(s.sums[1], 2ll * blocks * TOKENS);
    clear(s.sums[0] + TOKENS, 2ll * (blocks - 1) * TOKENS);
    clear(s.stop, 1);
    clear(s.counters, (long long)s.n_layers * TOKENS * s.n_kv);
    const int t = blockIdx.x;
    if (t >= s.n_tok) return;
    int id = ids[t];
    if (id < 0 && device_tokens) id = device_tokens[-id - 1];   // (the sampler's token, see embed_gather_kernel)
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    float ss = 0.f;
    for (int i = threadIdx.x; i < s.hidden; i += 256) {
        const float v = to_f32(table[(size_t)id * s.hidden + i]) * scale;
        const size_t to = (size_t)t * s.hidden + i;
        s.x[to] = v;
        s.h[0][to] = tagged(v * load_any(w, s.norm_dtype, i), 1);
        ss += v * v;
    }
    ss = block_sum(ss, red);
    if (threadIdx.x == 0) s.sums[0][t] = make_uint2(__float_as_uint(ss), 1);
}

long long up(long long v) { return (v + 255) / 256 * 256; }

}  // namespace

// Scratch of a step of up to TOKENS tokens; sets the step's pointers into `at`.
long long infero_resident_scratch(ResidentStep* s, uint8_t* at, int head_dim, int blocks) {
    long long off = 0;
    auto take = [&](long long bytes) { const long long here = off; off += up(bytes); return at ? at + here : nullptr; };
    const long long da = (long long)s->n_heads * head_dim, nqkv = (long long)(s->n_heads + 2 * s->n_kv) * head_dim, pieces = blocks + TOKENS * s->n_kv;
    for (int i = 0; i < 2; ++i) s->h[i] = (uint32_t*)take(TOKENS * (long long)s->hidden * 4), s->sums[i] = (uint2*)take((long long)blocks * TOKENS * 8);
    s->qkv = (uint2*)take(TOKENS * nqkv * 8);
    s->attn = (uint32_t*)take(TOKENS * da * 4);
    s->act = (uint32_t*)take(TOKENS * (long long)s->ff * 4);
    s->part_o = (float*)take(pieces * GROUP * head_dim * 4);
    s->part_ml = (float*)take(pieces * GROUP * 8);
    s->stop = (unsigned int*)take(4);
    s->counters = (int*)take((long long)RESIDENT_LAYERS * TOKENS * s->n_kv * 4);
    return off;
}

// Can a step of these sizes run here?  All of K must come in whole 32 columns and rows start on 16 bytes; a block's part of the
// residual stream, a product's activations and a kv head's query heads have to fit their places; every block needs a part of every
// product worth a unit.
int infero_resident_supported(const ResidentStep* s, int head_dim, int blocks) {
    const long long H = s->hidden, da = (long long)s->n_heads * head_dim;
    return s->n_tok >= 1 && s->n_tok <= TOKENS && s->n_layers >= 1 && s->n_layers <= RESIDENT_LAYERS && (head_dim == 64 || head_dim == 128) &&
           s->page_size % 16 == 0 && s->n_kv > 0 && s->n_heads % s->n_kv == 0 && s->n_heads / s->n_kv <= GROUP && H % 64 == 0 &&
           s->ff % 64 == 0 && da % 64 == 0 && H / blocks + 1 <= MAX_ROWS && s->rotary_dim % 2 == 0 && s->rotary_dim <= head_dim &&
           blocks <= 256 && s->ff >= blocks && H >= 4 * blocks && s->n_tok * std::max({(long long)s->ff, H, da}) * 2 <= ACT_BYTES;
}

// Is it the faster way?  What it saves are the waits between launches; what it pays are a copy per slot and block (about 7 us a slot
// of a layer, over 24 layers) and keys that few warps go through (22 us a thousand, where the launches hardly notice them).  `visible`:
// keys of the longest request that some layer sees.  Launches and this, replayed, us a step of 24 layers:
//   width 896, 14 heads of 64 over 2, ff 4,864 (197 KiB of a layer's weights a block, 17 slots): one token at 20 keys 643 and 520, 300 687
//   and 585, 1,000 695 and 609, 2,000 699 and 627, 3,000 684 and 649, 4,095 684 and 660, 8,191 750 and 766, 16,383 805 and 858; two at 300 706 and
//   610, at 2,000 692 and 659, at 4,095 each 700 and 695, at 8,191 769 and 817.
//   up to 256 KiB: width 640, ff 8,192 (26 slots) one token at 2,040 684 and 662, at 4,090 668 and 704; 1,024, ff 5,120 (30 slots) 677 and
//   664, 685 and 707; 2,048, ff 1,536 767 and 766, 775 and 853; 640, ff 6,144 (20 slots) at 4,090 652 and 653; 896, ff 6,272 (20 slots) 695
//   and 654.  So 2,048 keys in all, 4,096 where a layer takes up to 20 slots.
//   beyond: width 1,024, ff 5,504 (258 KiB) one token at 300 683 and 644, two 671 and 675; ff 6,912 (315) 698 and 699, two 713 and 739; 1,536, ff
//   8,960 (616) 886 and 920; at 7B sizes 2,689 and 3,381.
//   where the pairs' rounds of 112 keys are more than the blocks, a block has pieces of several pairs: 1,024, ff 4,096, 8 heads of 128 over 8,
//   one token at 2,040 688 and 752; 16 heads of 64 over 16, ff 4,608 696 and 747.  Layers of up to 128 KiB bear it: 640, ff 2,560, 10 of 64
//   over 10 at 4,090 (2.5 times the blocks) 686 and 615; 640, ff 1,024, 16 of 128 over 16 at 2,040 (2.05) 731 and 705, at 4,090 (4) 706 and 811.
int infero_resident_worth(const ResidentStep* s, int head_dim, int blocks, int visible) {
    const long long H = s->hidden, da = (long long)s->n_heads * head_dim, nqkv = (long long)(s->n_heads + 2 * s->n_kv) * head_dim;
    const long long bytes = 2 * H * (nqkv + da + 3ll * s->ff) / blocks, keys = (long long)s->n_tok * visible;
    auto slots = [&](long long n, long long K, int pairs) { return (((n + blocks - 1) / blocks) * pairs + 7) / 8 * ((K + PIECE - 1) / PIECE); };
    const long long a_layer = slots(nqkv, H, 1) + slots(H, da, 1) + slots(s->ff, H, 2) + slots(H, s->ff, 1);
    const long long rounds = (long long)s->n_tok * s->n_kv * ((visible / KEYS16 + CW) / CW);
    return bytes <= 256 * 1024 && keys <= (a_layer <= 20 || bytes <= 128 * 1024 ? 4096 : 2048) &&
           2 * rounds <= (bytes <= 128 * 1024 ? 5 : 2) * blocks;
}

// Returns 0, 1 with the error recorded, or 2 when the device cannot hold the blocks all at once: a multiprocessor has no room for one, there are
// fewer multiprocessors than blocks, or the launch is refused because part of them is set aside (all that has run then is the step's first
// kernel, whose results nobody else reads).
int infero_decode_resident(const ResidentStep* s, const ResidentLayer* layers, int head_dim, const int* num_pages, const void* embed,
                           int embed_dtype, const int* ids, const int* device_tokens, int vocab, float embed_scale, int blocks,
                           cudaStream_t stream) {
    static std::mutex mutex;
    static int fits[2] = {-1, -1};                              // blocks a multiprocessor holds, by head size
    void* kernel = head_dim == 64 ? (void*)decode_resident_kernel<64> : (void*)decode_resident_kernel<128>;
    {
        std::lock_guard<std::mutex> lock(mutex);
        int& n = fits[head_dim == 128];
        if (n < 0) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::TOTAL);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, THREADS, Smem::TOTAL);
            if (e != cudaSuccess) n = 0, cudaGetLastError();
        }
        if (n < 1 || blocks > (long long)n * infero_sm_count()) return 2;
    }
    Params p;
    p.s = *s;
    if (infero_tc_err_flag(&p.err_flag)) return 1;
    for (int l = 0; l < s->n_layers; ++l) {
        p.layer[l] = layers[l];
        if (infero_tensor_map_bf16(layers[l].k_cache, num_pages[l] * s->n_kv * s->page_size, head_dim, head_dim, 16, &p.k_map[l]) ||
            infero_tensor_map_bf16(layers[l].v_cache, num_pages[l] * s->n_kv * s->page_size, head_dim, head_dim, 16, &p.v_map[l]))
            return 1;
    }
    auto begin = [&](auto* table) {
        resident_begin_kernel<<<BEGIN_BLOCKS, 256, 0, stream>>>(table, ids, device_tokens, vocab, embed_scale, layers[0].norm_mixer, *s, head_dim, blocks);
    };
    if (embed_dtype == INFERO_F32) begin((const float*)embed);
    else begin((const bf16*)embed);
    if (infero_check_launch("resident_begin")) return 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks;
    cfg.blockDim = THREADS;
    cfg.dynamicSmemBytes = Smem::TOTAL;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;                // the blocks wait for one another: all of them or none
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {&p};
    if (cudaLaunchKernelExC(&cfg, kernel, args) == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return 2;
    }
    return infero_check_launch("decode_resident");
}
