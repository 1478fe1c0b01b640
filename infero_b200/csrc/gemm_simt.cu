// Matrix products on the ordinary cores: out[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
//
//  * gemm_tiled: any shape, any mix of float / bf16 operands, 32-bit accumulation with one
//    fused multiply-add per k, in an order that depends on K alone.  The value of out[m,n] therefore
//    does not depend on M, on the tile it falls in or on its batch-mates: this is the product of the
//    true 32-bit path (no reduced-precision matrix mode anywhere).
//  * gemm_skinny: up to 4 rows of A (decode at tiny batch): one warp per pair of output
//    features streams the weight rows with 16-byte loads.  The reference switches to its
//    own mat-vec at the same point (crates/model/src/lib.rs:1574, cu/quant.cu:266-286).
//
// W is [N,K] row-major, as checkpoints store it (crates/model/src/weights.rs:2276-2277).
#include "common.cuh"

extern "C" int infero_sm_count();

namespace {

// One block works out BM x BN results, TM x TN a thread.  Both operands keep their rows in shared memory as they lie in
// memory ([row][k], rows padded by 16 bytes): a stage of BK columns arrives by 16-byte asynchronous copies, STAGES - 1 stages
// ahead, and a thread reads four k of a row at a time.  Thread (ty, tx) has rows ty + i * (BM / TM) and columns
// tx + j * (BN / TN); a warp is eight threads wide and four high where there are so many rows, so that eight neighbouring lanes
// read eight neighbouring rows, whose starts lie 4 banks apart (BK + 4 is an odd multiple of 4): no bank conflict.  Operands that
// 16-byte copies cannot take (bf16, rows that start anywhere) come by plain loads into the same ring.
//
// K is cut into parts of equal length that depend on K alone (parts_of).  A part's result is two chains of fused multiply-adds,
// over its even and its odd k in ascending order (one instruction takes a step of both), and their sum; a result is the sum of its
// parts in ascending order.  That holds whatever the tile and whether a block runs through all parts or (SPLIT) the blocks of a
// cluster take one each and add them up through each other's shared memory, so the choice never shows in the numbers.  Against
// 64-bit products of normal numbers: 2.7e-7 (2-norm) at K = 896 and 3.2e-7 at 4,864; one chain in ascending k had 5.4e-7 and 1.3e-6.
template <int BM, int BN, int TM, int TN, int BK, int STAGES>
struct Tile {
    static constexpr int TX = BN / TN, TY = BM / TM, WORK = TX * TY, THREADS = WORK < 32 ? 32 : WORK;
    static constexpr int LY = TY < 4 ? TY : 4, LX = WORK < 32 ? TX : 32 / LY;              // a warp has LX x LY threads
    static constexpr int LD = BK + 4, A_FLOATS = BM * LD, STAGE = (BM + BN) * LD;
    static constexpr int Q = BK / 4;                                                       // copies a row
    static constexpr int FLOATS = STAGES * STAGE > BM * BN ? STAGES * STAGE : BM * BN;     // (a part's results take the ring's place)
    static constexpr size_t SMEM = (size_t)FLOATS * sizeof(float);
    static_assert(SMEM <= 48 * 1024, "more shared memory than a launch gets without asking");
    static_assert(BK % 4 == 0 && (BK / 4) % 2 == 0 && THREADS % Q == 0, "");
    static_assert(TX % LX == 0 && TY % LY == 0, "");
};

constexpr int PART = 640, MAX_SPLIT = 8;
struct Parts { int n, len; };
Parts parts_of(int K) {
    const int n = (K + PART - 1) / PART, len = ((K + n - 1) / n + 31) / 32 * 32;
    return {(K + len - 1) / len, len};
}

// a + b * c for two numbers at a time, each rounded once
__device__ __forceinline__ void fma2(unsigned long long& a, unsigned long long b, unsigned long long c) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(b), "l"(c));
}

// The rows of an operand in a stage, zeros from column k_end on and where there is no row.  This thread copies 16 bytes of every
// STEP-th row from row `row` on, src being its place in the first of them.
template <int ROWS, int LD, int STEP>
__device__ __forceinline__ void copy_rows(unsigned int dst, const float* src, const float* any, long long ld, int row, int n_rows, bool in) {
#pragma unroll
    for (int i = 0; i < (ROWS + STEP - 1) / STEP; ++i, src += ld * STEP) {
        if (ROWS % STEP != 0 && row + i * STEP >= ROWS) break;
        const bool ok = in && row + i * STEP < n_rows;          // (nothing is read of a row that is not there)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * STEP * LD * 4), "l"(ok ? src : any), "r"(ok ? 16 : 0) : "memory");
    }
}
// The same element by element, widened on the way: this thread takes a column of every STEP-th row; its loads are on their way
// together before the first is stored.
template <int ROWS, int LD, int STEP, typename T>
__device__ __forceinline__ void widen_rows(float* dst, const T* src, long long ld, int row, int n_rows, bool in) {
    constexpr int N = (ROWS + STEP - 1) / STEP;
    float v[N];
#pragma unroll
    for (int i = 0; i < N; ++i, src += ld * STEP) v[i] = in && row + i * STEP < n_rows && (ROWS % STEP == 0 || row + i * STEP < ROWS) ? to_f32(*src) : 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (ROWS % STEP == 0 || row + i * STEP < ROWS) dst[i * STEP * LD] = v[i];
}
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename TL, int BM, int BN, int TM, int TN, int BK, int STAGES, bool SPLIT, bool VEC, typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(TL::THREADS)
gemm_tiled_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const void* __restrict__ bias,
                  int bias_dtype, TC* __restrict__ C, int M, int N, int K, int lda, int ldc, int part_len) {
    extern __shared__ float4 ring4[];
    float* ring = reinterpret_cast<float*>(ring4);
    constexpr int LD = TL::LD;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int ty = warp / (TL::TX / TL::LX) * TL::LY + lane / TL::LX, tx = warp % (TL::TX / TL::LX) * TL::LX + lane % TL::LX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const bool works = TL::WORK == TL::THREADS || tid < TL::WORK;
    const int k_first = SPLIT ? blockIdx.z * part_len : 0, k_last = SPLIT ? min(K, k_first + part_len) : K;
    static_assert(VEC || TL::THREADS % BK == 0, "a round of loads is whole rows");
    const int row = tid / (VEC ? TL::Q : BK), col = VEC ? tid % TL::Q * 4 : tid % BK;
    const TA* a_src = A + (long long)(m0 + row) * lda + col;
    const TW* w_src = W + (long long)(n0 + row) * K + col;
    const unsigned int ring_at = (unsigned int)__cvta_generic_to_shared(ring);
    int next_k = k_first, next_end = min(K, k_first + part_len), slot = 0;      // the next stage to load
    auto load = [&]() {
        if (next_k < k_last) {
            if constexpr (VEC) {
                const unsigned int dst = ring_at + (slot * TL::STAGE + row * LD + col) * 4;
                const bool in = next_k + col < next_end;        // (K is a multiple of 4 here)
                copy_rows<BM, LD, TL::THREADS / TL::Q>(dst, a_src + next_k, A, lda, row, M - m0, in);
                copy_rows<BN, LD, TL::THREADS / TL::Q>(dst + TL::A_FLOATS * 4, w_src + next_k, W, K, row, N - n0, in);
            } else {
                float* dst = ring + slot * TL::STAGE + row * LD + col;
                const bool in = next_k + col < next_end;
                widen_rows<BM, LD, TL::THREADS / BK>(dst, a_src + next_k, lda, row, M - m0, in);
                widen_rows<BN, LD, TL::THREADS / BK>(dst + TL::A_FLOATS, w_src + next_k, K, row, N - n0, in);
            }
            next_k += BK;
            if (next_k >= next_end) next_k = next_end, next_end = min(K, next_end + part_len);
            slot = slot + 1 == STAGES ? 0 : slot + 1;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float sum[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sum[i][j] = 0.f;
    for (int s = 0; s < STAGES - 1; ++s) load();
    int here = 0, first = k_first;
    do {                                                        // a part
        const int end = min(K, first + part_len);
        unsigned long long acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0;
        for (int k0 = first; k0 < end; k0 += BK) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();                                    // this stage is here, and everyone is done with the one before,
            load();                                             // whose place this fills
            const float* a_s = ring + here * TL::STAGE + ty * LD;
            const float* w_s = ring + here * TL::STAGE + TL::A_FLOATS + tx * LD;
            here = here + 1 == STAGES ? 0 : here + 1;
            if (!works) continue;
#pragma unroll
            for (int k = 0; k < BK; k += 4) {
                ulonglong2 w[TN], a[TM];
#pragma unroll
                for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(w_s + j * TL::TX * LD + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a_s + i * TL::TY * LD + k);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) fma2(acc[i][j], a[i].x, w[j].x);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) fma2(acc[i][j], a[i].y, w[j].y);
            }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) sum[i][j] += __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
        first = end;
    } while (!SPLIT && first < K);
    if constexpr (SPLIT) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                        // the ring's place is free: this block's part of the results
        if (works) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) ring[(ty + i * TL::TY) * BN + tx + j * TL::TX] = sum[i][j];
        }
        cluster_meet();
        for (int e = blockIdx.z * TL::THREADS + tid; e < BM * BN; e += gridDim.z * TL::THREADS) {
            const int gm = m0 + e / BN, gn = n0 + e % BN;
            if (gm >= M || gn >= N) continue;
            float part[MAX_SPLIT], v = 0.f;
#pragma unroll
            for (int p = 0; p < MAX_SPLIT; ++p)
                if (p < gridDim.z) {
                    unsigned int at;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(ring_at + e * 4), "r"(p));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[p]) : "r"(at) : "memory");
                }
#pragma unroll
            for (int p = 0; p < MAX_SPLIT; ++p)
                if (p < gridDim.z) v += part[p];
            if (bias) v += load_any(bias, bias_dtype, gn);
            C[(size_t)gm * ldc + gn] = from_f32<TC>(v);
        }
        cluster_meet();                                         // nobody's part goes before it has been read
        return;
    }
    if (!works) return;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + i * TL::TY;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx + j * TL::TX;
            if (gn >= N) continue;
            float v = sum[i][j];
            if (bias) v += load_any(bias, bias_dtype, gn);
            C[(size_t)gm * ldc + gn] = from_f32<TC>(v);
        }
    }
}

// bf16 weights and activations, M <= 4.  Each warp owns ROWS output features and walks K
// in steps of 256 (32 lanes x 8 elements).  K % 8 == 0 and 16-byte aligned rows required.
constexpr int SK_ROWS = 2;
template <int MT, typename TC>
__global__ void __launch_bounds__(256)
gemm_skinny_kernel(const bf16* __restrict__ A, const bf16* __restrict__ W, const void* __restrict__ bias,
                   int bias_dtype, TC* __restrict__ C, int M, int N, int K, int lda, int ldc) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_base = (blockIdx.x * 8 + warp) * SK_ROWS;
    if (n_base >= N) return;
    float acc[SK_ROWS][MT];
#pragma unroll
    for (int r = 0; r < SK_ROWS; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;

    for (int k = lane * 8; k < K; k += 256) {
        uint4 wv[SK_ROWS];
#pragma unroll
        for (int r = 0; r < SK_ROWS; ++r) {
            const int n = n_base + r < N ? n_base + r : N - 1;
            wv[r] = __ldg(reinterpret_cast<const uint4*>(W + (size_t)n * K + k));
        }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m < M) {
                const uint4 av = *reinterpret_cast<const uint4*>(A + (size_t)m * lda + k);
                const uint32_t au[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
                for (int r = 0; r < SK_ROWS; ++r) {
                    const uint32_t wu[4] = {wv[r].x, wv[r].y, wv[r].z, wv[r].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        // a bf16 is the upper half of a float
                        const float a0 = __uint_as_float(au[q] << 16), a1 = __uint_as_float(au[q] & 0xffff0000u);
                        const float w0 = __uint_as_float(wu[q] << 16), w1 = __uint_as_float(wu[q] & 0xffff0000u);
                        acc[r][m] = fmaf(a0, w0, acc[r][m]);
                        acc[r][m] = fmaf(a1, w1, acc[r][m]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < SK_ROWS; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float v = warp_sum(acc[r][m]);
            const int n = n_base + r;
            if (lane == 0 && m < M && n < N) {
                if (bias) v += load_any(bias, bias_dtype, n);
                C[(size_t)m * ldc + n] = from_f32<TC>(v);
            }
        }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool SPLIT, bool VEC, typename TA, typename TW, typename TC>
int launch_tile(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N,
                int K, int lda, int ldc, cudaStream_t stream) {
    using TL = Tile<BM, BN, TM, TN, BK, STAGES>;
    const Parts parts = parts_of(K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((N + BN - 1) / BN, (M + BM - 1) / BM, SPLIT ? parts.n : 1);
    cfg.blockDim = TL::THREADS;
    cfg.dynamicSmemBytes = TL::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = parts.n;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 1 : 0;
    cudaLaunchKernelEx(&cfg, gemm_tiled_kernel<TL, BM, BN, TM, TN, BK, STAGES, SPLIT, VEC, TA, TW, TC>,
                       (const TA*)A, (const TW*)W, bias, bias_dtype, (TC*)C, M, N, K, lda, ldc, parts.len);
    return infero_check_launch("gemm_tiled");
}

// The tile.  Few rows: a block streams rows of W past all rows of A; where N is small, few rows of W a block and a block per part
// of K, so that every multiprocessor streams some and no chain is long (us, before one block ran one chain over all of K: 1 x 896,
// K = 4,864 25 and 8.4; 8 rows 33 and 13; 1 x 1,152, K = 896 6.8 and 6.3); where N alone gives four blocks a multiprocessor, all
// parts to a block (8 x 151,936, K = 896 132, split 146; before 228).  Many rows: the largest tile that gives three blocks a
// multiprocessor, 64 rows only where they are not much more than 32 would be (301 x 896, K = 4,864: 148 before, 73 with 64 x 64,
// 104 with 32 x 64; 301 x 9,728, K = 896: 156 before, 138 and 141; 150 x 9,728 121 before, 93 with 32 x 64; 301 x 1,152 35 before,
// 29 with 32 x 32, 31 with 32 x 64; 64 x 896 14.5 before, 12.4 with four results a thread, 14.4 with eight).  In large products
// (2,048 x 9,728, K = 896: 857 before, 795 now) the bound is the rate of the paired multiply-adds, 0.6 of it reached.
// Where blocks are few (few rows of W, and of K one part, two, or more than a cluster has blocks), a tile with fewer results a
// thread (us before parts, with the larger tile, now: 16 x 512, K = 512 4.6, 5.5, 3.9; 16 x 1,152, K = 896 7.1, 7.3, 6.2; 16 x 200, K = 5,124
// 33, 41, 27; 64 x 200 60, 65, 41; 17 x 2,048, K = 6,144 73, 77, 68; 16 x 2,048, K = 6,144 with 8 x 16 51, with 16 x 16 50).
template <bool VEC, typename TA, typename TW, typename TC>
int launch_tiled(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N,
                 int K, int lda, int ldc, cudaStream_t stream) {
    // (operands that are widened on the way come with all parts to a block)
#define TILE(...)                                                                                                                      \
    do {                                                                                                                               \
        if constexpr (VEC)                                                                                                             \
            if (split) return launch_tile<__VA_ARGS__, true, VEC, TA, TW, TC>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);   \
        return launch_tile<__VA_ARGS__, false, VEC, TA, TW, TC>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);                 \
    } while (0)
    const int parts = parts_of(K).n, sms = infero_sm_count();
    bool split = VEC && parts >= 2 && parts <= MAX_SPLIT;
    const int by = split ? parts : 1;
    auto blocks = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    // Operands that are widened on the way have no copies in flight while a block works, so what counts is that many threads load.
    // (us before K came in parts, with tiles for 16-byte copies, now; bf16 on both sides but for the rows of 897 and 4,865 32-bit columns:
    // 8 x 896, K = 896 24, 37, 11; 8 x 896, K = 4,865 121, 191, 41; 4 x 32,000, K = 896 126, 126, 47; 16 x 6,144, K = 2,048 93, 91, 48;
    // 64 x 2,048, K = 2,048 116, 137, 52; 150 x 896, K = 4,864 215, 324, 126; 301 x 9,728, K = 897 210, 242, 198; 2,048 x 9,728, K = 896 1,221,
    // 1,311, 1,064.  Wider tiles at 64 x 9,728: 65 against 59; 16 x 32 for 301 x 896, K = 4,864: above 197 against 186.)
    if constexpr (!VEC) {
        if (M <= 16) {
            if (blocks(16, 64) >= 2 * sms) TILE(16, 64, 4, 2, 64, 2);
            if (M <= 8 || blocks(8, 16) < 2 * sms) TILE(8, 16, 1, 1, 64, 4);
            TILE(16, 16, 2, 1, 64, 4);
        }
        if (blocks(64, 64) >= sms && (M + 63) / 64 * 64 <= (M + 31) / 32 * 35) TILE(64, 64, 4, 4, 32, 2);
        if (5 * blocks(32, 32) >= 8 * sms) TILE(32, 32, 4, 2, 32, 3);
        TILE(32, 16, 2, 1, 64, 3);
    } else {
        if (M <= 16) {
            const bool narrow = blocks(16, 32) < 2 * sms;
            split = split && blocks(16, 32) < 4 * sms;
            if (M == 1 && narrow && split) TILE(1, 16, 1, 1, 128, 4);
            if (M == 1 && narrow) TILE(1, 8, 1, 1, 128, 6);
            if (M == 1) TILE(1, 32, 1, 1, 64, 4);
            if (M <= 4 && narrow) TILE(4, 8, 1, 1, 128, 4);
            if (M <= 4) TILE(4, 32, 4, 1, 64, 4);
            if (M <= 8 && narrow) TILE(4, 16, 2, 1, 64, 5);
            if (M <= 8) TILE(8, 32, 4, 1, 64, 3);
            if (narrow && blocks(8, 16) * by < (split ? 2 : 1) * sms) TILE(8, 16, 1, 1, 64, 4);
            if (narrow) TILE(16, 16, 2, 1, 64, 4);
            TILE(16, 32, 4, 1, 64, 3);
        }
        if (blocks(64, 64) * by >= 3 * sms && (M + 63) / 64 * 64 <= (M + 31) / 32 * 35) TILE(64, 64, 8, 4, 32, 2);
        if (blocks(32, 64) * by >= 3 * sms) TILE(32, 64, 4, 4, 32, 3);
        if (blocks(32, 32) * by >= sms) TILE(32, 32, 4, 2, 32, 3);
        if (3 * blocks(32, 32) * by >= 2 * sms) TILE(32, 32, 2, 2, 32, 3);
        if (!split) TILE(16, 16, 2, 1, 64, 4);
        TILE(32, 16, 2, 1, 32, 4);
    }
#undef TILE
}

// 16-byte copies: 32-bit operands whose rows all start on 16 bytes
template <typename TC>
int launch_f32(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N,
               int K, int lda, int ldc, cudaStream_t stream) {
    if (K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0)
        return launch_tiled<true, float, float, TC>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
    return launch_tiled<false, float, float, TC>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
}

}  // namespace

extern "C" {

// Any of A, W, C may be float or bf16; accumulation is 32-bit in an order that depends on K alone.
int infero_gemm_tiled(const void* A, int a_dtype, const void* W, int w_dtype, const void* bias,
                      int bias_dtype, void* C, int c_dtype, int M, int N, int K, int lda, int ldc,
                      cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    INFERO_REQUIRE(K > 0 && lda >= K && ldc >= N, "gemm_tiled: bad sizes M=%d N=%d K=%d lda=%d ldc=%d", M, N, K, lda, ldc);
    INFERO_REQUIRE((M + 63) / 64 <= 65535, "gemm_tiled: M=%d too large", M);
    const int key = a_dtype * 4 + w_dtype * 2 + c_dtype;
    switch (key) {
        case 0: return launch_f32<float>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 1: return launch_f32<bf16>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 2: return launch_tiled<false, float, bf16, float>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 3: return launch_tiled<false, float, bf16, bf16>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 4: return launch_tiled<false, bf16, float, float>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 5: return launch_tiled<false, bf16, float, bf16>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 6: return launch_tiled<false, bf16, bf16, float>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
        case 7: return launch_tiled<false, bf16, bf16, bf16>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream);
    }
    infero_set_error("gemm_tiled: unknown dtype tags %d %d %d", a_dtype, w_dtype, c_dtype);
    return 1;
}

// bf16 x bf16, 1 <= M <= 4, K % 8 == 0, A rows and W 16-byte aligned.
int infero_gemm_skinny(const void* A, const void* W, const void* bias, int bias_dtype, void* C,
                       int c_dtype, int M, int N, int K, int lda, int ldc, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    INFERO_REQUIRE(M >= 1 && M <= 4, "gemm_skinny: M=%d outside 1..4", M);
    INFERO_REQUIRE(K > 0 && K % 8 == 0 && lda % 8 == 0, "gemm_skinny: K=%d and lda=%d must be multiples of 8", K, lda);
    INFERO_REQUIRE(((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0, "gemm_skinny: operands must be 16-byte aligned");
    const int blocks = (N + 8 * SK_ROWS - 1) / (8 * SK_ROWS);
#define LAUNCH(MT)                                                                                       \
    do {                                                                                                 \
        if (c_dtype == INFERO_F32)                                                                       \
            gemm_skinny_kernel<MT, float><<<blocks, 256, 0, stream>>>((const bf16*)A, (const bf16*)W, bias, \
                                                                      bias_dtype, (float*)C, M, N, K, lda, ldc); \
        else                                                                                             \
            gemm_skinny_kernel<MT, bf16><<<blocks, 256, 0, stream>>>((const bf16*)A, (const bf16*)W, bias, \
                                                                     bias_dtype, (bf16*)C, M, N, K, lda, ldc); \
    } while (0)
    if (M == 1) LAUNCH(1);
    else if (M == 2) LAUNCH(2);
    else LAUNCH(4);
#undef LAUNCH
    return infero_check_launch("gemm_skinny");
}

}  // extern "C"
