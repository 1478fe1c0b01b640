// Matrix products on the ordinary cores: out[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
//
//  * gemm_tiled: any shape, any mix of float / bf16 operands, 32-bit accumulation with one
//    fused multiply-add per k in ascending k.  The value of out[m,n] therefore does not
//    depend on M, on the tile it falls in or on its batch-mates: this is the product of the
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
// tx + j * (BN / TN), so that eight neighbouring lanes read eight neighbouring rows, whose starts lie 4 banks apart
// (BK + 4 is an odd multiple of 4): no bank conflict.  Operands that 16-byte copies cannot take (bf16, rows that
// start anywhere) come by plain loads into the same ring.
// Every result is one chain of fused multiply-adds in ascending k whatever the tile, so the choice of a tile never
// shows in the numbers.
template <int BM, int BN, int TM, int TN, int BK, int STAGES>
struct Tile {
    static constexpr int TX = BN / TN, TY = BM / TM, WORK = TX * TY, THREADS = WORK < 32 ? 32 : WORK;
    static constexpr int LD = BK + 4, A_FLOATS = BM * LD, STAGE = (BM + BN) * LD;
    static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float);
    static_assert(SMEM <= 48 * 1024, "more shared memory than a launch gets without asking");
    static_assert(BK % 4 == 0 && (BK / 4) % 2 == 0, "");
};

__device__ __forceinline__ void copy16(float* dst, const float* src, bool ok) {
    const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
    const int bytes = ok ? 16 : 0;                          // (nothing is read of a row that is not there: zeros)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// ROWS rows of BK columns from column k0 on
template <int ROWS, int BK, int LD, int THREADS, bool VEC, typename T>
__device__ __forceinline__ void fill(float* dst, const T* src, int row0, int n_rows, int k0, int K, long long ld, int tid) {
    if constexpr (VEC) {
        constexpr int Q = BK / 4;
        for (int e = tid; e < ROWS * Q; e += THREADS) {
            const int r = e / Q, k = k0 + (e % Q) * 4;
            const bool ok = row0 + r < n_rows && k < K;     // (K is a multiple of 4 here)
            copy16(dst + r * LD + (e % Q) * 4, ok ? src + (long long)(row0 + r) * ld + k : src, ok);
        }
    } else {
        for (int e = tid; e < ROWS * BK; e += THREADS) {
            const int r = e / BK, k = k0 + e % BK;
            dst[r * LD + e % BK] = row0 + r < n_rows && k < K ? to_f32(src[(long long)(row0 + r) * ld + k]) : 0.f;
        }
    }
}

template <typename TL, int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC, typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(TL::THREADS)
gemm_tiled_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const void* __restrict__ bias,
                  int bias_dtype, TC* __restrict__ C, int M, int N, int K, int lda, int ldc) {
    extern __shared__ float4 ring4[];
    float* ring = reinterpret_cast<float*>(ring4);
    constexpr int LD = TL::LD;
    const int tid = threadIdx.x;
    const int ty = tid / TL::TX, tx = tid % TL::TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const bool works = TL::WORK == TL::THREADS || tid < TL::WORK;
    const int n_stages = (K + BK - 1) / BK;
    auto load = [&](int s) {
        if (s < n_stages) {
            float* at = ring + (s % STAGES) * TL::STAGE;
            fill<BM, BK, LD, TL::THREADS, VEC>(at, A, m0, M, s * BK, K, lda, tid);
            fill<BN, BK, LD, TL::THREADS, VEC>(at + TL::A_FLOATS, W, n0, N, s * BK, K, K, tid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int s = 0; s < STAGES - 1; ++s) load(s);
    for (int s = 0; s < n_stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                    // stage s is here, and everyone is done with stage s - 1,
        load(s + STAGES - 1);                               // whose place this fills
        if (!works) continue;
        const float* a_s = ring + (s % STAGES) * TL::STAGE + ty * LD;
        const float* w_s = ring + (s % STAGES) * TL::STAGE + TL::A_FLOATS + tx * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(w_s + j * TL::TX * LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + i * TL::TY * LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
                }
            }
        }
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
            float v = acc[i][j];
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

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC, typename TA, typename TW, typename TC>
int launch_tile(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N,
                int K, int lda, int ldc, cudaStream_t stream) {
    using TL = Tile<BM, BN, TM, TN, BK, STAGES>;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    gemm_tiled_kernel<TL, BM, BN, TM, TN, BK, STAGES, VEC, TA, TW, TC><<<grid, TL::THREADS, TL::SMEM, stream>>>(
        (const TA*)A, (const TW*)W, bias, bias_dtype, (TC*)C, M, N, K, lda, ldc);
    return infero_check_launch("gemm_tiled");
}

// The tile.  Few rows: a block streams rows of W past all rows of A; where N is small, few rows of W a block, so that every
// SM streams some (1 x 896, K = 4,864: 25 us with 8 rows of W a block, 37 with 16, 47 with 32; the chain alone is 10).  Many
// rows: the largest tile that still gives nearly every SM a block (301 x 9,728, K = 896: 157 us with 64 x 128, 178 with
// 64 x 64; 301 x 896, K = 4,864: 144 with 32 x 32, 166 with twice the results a thread; 64 x 896: 60 with 32 x 16, 112 with
// 32 x 32).  In large products the bound is the rate at which shared memory feeds the multiply-adds (42 TFLOP/s of the 74 that
// the cores have; pairs of multiply-adds in one instruction need more moves than they save: 1,160 against 840 us at
// 2,048 x 9,728).  Before, with one 64 x 64 tile and loads waited for in place: 1 x 896, K = 4,864 342 us, 301 x 9,728 285 us,
// 2,048 x 9,728 1,512 us, 1 x 151,936 782 us (now 95: 5.7 TB/s).
template <bool VEC, typename TA, typename TW, typename TC>
int launch_tiled(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N,
                 int K, int lda, int ldc, cudaStream_t stream) {
#define TILE(...) return launch_tile<__VA_ARGS__, VEC, TA, TW, TC>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, stream)
    const int enough = infero_sm_count() * 7 / 8;
    auto blocks = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    if (M <= 16) {
        const bool narrow = blocks(16, 32) < 2 * enough;
        if (M == 1 && narrow) TILE(1, 8, 1, 1, 128, 6);
        if (narrow) TILE(16, 8, 1, 1, 64, 4);
        if (M == 1) TILE(1, 32, 1, 1, 64, 4);
        if (M <= 4) TILE(4, 32, 4, 1, 64, 4);
        TILE(16, 32, 4, 1, 64, 3);
    }
    if (blocks(64, 128) >= enough) TILE(64, 128, 8, 8, 16, 3);
    if (blocks(32, 32) >= enough) TILE(32, 32, 4, 2, 32, 3);
    TILE(32, 16, 2, 1, 32, 4);
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

// Any of A, W, C may be float or bf16; accumulation is 32-bit in ascending k.
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
