// Layer norm, and a residual kept as several streams ("hyper-connections").
//
// layer norm (weight, no bias):  h = (v - mean(v)) / sqrt(mean((v - mean(v))^2) + eps) * w, v = x (+ delta), all
//   32-bit, the variance from the deviations (two passes over the row, which sits in shared memory).
//
// streams: the residual of a token is S vectors xs[s] of width d (float32 [T, S, d]).  A sublayer reads
//   u = sum_s a[s] xs[s], works on h = norm(u), and its result y updates all streams at once from the old ones,
//   xs'[r] = sum_s m[s, r] xs[s] + b[r] y.  One kernel does the update of the sublayer before (if y is given) and the
//   read-out and norm for the sublayer after (if a is given): one pass over a token's streams per sublayer, as
//   the single-stream blocks have one pass for add + norm.  Without a norm weight the read-out is written as it is
//   (float32): the sum of the streams at the end of the model is a read-out with a = 1.
// The small vectors a, b, m are float32 on both precisions.  One block per token; nothing depends on the batch.
#include "common.cuh"

namespace {

constexpr int THREADS = 256;          // per token in steps of many tokens
constexpr int THREADS_FEW = 1024;     // in steps of few tokens, where a block's own latency is what counts
constexpr int THREADS_VEC = 512;      // at most, four columns a thread at a time
constexpr int MAX_STREAMS = 8;

// the row v[0..d) in shared memory -> out = layer norm(v) * w
template <typename OutT>
__device__ __forceinline__ void layernorm_row(const float* v, const float* __restrict__ w, float eps, OutT* __restrict__ out,
                                              int d, float* red) {
    float s = 0.f;
    for (int i = threadIdx.x; i < d; i += blockDim.x) s += v[i];
    const float mean = block_sum(s, red) / (float)d;
    float q = 0.f;
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        const float c = v[i] - mean;
        q = fmaf(c, c, q);
    }
    const float rstd = 1.0f / sqrtf(block_sum(q, red) / (float)d + eps);
    for (int i = threadIdx.x; i < d; i += blockDim.x) out[i] = from_f32<OutT>((v[i] - mean) * rstd * w[i]);
}

template <typename OutT>
__global__ void __launch_bounds__(THREADS_FEW)
add_layernorm_kernel(float* __restrict__ x, const float* __restrict__ delta, const float* __restrict__ w, float eps,
                     OutT* __restrict__ out, const int* __restrict__ rows, int d) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float row[];
    __shared__ float red[32];
    const size_t t = rows ? (size_t)rows[blockIdx.x] : (size_t)blockIdx.x;
    float* xr = x + t * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float v = xr[i];
        if (delta) {
            v += delta[t * d + i];
            if (!rows) xr[i] = v;
        }
        row[i] = v;
    }
    __syncthreads();
    layernorm_row(row, w, eps, out + (size_t)blockIdx.x * d, d, red);
}

template <typename OutT>
__global__ void __launch_bounds__(THREADS_FEW)
hyper_step_kernel(float* __restrict__ xs, const float* __restrict__ y, int y_stride, int y_splits, long long y_split_stride,
                  const float* __restrict__ mix,
                  const float* __restrict__ w_out, const float* __restrict__ w_in, const float* __restrict__ norm_w,
                  float eps, OutT* __restrict__ h_out, float* __restrict__ u_out, const int* __restrict__ rows, int S, int d) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float row[];
    __shared__ float red[32];
    __shared__ float m_s[MAX_STREAMS * MAX_STREAMS], b_s[MAX_STREAMS], a_s[MAX_STREAMS];
    if (threadIdx.x < S * S && y) m_s[threadIdx.x] = mix[threadIdx.x];
    if (threadIdx.x < S) {
        if (y) b_s[threadIdx.x] = w_out[threadIdx.x];
        a_s[threadIdx.x] = w_in ? w_in[threadIdx.x] : 1.0f;
    }
    __syncthreads();
    const size_t t = rows ? (size_t)rows[blockIdx.x] : (size_t)blockIdx.x;
    float* xt = xs + t * S * d;
    const bool read_out = w_in || u_out || norm_w;       // (without w_in: the plain sum of the streams)
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float v[MAX_STREAMS];
#pragma unroll
        for (int s = 0; s < MAX_STREAMS; ++s) v[s] = s < S ? xt[(size_t)s * d + i] : 0.f;
        if (y) {
            float yv = y[t * y_stride + i];
            for (int k = 1; k < y_splits; ++k) yv += y[(size_t)k * y_split_stride + t * y_stride + i];     // ascending order
            float nv[MAX_STREAMS];
#pragma unroll
            for (int r = 0; r < MAX_STREAMS; ++r) {
                float acc = 0.f;
                if (r < S) {
#pragma unroll
                    for (int s = 0; s < MAX_STREAMS; ++s)
                        if (s < S) acc = fmaf(m_s[s * S + r], v[s], acc);
                    acc = fmaf(b_s[r], yv, acc);
                    xt[(size_t)r * d + i] = acc;
                }
                nv[r] = acc;
            }
#pragma unroll
            for (int s = 0; s < MAX_STREAMS; ++s) v[s] = nv[s];
        }
        if (read_out) {
            float u = 0.f;
#pragma unroll
            for (int s = 0; s < MAX_STREAMS; ++s)
                if (s < S) u = fmaf(a_s[s], v[s], u);
            if (norm_w) row[i] = u;
            else u_out[(size_t)blockIdx.x * d + i] = u;
        }
    }
    if (!read_out || !norm_w) return;
    __syncthreads();
    layernorm_row(row, norm_w, eps, h_out + (size_t)blockIdx.x * d, d, red);
}

// Rows of whole 16-byte pieces (d, strides and addresses): a thread takes four neighbouring columns of all streams at a time, all
// loads of a piece ahead of its arithmetic, and keeps its NI pieces of the read-out in registers for the norm.  What bounds it is
// the streams' traffic: 2,048 tokens of four streams of 2,048 are 159 MB (24 us at the copy rate), 48 us an element at a time, 30 in pieces; a pass of
// nine such steps among its products takes 1.70 ms with those and 1.52 with these, launched early.
template <int S, int NI, typename OutT>
__global__ void __launch_bounds__(THREADS_VEC)
hyper_step_vec_kernel(float* __restrict__ xs, const float* __restrict__ y, int y_stride, int y_splits, long long y_split_stride,
                      const float* __restrict__ mix, const float* __restrict__ w_out, const float* __restrict__ w_in,
                      const float* __restrict__ norm_w, float eps, OutT* __restrict__ h_out, float* __restrict__ u_out,
                      const int* __restrict__ rows, int d) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    float m[S][S], b[S], a[S];
#pragma unroll
    for (int r = 0; r < S; ++r) {
        a[r] = w_in ? w_in[r] : 1.0f;
        b[r] = y ? w_out[r] : 0.f;
#pragma unroll
        for (int q = 0; q < S; ++q) m[r][q] = y ? mix[r * S + q] : 0.f;
    }
    const size_t t = rows ? (size_t)rows[blockIdx.x] : (size_t)blockIdx.x;
    const int d4 = d / 4;
    float4* xt = reinterpret_cast<float4*>(xs + t * S * d);
    const bool read_out = w_in || u_out || norm_w;       // (without w_in: the plain sum of the streams)
    float u[NI][4];
    float sum = 0.f;
#pragma unroll
    for (int n = 0; n < NI; ++n) {
        const int i = n * blockDim.x + threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; ++k) u[n][k] = 0.f;
        if (i >= d4) continue;
        float v[S][4];
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const float4 f = xt[(size_t)r * d4 + i];
            v[r][0] = f.x, v[r][1] = f.y, v[r][2] = f.z, v[r][3] = f.w;
        }
        if (y) {
            const float* yr = y + t * y_stride + 4 * i;
            float4 f = *reinterpret_cast<const float4*>(yr);
            for (int k = 1; k < y_splits; ++k) {                     // ascending order
                const float4 g = *reinterpret_cast<const float4*>(yr + (size_t)k * y_split_stride);
                f.x += g.x, f.y += g.y, f.z += g.z, f.w += g.w;
            }
            const float yv[4] = {f.x, f.y, f.z, f.w};
            float nv[S][4];
#pragma unroll
            for (int r = 0; r < S; ++r) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float acc = 0.f;
#pragma unroll
                    for (int q = 0; q < S; ++q) acc = fmaf(m[q][r], v[q][k], acc);
                    nv[r][k] = fmaf(b[r], yv[k], acc);
                }
                xt[(size_t)r * d4 + i] = make_float4(nv[r][0], nv[r][1], nv[r][2], nv[r][3]);
            }
#pragma unroll
            for (int r = 0; r < S; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k) v[r][k] = nv[r][k];
        }
        if (read_out) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
#pragma unroll
                for (int r = 0; r < S; ++r) u[n][k] = fmaf(a[r], v[r][k], u[n][k]);
                sum += u[n][k];
            }
            if (!norm_w) reinterpret_cast<float4*>(u_out + (size_t)blockIdx.x * d)[i] = make_float4(u[n][0], u[n][1], u[n][2], u[n][3]);
        }
    }
    if (!norm_w) return;                                 // (uniform)
    const float mean = block_sum(sum, red) / (float)d;
    float sq = 0.f;
#pragma unroll
    for (int n = 0; n < NI; ++n)
        if (n * (int)blockDim.x + (int)threadIdx.x < d4)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float c = u[n][k] - mean;
                sq = fmaf(c, c, sq);
            }
    const float rstd = 1.0f / sqrtf(block_sum(sq, red) / (float)d + eps);
    OutT* out = h_out + (size_t)blockIdx.x * d;
#pragma unroll
    for (int n = 0; n < NI; ++n) {
        const int i = n * blockDim.x + threadIdx.x;
        if (i >= d4) continue;
        const float4 w = reinterpret_cast<const float4*>(norm_w)[i];
        const float h[4] = {(u[n][0] - mean) * rstd * w.x, (u[n][1] - mean) * rstd * w.y, (u[n][2] - mean) * rstd * w.z, (u[n][3] - mean) * rstd * w.w};
        if constexpr (sizeof(OutT) == 4) {
            reinterpret_cast<float4*>(out)[i] = make_float4(h[0], h[1], h[2], h[3]);
        } else {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(h[0], h[1]), hi = __floats2bfloat162_rn(h[2], h[3]);
            uint2 p;
            p.x = *reinterpret_cast<const uint32_t*>(&lo), p.y = *reinterpret_cast<const uint32_t*>(&hi);
            reinterpret_cast<uint2*>(out)[i] = p;
        }
    }
}

__global__ void streams_fill_kernel(const float* __restrict__ x, float* __restrict__ xs, int S, int d) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        const float v = x[t * d + i];
        for (int s = 0; s < S; ++s) xs[(t * S + s) * d + i] = v;
    }
}

}  // namespace

extern "C" {

// x float32 [T, d] (+= delta float32 [T, d] if given; with `rows` x is left as it is); out [n, d] = layer norm of rows.
int infero_add_layernorm(float* x, const float* delta, const float* w, float eps, void* out, int out_dtype,
                         const int* rows, int n, int d, cudaStream_t stream) {
    if (n == 0) return 0;
    const size_t sh = (size_t)d * sizeof(float);
    INFERO_REQUIRE(d >= 1 && sh <= 48 * 1024, "layer norm: width %d outside 1..12288", d);
    const int threads = n <= 64 && d > THREADS ? THREADS_FEW : THREADS;
    if (out_dtype == INFERO_F32)
        launch_pdl(add_layernorm_kernel<float>, dim3(n), dim3(threads), sh, stream, x, delta, w, eps, (float*)out, rows, d);
    else
        launch_pdl(add_layernorm_kernel<bf16>, dim3(n), dim3(threads), sh, stream, x, delta, w, eps, (bf16*)out, rows, d);
    return infero_check_launch("add_layernorm");
}

// xs float32 [T, S, d].  y (float32, row stride y_stride; or y_splits partial sums of a product, y_split_stride elements
// apart, added up here) with mix [S, S] (from, to) and w_out [S]: update the streams.
// w_in [S] with norm_w [d]: h_out [n, d] = layer norm(sum_s w_in[s] xs[s]) * norm_w.  norm_w null: u_out float32 [n, d]
// = sum_s w_in[s] xs[s] (w_in null: the plain sum).  rows (or null): the tokens to work on, n of them.
int infero_hyper_step(float* xs, const float* y, int y_stride, int y_splits, long long y_split_stride, const float* mix,
                      const float* w_out, const float* w_in,
                      const float* norm_w, float eps, void* h_out, int h_dtype, float* u_out, const int* rows, int n,
                      int S, int d, cudaStream_t stream) {
    if (n == 0) return 0;
    const size_t sh = (size_t)d * sizeof(float);
    INFERO_REQUIRE(S >= 1 && S <= MAX_STREAMS, "hyper-connections: %d streams outside 1..%d", S, MAX_STREAMS);
    INFERO_REQUIRE(d >= 1 && sh <= 48 * 1024, "hyper-connections: width %d outside 1..12288", d);
    INFERO_REQUIRE(!y || (mix && w_out && y_splits >= 1), "hyper-connections: an update needs its mix matrix and output weights");
    INFERO_REQUIRE(!norm_w || h_out, "hyper-connections: a norm needs somewhere to write");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if ((S == 2 || S == 4) && d % 4 == 0 && d <= 8192 && y_stride % 4 == 0 && y_split_stride % 4 == 0 && al16(xs) && al16(y) && al16(norm_w) &&
        al16(h_out) && al16(u_out)) {
        // few tokens: a piece a thread; many: as few threads as leave each at most four pieces
        int threads = n <= 64 || d > 4096 ? THREADS_VEC : THREADS;
        if (threads > d / 4) threads = (d / 4 + 31) / 32 * 32;
        const int pieces = (d / 4 + threads - 1) / threads;
#define VEC(S_, N_)                                                                                                                   \
    do {                                                                                                                              \
        if (h_dtype == INFERO_F32)                                                                                                    \
            launch_pdl(hyper_step_vec_kernel<S_, N_, float>, dim3(n), dim3(threads), 0, stream, xs, y, y_stride, y_splits, y_split_stride, \
                       mix, w_out, w_in, norm_w, eps, (float*)h_out, u_out, rows, d);                                                 \
        else                                                                                                                          \
            launch_pdl(hyper_step_vec_kernel<S_, N_, bf16>, dim3(n), dim3(threads), 0, stream, xs, y, y_stride, y_splits, y_split_stride, \
                       mix, w_out, w_in, norm_w, eps, (bf16*)h_out, u_out, rows, d);                                                  \
    } while (0)
        if (S == 4) {
            if (pieces == 1) VEC(4, 1);
            else if (pieces == 2) VEC(4, 2);
            else VEC(4, 4);
        } else {
            if (pieces == 1) VEC(2, 1);
            else if (pieces == 2) VEC(2, 2);
            else VEC(2, 4);
        }
#undef VEC
        return infero_check_launch("hyper_step");
    }
    const int threads = n <= 64 && d > THREADS ? THREADS_FEW : THREADS;
    if (h_dtype == INFERO_F32)
        launch_pdl(hyper_step_kernel<float>, dim3(n), dim3(threads), sh, stream, xs, y, y_stride, y_splits, y_split_stride, mix, w_out, w_in, norm_w, eps,
                                                           (float*)h_out,
                                                           u_out, rows, S, d);
    else
        launch_pdl(hyper_step_kernel<bf16>, dim3(n), dim3(threads), sh, stream, xs, y, y_stride, y_splits, y_split_stride, mix, w_out, w_in, norm_w, eps,
                                                          (bf16*)h_out,
                                                          u_out, rows, S, d);
    return infero_check_launch("hyper_step");
}

int infero_streams_fill(const float* x, float* xs, int n, int S, int d, cudaStream_t stream) {
    if (n == 0) return 0;
    launch_pdl(streams_fill_kernel, dim3(n), dim3(THREADS), 0, stream, x, xs, S, d);
    return infero_check_launch("streams_fill");
}

}  // extern "C"
