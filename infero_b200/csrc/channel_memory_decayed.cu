// Gated linear attention: the scan's instances (channel_memory.cuh).  Its records come from low_rank.cu.
#include "channel_memory.cuh"

namespace {

using namespace memory;

// starts holds the segments' ends from an empty state and receives their starts; an element a thread, the ends of a few segments
// on their way ahead of the chain.
__global__ void __launch_bounds__(256)
chain_segments_kernel(const Segments seg, const float* __restrict__ state, long long state_stride, long long s_off,
                      const int* __restrict__ entry_q_len, const int* __restrict__ entry_slot, int H, int W, int K) {
    const int e = blockIdx.x, h = blockIdx.y, i = blockIdx.z * blockDim.x + threadIdx.x;
    const int count = segments_of(entry_q_len[e], seg.len);
    if (count == 1 || i >= W * K) return;
    int slot = 0;
    for (int b = 0; b < e; ++b) {
        const int c = segments_of(entry_q_len[b], seg.len);
        if (c > 1) slot += c;
    }
    const size_t step = (size_t)H * W * K, t_step = (size_t)H * K;
    float* p = seg.starts + ((size_t)slot * H + h) * W * K + i;
    const float* d = seg.totals + ((size_t)slot * H + h) * K + i % K;
    float S = state[(long long)entry_slot[e] * state_stride + s_off + (size_t)h * W * K + i];
    constexpr int AHEAD = 8;
    for (int s0 = 0; s0 < count; s0 += AHEAD) {
        float end[AHEAD], dec[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (s0 + k < count - 1) end[k] = p[(s0 + k) * step], dec[k] = d[(s0 + k) * t_step];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (s0 + k < count) {
                p[(s0 + k) * step] = S;
                if (s0 + k < count - 1) S = fmaf(dec[k], S, end[k]);
            }
    }
}

}  // namespace

int memory::chain_segments(const Segments& seg, const float* state, long long state_stride, long long s_off, const int* entry_q_len,
                           const int* entry_slot, int n_entries, int H, int W, int K, cudaStream_t stream) {
    const unsigned blocks = (unsigned)(((long long)W * K + 255) / 256);
    INFERO_REQUIRE(blocks <= 65535, "chain_segments: a state of %d x %d", W, K);
    chain_segments_kernel<<<dim3(n_entries, H, blocks), 256, 0, stream>>>(seg, state, state_stride, s_off, entry_q_len, entry_slot, H, W, K);
    return infero_check_launch("chain_segments");
}

extern "C" {

// segment_len > 0 (portions; a multiple of 16): portions longer than that run in segments of it, n_segments in all (a shorter portion
// counts as one); starts [segments of the longer ones, H, V, K] and totals [the same, H, K] are scratch, 16-byte aligned.
// rec [H, T, 3 Kp]; y [T, H V] receives S^T q times q_scale; S [H, V, K] at s_off of the requests' state moves on.
int infero_decayed_scan(const float* rec, int n_tokens, const float* v, long long v_stride, float q_scale, float* state,
                        long long state_stride, long long s_off, const int* entry_q_start, const int* entry_q_len, const int* entry_slot,
                        float* y, int n_entries, int single, int H, int K, int V, int segment_len, int n_segments, float* starts,
                        float* totals, int sm_count, cudaStream_t stream) {
    INFERO_REQUIRE(segment_len >= 0 && segment_len % 16 == 0 && (!segment_len || (starts && totals && memory::al16(starts) && n_segments >= n_entries)),
                   "decayed_scan: segments of %d, %d of them", segment_len, n_segments);
    return memory::channel_scan<false>(rec, n_tokens, v, v_stride, state, state_stride, s_off, entry_q_start, entry_q_len, entry_slot, y,
                                       q_scale, n_entries, single, H, K, V, sm_count, stream, memory::Segments{segment_len, starts, totals}, n_segments);
}

}  // extern "C"
