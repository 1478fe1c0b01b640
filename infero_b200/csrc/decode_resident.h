// What the resident decode kernel (decode_resident.cu) takes from the native launcher (host_block.cpp).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

constexpr int RESIDENT_LAYERS = 48;      // layers a launch takes (their descriptors are kernel parameters)

struct ResidentLayer {
    const __nv_bfloat16 *w_qkv, *w_o, *w_gate_up, *w_down;      // w_gate_up: rows alternate gate_j, up_j
    const void *b_qkv, *b_o, *norm_mixer, *norm_ffn;            // biases may be null
    const float* inv_freq;
    __nv_bfloat16 *k_cache, *v_cache;
    const int* table;                                           // block table of the layer's group
    float eps_mixer, eps_ffn, scale_log2;
    int window;
};

// Sizes are the same for all layers of a launch.
struct ResidentStep {
    int n_tok, n_layers, hidden, n_heads, n_kv, ff, rotary_dim, page_size, max_blocks;
    int norm_dtype, qkv_bias_dtype, o_bias_dtype;
    float inv_hidden;
    const int *positions, *tok_entry;
    float* x;                            // residual stream [n_tok, hidden]
    // scratch (infero_resident_scratch), values beside tags: h, sums [0] of the first norm, [1] of the second
    uint32_t* h[2];
    uint2* sums[2];
    uint2* qkv;
    uint32_t *attn, *act;
    float *part_o, *part_ml;
    unsigned int* stop;                  // a block has given up
    int* counters;                       // arrivals per (layer, token, kv head)
};

extern "C" {
long long infero_resident_scratch(ResidentStep* s, uint8_t* at, int head_dim, int blocks);
int infero_resident_supported(const ResidentStep* s, int head_dim, int blocks);
int infero_resident_worth(const ResidentStep* s, int head_dim, int blocks, int visible);
int infero_decode_resident(const ResidentStep* s, const ResidentLayer* layers, int head_dim, const int* num_pages, const void* embed,
                           int embed_dtype, const int* ids, const int* device_tokens, int vocab, float embed_scale, int blocks,
                           cudaStream_t stream);
}
