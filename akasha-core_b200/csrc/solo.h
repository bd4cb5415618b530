// Batch-1 decode step as one persistent kernel (solo.cu): launch interface.
#pragma once
#include "kernels.h"

namespace ak {

constexpr uint32_t SOLO_MAX_SPLITS = 4;   // CTAs a head's positions are divided over

struct SoloLayer {   // device array, one per layer; matrices [out, in]
    const float* norm_1;
    const void* qkv;
    const void* out;
    const float* norm_2;
    const void* up;
    const void* down;
    void* k_pool;                // block i of the pools holds positions 16 i .. 16 i + 15 of the sequence
    void* v_pool;
};

struct SoloArgs {
    const SoloLayer* layers;
    const void* embedding;
    const float* final_norm;
    const void* lm_head;
    const float2* rope;          // [rope_len][head_dim / 2] (cos, sin)
    uint64_t* xch;               // solo_xch_words() 64-bit words, zero before the first launch
    uint32_t* sampled;           // device word: the token fed back when tok_src < 0, overwritten by the greedy pick
    float* logits;               // [vocab] device, or nullptr
    float* logits_host;          // [vocab] mapped host memory, or nullptr
    uint64_t* done_host;         // mapped host word {token, or solo::STEP_FAILED; step}: written after everything else, or nullptr
    uint32_t n_layers, dim, ffn, heads, vocab;
    uint32_t pos;                // position of the token fed in; positions 0 .. pos are attended to
    int32_t tok_src;             // >= 0 literal id; < 0: *sampled
    uint32_t step;               // non-zero, different for every launch on the same xch
    float eps, scale;
};

#ifdef __CUDACC__
// Weights that a decode step reads. Where they take no more than half of the L2 they are left in it for the next step; larger models stream through it
// (evict-first: 162M model, 8 / 32 sequences 162 / 295 us a step, 165 / 300 without; 320-wide model, 52 MB, 21 sequences 123.7, 120.4 without; 64 tokens of
// one in bf16 7.64, 7.49 ms).
__host__ __device__ inline uint64_t step_weight_bytes(uint32_t esz, uint32_t dim, uint32_t ffn, uint32_t n_layers, uint32_t vocab) {
    return ((uint64_t)n_layers * (4ull * dim + 2ull * ffn) * dim + (uint64_t)vocab * dim) * esz;
}
__host__ __device__ inline bool stays_in_l2(uint64_t bytes) { return bytes <= 64ull << 20; }
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
#endif

bool solo_supported(uint32_t dtype, uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers, uint32_t vocab);
size_t solo_xch_words(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers);
int launch_solo(cudaStream_t st, uint32_t dtype, const SoloArgs& a);
int solo_status(unsigned int* out);

}  // namespace ak
