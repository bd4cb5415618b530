// Decode step of up to 64 sequences as one persistent kernel (batch.cu): launch interface.
#pragma once
#include "batch_plan.h"
#include "kernels.h"
#include "solo.h"

namespace ak {

constexpr uint32_t BATCH_ROWS = batch::ROWS * batch::MAX_PARTS;

struct BatchArgs {
    const SoloLayer* layers;     // device array, one per layer; matrices [out, in] bf16
    const void* maps;            // device array of CUtensorMap (batch_maps): qkv, out, up, down of each layer, lm_head
    const void* embedding;
    const float* final_norm;
    const float2* rope;          // [max_len][head_dim / 2] (cos, sin)
    uint8_t* xch;                // exchange sets of every part, batch_sets_bytes() each: all 0xff before the first launch
    batch::State* state;         // of every part, zero before the first launch
    uint32_t* sampled;           // [seqs]: the token fed back to a row with tok_src < 0 (its own last pick), overwritten by the row's greedy pick
    // The step, in device memory or (rows == nullptr) by value
    const int32_t* rows;         // [seqs] of int4 {tok_src, pos, slot, seq}
    const int32_t* kv_lens;      // [seqs]: positions attended to, the new one included; 0: the row is not there
    int32_t tok_src[BATCH_ROWS], lens[BATCH_ROWS];
    const int32_t* block_tables; // [seqs][max_blocks]
    uint32_t* sampled_host;      // where else the picks go: [seqs] in mapped host memory and behind them the status word, or nullptr
    uint32_t* status;            // device word: made non-zero when a wait runs out; a step that finds it so does nothing
    uint64_t max_cycles;         // time limit of the step, in SM clocks
    uint32_t n_layers, dim, ffn, heads, vocab, seqs, max_blocks, max_len;
    uint32_t sms;                // blocks a part is divided over
    uint32_t part_seqs, part_bytes;   // rows and bytes of sets of a part (batch_plan.h)
    float eps, scale;
};

bool batch_supported(uint32_t dtype, uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers, uint32_t seqs, uint32_t max_len);
// the weights' tensor maps, 4 n_layers + 1 of 128 bytes in host memory (layers: host array)
int batch_maps(void* out, const SoloLayer* layers, const void* lm_head, uint32_t n_layers, uint32_t dim, uint32_t ffn, uint32_t vocab);
// a part's sets; seqs: of a part
size_t batch_sets_bytes(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t seqs, uint32_t max_len);
constexpr uint64_t BATCH_MAX_CYCLES = 1ull << 32;   // two seconds or so, for a step of milliseconds
// missing: blocks left out, so that the others' waits run out (a drill)
int launch_batch(cudaStream_t st, const BatchArgs& a, uint32_t missing = 0);
int batch_status(unsigned int* out);

}  // namespace ak
