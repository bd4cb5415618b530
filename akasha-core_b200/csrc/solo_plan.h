// Batch-1 decode step (solo.cu): how a model's weight rows travel through an SM's shared memory, and which models that fits.
// Plain C++ (no CUDA header), so that the plan can be checked on the host.
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define AK_PLAN_FN __host__ __device__ inline
#else
#define AK_PLAN_FN inline
#endif

namespace ak {
namespace solo {

constexpr uint32_t CTAS = 148;           // one block per SM
constexpr uint32_t NW = 12;              // compute warps
constexpr uint32_t SLOT = 12288;         // ring slot: one f32 row of 3072, four of 768
constexpr uint32_t SLICE = 64;           // K elements of a slice
constexpr uint32_t NQ = 6, BLK = 4 * NQ;  // most rows of a block: six per lane group
constexpr uint32_t MAX_SLOTS = 12;
constexpr uint32_t MAX_LAYERS = 48;
constexpr uint32_t N_KINDS = 5;          // weight matrices: qkv, out-proj, ffn-up, ffn-down, lm_head
constexpr uint32_t MAX_DYN_SMEM = 213 * 1024;   // 227 KB less the static variables

// Compute warps that take part in attention: 48 KB of cache tiles for both types (a tile is 4 KB in f32, 2 KB in bf16), the
// rest of shared memory is worth more to the weight ring.
AK_PLAN_FN constexpr uint32_t att_warps(uint32_t esz) { return esz == 4 ? 6 : 12; }
// The cache tiles' bytes. The lm_head phase, when no tile is in use any more, keeps the SM's logits there.
AK_PLAN_FN constexpr uint32_t kv_bytes(uint32_t esz) { return att_warps(esz) * 2 * 1024 * esz; }

// One kind of weight matrix [n, k] as this SM sees it: its rows r0 .. r0 + rows, and how they travel through the ring: rpc
// whole rows to a slot, or (rows wider than a slot) ppr pieces of `piece` elements. The compute warps work on blocks of blk
// rows, a multiple of rpc (no chunk belongs to two blocks) whose chunks fit the ring. Divisions by rpc and by the slices of a
// piece are multiplications by 65536 / d + 1 (see div_exact).
struct Kind {
    uint32_t k, r0, rows, rpc, ppr, piece, blk, inv_rpc, inv_pslices;
    uint32_t n0, chunks0, chunks; // rows and chunks of the first block, all chunks
    uint32_t row_off[4][8];       // [r][i]: ring offset of row r + 4 i of a block, in bytes from the block's first chunk
};
AK_PLAN_FN uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }
AK_PLAN_FN uint32_t udiv_up(uint32_t a, uint32_t b) { return (a + b - 1) / b; }
AK_PLAN_FN uint32_t div_inv(uint32_t v, uint32_t inv) { return (v * inv) >> 16; }
// div_inv(v, 65536 / d + 1) == v / d for every v < n: with e = inv * d - 65536 the product is 65536 v / d + v e / d, so v e must stay
// below 65536; and it must fit 32 bits.
AK_PLAN_FN bool div_exact(uint32_t d, uint64_t n) {
    const uint64_t inv = 65536 / d + 1, e = inv * d - 65536;
    return n == 0 || ((n - 1) * e < 65536 && (n - 1) * inv <= 0xffffffffull);
}
AK_PLAN_FN uint32_t row_begin(uint32_t n, uint32_t cta, uint32_t ctas) { return (uint32_t)(((uint64_t)n * cta) / ctas); }
AK_PLAN_FN void make_kind(Kind& d, uint32_t n, uint32_t k, uint32_t esz, uint32_t slots, uint32_t cta, uint32_t ctas) {
    d.k = k;
    d.r0 = row_begin(n, cta, ctas);
    d.rows = row_begin(n, cta + 1, ctas) - d.r0;
    const uint32_t row = k * esz;
    d.rpc = row <= SLOT ? umin(SLOT / row, BLK) : 1;
    d.piece = row <= SLOT ? k : SLOT / (SLICE * esz) * SLICE;
    d.ppr = udiv_up(k, d.piece);
    const uint32_t fit = umin(BLK / d.rpc, (slots - 2) / d.ppr);
    d.blk = (fit ? fit : 1) * d.rpc;
    d.n0 = umin(d.blk, d.rows);
    d.chunks0 = d.ppr > 1 ? d.n0 * d.ppr : udiv_up(d.n0, d.rpc);
    d.chunks = d.ppr > 1 ? d.rows * d.ppr : udiv_up(d.rows, d.rpc);
    for (uint32_t r = 0; r < BLK; r++) d.row_off[r & 3][r >> 2] = d.ppr > 1 ? r * d.ppr * SLOT : r / d.rpc * SLOT + r % d.rpc * row;
    d.inv_rpc = 65536 / d.rpc + 1;
    d.inv_pslices = 65536 / udiv_up(d.piece, SLICE) + 1;
}

struct Plan {
    uint32_t slots;
    size_t smem;
};
inline bool make_plan(uint32_t esz, uint32_t dim, uint32_t ffn, Plan& p) {
    // beside the ring: the cache tiles of the compute warps, their slices of the residual stream and of a phase's input
    const size_t rest = kv_bytes(esz) + (size_t)NW * (udiv_up(dim / SLICE, NW) + udiv_up(udiv_up(ffn, SLICE), NW)) * SLICE * 4;
    if (rest + 6 * SLOT > MAX_DYN_SMEM) return false;
    p.slots = umin((uint32_t)((MAX_DYN_SMEM - rest) / SLOT), MAX_SLOTS);
    p.smem = (size_t)p.slots * SLOT + rest;
    return true;
}

// esz: bytes of a weight and cache element
inline bool shape_supported(uint32_t esz, uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers, uint32_t vocab) {
    const uint32_t hd = heads ? dim / heads : 0;
    if ((hd != 64 && hd != 128) || dim != heads * hd || heads > CTAS || n_layers > MAX_LAYERS) return false;
    if (dim < SLICE || dim * esz > SLOT || ffn < CTAS || ffn > 32768 || (ffn * esz) % 16 != 0) return false;
    Plan p;
    if (!make_plan(esz, dim, ffn, p)) return false;
    // A block's chunks are waited for together: a row sent in pieces has to fit the ring whole.
    Kind down, head;
    make_kind(down, dim, ffn, esz, p.slots, 0, CTAS);
    make_kind(head, vocab, dim, esz, p.slots, 0, CTAS);
    if (down.ppr > p.slots || !div_exact(udiv_up(down.piece, SLICE), udiv_up(ffn, SLICE))) return false;
    // The lm_head counts its rows by chunks, and keeps their logits where the cache tiles were.
    const uint64_t rows = ((uint64_t)vocab + CTAS - 1) / CTAS;
    return rows * 4 <= kv_bytes(esz) && div_exact(head.rpc, rows);
}

// ---- the word {value, tag} in which the device reports that step `tag` is done
constexpr uint32_t STEP_FAILED = 0xffffffffu;   // in the place of the token: a device-side wait ran out
inline bool read_word(uint64_t word, uint32_t tag, uint32_t& value) {   // false: not written yet
    if ((uint32_t)(word >> 32) != tag) return false;
    value = (uint32_t)word;
    return true;
}

}  // namespace solo
}  // namespace ak
