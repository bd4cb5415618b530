// Decode step of up to 64 sequences (batch.cu): tiles, exchange buffers and shared memory, and which models they fit.
// Plain C++ (no CUDA header), so that the plan can be checked on the host.
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifndef AK_PLAN_FN
#ifdef __CUDACC__
#define AK_PLAN_FN __host__ __device__ inline
#else
#define AK_PLAN_FN inline
#endif
#endif

namespace ak {
namespace batch {

constexpr uint32_t SMS = 148;             // one block per SM
constexpr uint32_t SMS_BESIDE = 48, SMS_BESIDE_PARTS = 34;   // the fewest blocks of a step beside prompts; of each of its parts
constexpr uint32_t ROWS = 32;             // most sequences of a part
constexpr uint32_t MAX_PARTS = 2;
static_assert(SMS_BESIDE_PARTS >= ROWS && SMS_BESIDE >= ROWS, "block r picks the token of row r");
constexpr uint32_t NW = 12;               // compute warps
constexpr uint32_t NH = 3;                // epilogue warps
constexpr uint32_t TB = 3;                // weight tiles of a pass (accumulators, partial sums)
constexpr uint32_t CHUNK = 24;            // K slices (of 32) of a ring slot at most
constexpr uint32_t SLOT = 8 * CHUNK * 64; // 8 weight rows
constexpr uint32_t MAX_SLOTS = 8, MAX_EXTRA = 6;
constexpr uint32_t MAX_LAYERS = 48;
constexpr uint32_t KV_BUF = 4096;         // bytes of a warp's key (and of its value) buffer: 2048 / head_dim positions
constexpr uint32_t MAX_UNITS = 32;        // attention units of a group (a lane keeps one)
constexpr uint32_t MAX_DYN_SMEM = 216 * 1024;

AK_PLAN_FN constexpr uint32_t div_up(uint32_t a, uint32_t b) { return (a + b - 1) / b; }
// More than 32 sequences are two parts, each with half of the sequences and half of the SMs, that have nothing to do with each other
AK_PLAN_FN constexpr uint32_t parts_of(uint32_t seqs) { return seqs <= ROWS ? 1 : MAX_PARTS; }
AK_PLAN_FN constexpr uint32_t part_seqs(uint32_t seqs) { return div_up(seqs, parts_of(seqs)); }
// The sequences of a step of two parts are dealt in order of length (rank 0: the longest), there and back: 0 1 1 0 0 1 1 0 ... Dealt by halves of the slots, the
// part with the longer contexts set the step's time, and a queue that was half empty ran on half of the SMs: 162M model, 64 slots, us per step, so / now (as
// launches): 32 running at 380 of 512 positions 430 / 317 (472), 48 439 / 408 (498), 64 440 / 444 (531); at 1900 of 2048 1037 / 632 (830), 1042 / 878 (950), 1055 / 1045
// (1125); at 3900 of 4096 1824 / 1050 (1285), 1830 / 1470 (1510), 1873 / 1875 (1897); 128 ragged sequences through 64 slots 344 / 333 ms.
AK_PLAN_FN constexpr uint32_t part_of_rank(uint32_t rank) { return (rank ^ (rank >> 1)) & 1u; }
AK_PLAN_FN constexpr uint32_t row_of_rank(uint32_t rank) { return rank >> 1; }
AK_PLAN_FN constexpr uint32_t m_tiles(uint32_t seqs) { return seqs <= 16 ? 1 : 2; }
AK_PLAN_FN constexpr uint32_t tile_begin(uint32_t tiles, uint32_t cta, uint32_t sms) { return (tiles * cta) / sms; }   // of the step's sms blocks
// Positions of an attention unit. Where all sequences fit in 128 KB of keys (1024 positions of head size 64, 512 of 128) they are whole, which saves
// publishing and merging; longer ones are cut into 256 positions, so that the groups' shares come out even. Jobs of 30 to 40 steps near the
// capacity, ms, cut / whole: 162M model 8 slots, 520 positions 9.70 / 9.18, 768 10.31 / 9.82, 1024 11.32 / 11.10, 2048 16.3 / 15.3; 32 slots, 768 23.5 / 21.5,
// 1024 28.1 / 25.8, 2048 46.7 / 44.1; 320-wide model 21 slots, 1024 7.83 / 7.75, 4 slots, 2048 6.11 / 7.19; 1.4B model (head size 128) 4 slots, 1024
// 38.7 / 39.1, 16 slots, 1024 89.0 / 90.0, 2048 148 / 160. In units of 512 instead of 256: 0.92 to 1.06 of the speed; of 128: 0.87 to 1.03.
AK_PLAN_FN constexpr uint32_t unit_len(bool splits, uint32_t hd) { return splits ? 256 : 65536 / hd; }
AK_PLAN_FN constexpr bool has_splits(uint32_t max_len, uint32_t hd) { return max_len > unit_len(false, hd); }
AK_PLAN_FN constexpr uint32_t split_len(uint32_t max_len, uint32_t hd) { return unit_len(has_splits(max_len, hd), hd); }
// A weight row as pieces of the tensor map: 256 columns, or what divides the row
AK_PLAN_FN constexpr uint32_t piece_of(uint32_t k) { return k % 256 == 0 ? 256 : k % 64 == 0 ? 64 : 32; }
AK_PLAN_FN constexpr uint32_t chunk_cols(uint32_t k) { return k < CHUNK * 32 ? k : CHUNK * 32; }

// byte offsets inside an exchange set (and its size): x after ffn-down, attention, x after out-proj, ffn-up as A fragments; sums of squares; qkv and
// the splits of the attention in f32; an SM's best logit of a row {value, index}
struct SetOff {
    uint32_t x1, at, x2, up, s1, s2, qkv, best, part;
    size_t total;
    SetOff() = default;
    AK_PLAN_FN SetOff(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t mt, uint32_t splits) {
        const uint32_t r = mt * 16, hd = dim / heads, cx = dim * r * 2, cs = dim / 8 * r * 4;
        x1 = 0; at = x1 + cx; x2 = at + cx; up = x2 + cx;
        s1 = up + ffn * r * 2; s2 = s1 + cs;
        qkv = s2 + cs;
        best = qkv + r * 3 * dim * 4;
        part = best + SMS * r * 8;
        total = part + (splits > 1 ? (size_t)r * heads * splits * (hd + 4) * 4 : 0);
    }
};

// The exchange sets, used in turn: the step's embedding has set e0, layer l set e0 + 1 + l (mod SETS), the next step starts with the set behind.
// A set is cleared, by all SMs together, when what it holds has been read by everybody: the set of layer l - 1 (the embedding's for l = 0) once an SM
// has published its ffn-up of layer l, and the last layer's at the start of the next step. An SM counts itself in behind each of its clears.
constexpr uint32_t SETS = 4;
// Clears that every SM has counted itself in for before an SM's epilogue goes on to the out-proj of layer l: the one at the start and those behind
// the ffn-up of layers 0 .. l - 1. So the set of layer l + 2 is clean before anybody looks at it: the warp furthest ahead (one without
// a slice of x, on an SM that has ffn-up tiles only) comes to the attention of layer l + 2 knowing that its epilogue is through ffn-up of layer l.
// With three sets, and known by what was read only, such a warp could see a set before another SM had cleared it.
AK_PLAN_FN constexpr uint32_t clears_before_out(uint32_t l) { return 1 + l; }
AK_PLAN_FN constexpr uint32_t clears_of_step(uint32_t n_layers) { return 1 + n_layers; }

// What steps hand on to each other, behind the sets. Only the kernel writes it, at the end of a step: a launch that failed changes nothing.
struct State {
    uint32_t set;       // e0 of the next step
    uint32_t counted;   // what `cleared` is when the next step starts
    uint32_t pad0[30];
    uint32_t cleared;   // SMs counted in for clears since the beginning (mod 2^32)
    uint32_t pad1[31];
};

inline size_t sets_bytes(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t seqs, uint32_t max_len) {
    return (SETS * SetOff(dim, ffn, heads, m_tiles(seqs), div_up(max_len, split_len(max_len, dim / heads))).total + 127) / 128 * 128;
}

struct Plan {
    uint32_t slots, wpi;
    size_t smem;
};
// seqs: of a part; sms: blocks of a part
inline Plan make_plan(uint32_t dim, uint32_t n_layers, uint32_t heads, uint32_t seqs, uint32_t max_len, uint32_t sms = SMS, uint32_t parts = 1) {
    const uint32_t hd = dim / heads;
    const size_t rest = NW * 2 * KV_BUF + (size_t)NW * TB * m_tiles(seqs) * 16 * 32 + 2 * NW * hd * 4 + TB * 32 * 2 * 16 + (size_t)(2 * n_layers + 1) * div_up(dim / 8, sms) * 32;
    Plan p;
    p.slots = (uint32_t)((MAX_DYN_SMEM - rest) / SLOT);
    if (p.slots > MAX_SLOTS) p.slots = MAX_SLOTS;
    p.smem = p.slots * SLOT + rest;
    // Warps of an attention unit. Whole sequences: 12, 6 or 4, the most that leave a group for every unit, because a group's second unit starts when the first is done
    // (where four do not either, long units share a group with short ones). Contexts of 300, us per step, with 12 or 4 and now 6: 162M model, 13 sequences
    // 233 / 218, 16 234 / 219, 24 283 / 265; 320-wide model, 32 sequences 151 / 143. Fewer than four give 64 equal sequences 417 / 414, but a
    // long one among others then takes long: 128 ragged sequences through 64 slots 359 / 375 ms. Cut sequences: 12 up to one unit per SM, else 4. With 3
    // or 2 some shapes are faster and as many slower, by how the units of a step fall into rounds of the groups: heads of 64, 2048 positions, 4 / 3 / 2 warps, 8
    // sequences 266 / 290 / 254, 32 641 / 621 / 667, 320-wide model, 21 188 / 207 / 181; heads of 128, 4 / 3, 768 wide, 12 layers, 16 sequences at 2000 positions 382 / 444,
    // 24 534 / 513; 1.4B model, 16 at 540 1253 / 1336, 16 of random lengths up to 3072 1980, 1922, 1677 / 2008, 1897, 1769, 8 1315, 1446, 1438 / 1367, 1384, 1378.
    // (Not by the step's blocks: a unit's sums depend on it.)
    const uint32_t splits = div_up(max_len, split_len(max_len, hd)), units = seqs * heads * splits, own = SMS / parts;
    p.wpi = units <= own ? 12 : splits == 1 && units <= 2 * own ? 6 : 4;
    return p;
}
// Chunks of weights that are brought into L2 ahead of the ring of `slots`. Where the ring holds about a layer and the layer is short (16 rows at most), four more
// close its gaps: 162M model, contexts of 300, us per step without / with: 1 sequence 160 / 147, 8 176 / 163, 16 211 / 202 (with 8 chunks 164 and 203, with 16
// 166 and 205); 320-wide, 8 sequences 102 / 100. With 32 rows 294 / 295, 64 sequences 397 / 401, and models that stream many rings a layer
// (1.4B, 4 sequences of 500: 961 / 977; for head size 128 the walk is left out) are without.
AK_PLAN_FN constexpr bool can_ahead(uint32_t hd, uint32_t mt) { return hd == 64 && mt == 1; }
AK_PLAN_FN constexpr uint32_t ahead_of(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t seqs, uint32_t sms, uint32_t slots) {
    const uint32_t kd = div_up(dim, CHUNK * 32), kf = div_up(ffn, CHUNK * 32);
    const uint32_t layer = (div_up(3 * dim / 8, sms) + div_up(dim / 8, sms) + div_up(ffn / 8, sms)) * kd + div_up(dim / 8, sms) * kf;
    return can_ahead(dim / heads, m_tiles(seqs)) && layer <= 2 * slots ? 4 : 0;
}

// An attention unit: positions p0 .. p0 + n of (row, head), nb tiles.
struct Unit { uint32_t row, head, split, p0, n, nb; };
// The tiles a warp has yet to request, in order: tile b of unit j (u) of layer l, in the pool blocks pb0 (and pb1); nu: units of the warp's group.
struct Walk {
    Unit u;
    uint32_t l, j, b, pb0, pb1, nu, more, asked, sent;   // more: there is such a tile; asked: its keys are requested; sent: requests made for values
};
// To the next tile of the warp, the place-th of the wpi of its group, which has a tile in some unit. unit_at(j): unit j of the group. look_up(): the
// tile's pool blocks; asked for tiles that exist only.
template <class UnitAt, class LookUp>
AK_PLAN_FN void walk_on(Walk& k, uint32_t wpi, uint32_t place, uint32_t n_layers, UnitAt unit_at, LookUp look_up) {
    k.b += wpi;
#ifdef __CUDACC__
#pragma unroll 1
#endif
    while (k.b >= k.u.nb) {
        if (++k.j == k.nu) {
            k.j = 0;
            if (++k.l == n_layers) {
                k.more = 0;
                return;
            }
        }
        k.u = unit_at(k.j);
        k.b = place;
    }
    look_up();
}

inline bool shape_supported(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers, uint32_t seqs, uint32_t max_len) {
    const uint32_t hd = heads ? dim / heads : 0;
    if ((hd != 64 && hd != 128) || dim != heads * hd || heads > 4095) return false;
    if (seqs < 1 || seqs > ROWS * MAX_PARTS || n_layers < 1 || n_layers > MAX_LAYERS || dim < 96 || dim % 32 || ffn % 32 || ffn > 65536) return false;
    // Two parts where K is one chunk of the ring, so that activations stay in registers for the passes of a phase. Wider models were slower so than as launches:
    // 64 slots, 12 layers, us per step as launches / in parts: 768 wide, heads of 128, 1 to 64 running at 380 positions 438 .. 520 / 314 .. 442; 1024 wide 494 .. 700 /
    // 497 .. 744, at 1900 693 .. 1490 / 518 .. 1452 (48 running 1145 / 1234); heads of 64 491 .. 711 / 385 .. 675, 32 long and 32 short ones 962 / 1017;
    // 1536 wide 702 .. 975 / 796 .. 1052, heads of 64, 64 running at 1900 2046 / 2179.
    if (parts_of(seqs) > 1 && div_up(dim, CHUNK * 32) > 1) return false;
    const uint32_t sms = SMS / parts_of(seqs);
    seqs = part_seqs(seqs);
    if (ffn / 8 < SMS) return false;                                       // every SM has ffn-up rows (the clearing of the sets counts on it)
    if (div_up(dim / 8, sms) > TB) return false;                           // the residual stream is worked on in one pass
    if (dim * m_tiles(seqs) * 16 * 2 > NW * 2 * KV_BUF) return false;      // the lm_head keeps x where the cache tiles were
    const uint32_t splits = div_up(max_len, split_len(max_len, hd));
    const Plan p = make_plan(dim, n_layers, heads, seqs, max_len, sms, SMS / sms);
    if (splits > 16383 || (uint64_t)seqs * heads * splits > (uint64_t)MAX_UNITS * sms * (NW / p.wpi)) return false;
    return p.slots >= 4 && MAX_PARTS * sets_bytes(dim, ffn, heads, seqs, max_len) < (1ull << 32);   // (offsets of 32 bits; four slots: what a pass holds at a time)
}

// SMs of a step with prompts beside it, whose chain of launches gets the others. The chain is the longer of the two in almost every such step, so the step
// takes as few as its plan allows (what it computes does not depend on the number of its blocks). Jobs with prompts in most steps, ms: 162M model, 32
// slots, prompts of 1 to 24, 8 tokens on average: step and chain one after the other on all SMs 39.3, beside each other on 90 SMs 34.9, 74
// 33.1, 60 32.7, 48 30.7 (all rows through the chain, which shares its launches then: 31.2); 8 slots, prompts of 16 to 448, 2 tokens: 20.8, 19.2, 18.9,
// 18.9, 18.5 (19.8); 320-wide model, 32 slots: 20.8, 16.7, 16.0, 15.9, 15.9 (17.2); 1.4B model (86 SMs at least), 16 slots, prompts of 1 to
// 64, 4 tokens: 57.5, 55.8, 54.9 (53.9: both read all weights), prompts of 128 to 1024: 128.7, 129.3, 127.9 (128.8).
// Of each of two parts (seqs: the part's), 64 slots of the 162M model, with 34 / 48 / 60 / 74 SMs: 192 prompts of 1 to 24, 8 tokens on average, 17.7 / 18.9 / 20.4 /
// 20.8 ms (all rows through the chain 18.3); of 16 to 448, 4 tokens 21.5 / 21.5 / 22.0 / 22.4 (22.3), 32 tokens 89.9 / 92.7 / 97.7 / 101.1 (101.2).
inline uint32_t sms_beside(uint32_t dim, uint32_t n_layers, uint32_t heads, uint32_t seqs, uint32_t max_len, uint32_t parts = 1) {
    const uint64_t units = (uint64_t)seqs * heads * div_up(max_len, split_len(max_len, dim / heads));
    for (uint32_t sms = parts == 1 ? SMS_BESIDE : SMS_BESIDE_PARTS; sms < SMS / parts; sms++) {
        const Plan p = make_plan(dim, n_layers, heads, seqs, max_len, sms, parts);
        if (div_up(dim / 8, sms) <= TB && units <= (uint64_t)MAX_UNITS * sms * (NW / p.wpi) && p.slots >= 4) return sms;
    }
    return SMS / parts;
}

}  // namespace batch
}  // namespace ak
