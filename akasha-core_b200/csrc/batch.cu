// One decode step of up to 64 sequences (bf16 weights and cache) as a single persistent kernel: embedding, every layer,
// lm_head, greedy argmax.
//
// What bounds it. A decode-only step as a chain of 88 launches is bound by the launches: each is a boundary of ~2 us plus the latencies
// of its first loads, 3 to 5 us for work of 0.1 to 1 us (162M model, contexts of 300: 8 sequences 0.39 ms, 64 0.49; the bytes take 0.05 and
// 0.15 ms). Here, as in the batch-1 step (solo.cu), a layer is five phases of one kernel and only activations cross the chip:
//   qkv rows -> attention (sequence, head) -> out-proj rows -> ffn-up rows -> ffn-down rows.
// That step takes 0.162 ms with 8 sequences, 0.202 with 16, 0.295 with 32, 0.400 with 64 (320-wide model, 21 sequences 0.120; 1.4B model, 16 of 1600
// 1.8). What is left is latency: per phase the way from a store to the last SM's poll, and dependent instructions (with everything between
// two phases done by the same warps it was 0.29 ms for 8).
//   * Every SM reads all activations of a phase, which is what grows with the sequences. More than 32 (of models up to 768 wide) are two parts: half of the
//     sequences and half of the SMs each, all weights, nothing between the two. 64 sequences: 0.49 ms as launches, 0.58 with 64 rows on every SM, 0.400 in parts.
//   * A producer thread per SM walks the SM's weight tiles of all phases in order and keeps a shared-memory ring of tensor loads full.
//   * A phase's rows are dealt to the SMs in tiles of 8, all of K: no sum crosses SMs. The 12 compute warps split K and leave partial tiles in
//     shared memory; three epilogue warps add them in warp order and publish, while the compute warps are already at the next phase. The
//     products are mma.m16n8k16 with 16 sequences on the M side and 8 weight rows on the N side: a tcgen05 tile (128 x 8 at least,
//     operands through shared memory, the result back through tensor memory) costs more latency than these few products take.
//   * Activations are published in the order of the MMA's A fragments (a lane's 8 consecutive k of a sequence are one 16-byte vector), so
//     that a warp's fragment is one coalesced 512-byte load from L2 straight into registers. Both operands use the same order of k. What a
//     tile publishes for 8 sequences is one 128-byte line.
//   * A value is its own flag: an exchange buffer holds 0xffffffff words until it is written, a NaN no conversion and no arithmetic
//     gives, and consumers poll the words they need. No fence and no second round trip between the value and its flag. Four sets of
//     buffers are used in turn by the layers; the one of the layer before is filled with 0xff again after a layer's ffn-up (see clear).
//   * RMS norm: the producer of the residual stream publishes x * gain rounded to bf16 (one rounding, as of the normalised value) and
//     the sums of squares of its columns; 1 / rms is a factor of the row sums of the next phase, found by the epilogue warps meanwhile.
//   * The residual stream stays in shared memory of the SM that owns its columns (out-proj and ffn-down have the same tiles).
//   * Attention: a unit is (sequence, head, split of split_len positions); units are dealt to groups of 4 to 12 warps in order of length. Keys
//     and values go through per-warp shared-memory buffers, the next layer's first tiles already while this layer's ffn runs. Scores are
//     mma.m16n8k16 (7/8 of it for nothing, but an eighth of the instructions of f32 FMAs); P V is f32 FMAs, the transposing loads that an
//     MMA would need have 8-way bank conflicts on unswizzled tiles (32 sequences: 0.41 ms instead of 0.35).
//
// Arithmetic: bf16 inputs rounded once, f32 products and sums, as in the launch chain; the probabilities stay f32. The order of every sum
// depends on the model and on the number of slots only, never on which other sequences are there.
//
// The grid is launched cooperatively (its blocks wait on one another): one block per SM, all resident. The step has a time limit; a wait that goes on
// past it gives up and the block is `dead` (later waits give up soon). Its warps go through the rest of the step all the same, so that
// the barriers between them come out even, but a warp whose wait for a copy ran out releases no slot and requests no copy any more, and
// nobody leaves before the copies it started have landed. The status word is set, the host reports AK_ERR_DEVICE_WAIT, and a step
// launched behind it returns at once: the exchange sets are not clean.
#include "batch.h"
#include "batch_plan.h"
#include "tma.h"

#include <type_traits>

namespace ak {

__device__ unsigned int g_batch_status = 0;

namespace {

using namespace batch;
static_assert(SMS == B200_SMS, "a block per SM");
constexpr uint32_t NCT = NW * 32, NHT = NH * 32;   // threads of the compute and of the epilogue warps
constexpr uint32_t THREADS = 512, FIRST_COMPUTE = 4;
constexpr int REGS_FIRST = 104, REGS_COMPUTE = 136;
static_assert(REGS_FIRST * 128 + REGS_COMPUTE * 384 <= 65536, "the split draws on the registers of the launch");
constexpr uint32_t EMPTY = 0xffffffffu;   // an exchange word that is not written yet

// Bounds the waits of a block (in shared memory): `dead` is sticky and set when a wait goes on past the deadline, a time limit of the whole step.
struct Expiry {
    long long deadline;
    uint32_t dead;
    __device__ __forceinline__ bool is_dead() const { return *(const volatile uint32_t*)&dead != 0; }
    __device__ __forceinline__ bool expired() {
        if (is_dead()) return true;
        if (clock64() <= *(const volatile long long*)&deadline) return false;
        *(volatile uint32_t*)&dead = 1u;
        return true;
    }
};
struct Waiter {   // of one thread that polls
    Expiry* x;
    __device__ __forceinline__ bool give_up(uint32_t& n) { return (++n & 63u) == 0 && x->expired(); }
};
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, Expiry& x) {
    if (mbar_try_wait(bar, parity)) return true;
#pragma unroll 1
    for (;;) {
#pragma unroll 1
        for (uint32_t n = 0; n < 64; n++)
            if (mbar_try_wait(bar, parity)) return true;
        if (x.expired()) return false;
    }
}
// For warps of the same block. They always come, late when their own waits run out, so this one does not give up with them: a warp that went on without them
// would arrive at BAR_PART twice in one use. (2^33 cycles behind the deadline it ends all the same.)
__device__ __forceinline__ void wait_block(uint64_t* bar, uint32_t parity, const Expiry& x) {
    if (mbar_try_wait(bar, parity)) return;
#pragma unroll 1
    while (!mbar_try_wait(bar, parity))
        if (clock64() > *(const volatile long long*)&x.deadline + (1ll << 33)) return;
}

// ---- exchange words
// (16 bytes in one piece: a vector that has any of its words has all of them)
__device__ __forceinline__ uint4 xld4(const void* p) {
    uint64_t a, b;
    asm volatile("{\n.reg .b128 q;\nld.relaxed.gpu.global.b128 q, [%2];\nmov.b128 {%0, %1}, q;\n}\n" : "=l"(a), "=l"(b) : "l"(p));
    return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ uint32_t xld1(const void* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 xld2(const void* p) {
    uint2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void xst1(void* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void xst2(void* p, uint32_t a, uint32_t b) { asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory"); }
__device__ __forceinline__ void xst4(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint64_t x = a | ((uint64_t)b << 32), y = c | ((uint64_t)d << 32);
    asm volatile("{\n.reg .b128 q;\nmov.b128 q, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p), "l"(x), "l"(y) : "memory");
}
// (the result of an operation is never EMPTY: a NaN comes out as 0x7fffffff)
__device__ __forceinline__ uint32_t word(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {   // (a NaN becomes 0x7fff)
    const bf162 p = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&p);
}
template <uint32_t N> __device__ __forceinline__ void bar_sync(uint32_t id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(N) : "memory"); }
__device__ __forceinline__ void bar_sync_n(uint32_t id, uint32_t n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
template <uint32_t N> __device__ __forceinline__ void bar_arrive(uint32_t id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(N) : "memory"); }
enum { BAR_PART = 1, BAR_HELP = 2, BAR_HEAD = 3, BAR_FLAT = 4, BAR_GROUP = 5 };   // BAR_GROUP and the next two: by group

__device__ __forceinline__ void bulk_g2s_hint(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t pol) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ex2(float x) {   // 2^x
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float redux_max(float v) {   // of the warp (no NaN)
    float m;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}
__device__ __forceinline__ void unpack8(const uint4& r, float (&o)[8]) {
    o[0] = __uint_as_float(r.x << 16); o[1] = __uint_as_float(r.x & 0xffff0000u);
    o[2] = __uint_as_float(r.y << 16); o[3] = __uint_as_float(r.y & 0xffff0000u);
    o[4] = __uint_as_float(r.z << 16); o[5] = __uint_as_float(r.z & 0xffff0000u);
    o[6] = __uint_as_float(r.w << 16); o[7] = __uint_as_float(r.w & 0xffff0000u);
}
// 1 / sqrt(m): the hardware's approximation and one Newton step, which has no value where m is 0 or infinite (there the approximation is exact)
__device__ __forceinline__ float inv_rms(float m) {
    const float y = rsqrtf(m);
    return y > 0.0f && y < INFINITY ? y * fmaf(-0.5f * m * y, y, 1.5f) : y;
}

// A load from shared memory and a later arrival on a barrier (or the request of a copy) are not in order by themselves: a buffer could be overwritten
// under a load that nothing has waited for yet. True for every value, but known only when v, and with it all that v was computed from, is there in
// every lane.
__device__ __forceinline__ bool settled(float v) { return __any_sync(0xffffffffu, __float_as_uint(v) != EMPTY) != 0; }

struct Cursor {   // a place in the ring: slot and the parity of its current use
    uint32_t s = 0, ph = 0;
    __device__ __forceinline__ void advance(uint32_t by, uint32_t n) {   // by <= n
        s += by;
        if (s >= n) { s -= n; ph ^= 1u; }
    }
};
// A weight matrix [n, k] as this SM sees it (kept in shared memory: held in registers or recomputed, the four of them spill): its tiles of 8 rows, and K as
// ring chunks of CHUNK slices of 32 (the last may have fewer).
struct Kind {
    uint32_t t0, n, slices, chunks, pitch, pieces;   // pitch: bytes of a row in a slot; pieces of a chunk in the tensor map
    __device__ __forceinline__ uint32_t count(uint32_t c) const { return min(CHUNK, slices - c * CHUNK); }
};
__device__ __forceinline__ void make_kind(Kind& d, uint32_t rows, uint32_t k, uint32_t cta, uint32_t sms) {
    d.t0 = tile_begin(div_up(rows, 8), cta, sms);
    d.n = tile_begin(div_up(rows, 8), cta + 1, sms) - d.t0;
    d.slices = k >> 5;
    d.chunks = div_up(d.slices, CHUNK);
    d.pitch = chunk_cols(k) * 2;
    d.pieces = CHUNK * 32 / piece_of(k);
}
// Byte offset of vector v (columns 8 v .. 8 v + 7) of a row among the A fragments. The eight vectors that a tile publishes for eight rows are one 128-byte
// line: lane 4 g + t of a fragment reads vector 8 t + g of its 512 bytes.
template <int MT> __device__ __forceinline__ uint32_t frag(uint32_t row, uint32_t v) {
    return ((((v >> 2) * MT + (row >> 4)) * 2 + ((row >> 3) & 1)) * 32 + (v & 3) * 8 + (row & 7)) * 16;
}
enum { QKV = 0, OUT = 1, FFN_UP = 2, FFN_DOWN = 3, HEAD = 4, N_KINDS = 5 };
constexpr uint32_t NO_LOGIT = 0x7fffffffu;   // in the place of the index of a best logit

// SPLIT: sequences may be longer than an attention unit
template <int HD, int MT, bool SPLIT, int PARTS>
__global__ void __launch_bounds__(THREADS, 1) batch_kernel(const __grid_constant__ BatchArgs a, const uint32_t slots, const uint32_t wpi, const uint32_t inv_wpi, const uint32_t ahead) {
    constexpr uint32_t R = MT * 16;               // rows of the exchange buffers
    constexpr bool CAN_AHEAD = can_ahead(HD, MT);
    constexpr uint32_t PPC = CHUNK / NW;          // slices of a ring chunk that a warp has: 2
    constexpr bool KEEP = PARTS > 1;              // activations stay in registers for the passes of a phase (half of the SMs have twice the tiles)
    constexpr uint32_t Q = R / 4, TPL = 32 / Q;   // lanes that read a tile's sums of squares, tiles per load
    constexpr uint32_t CH = HD / 8;               // 16-byte vectors of a cache row
    constexpr uint32_t PPI = 32 / CH;             // positions a warp reads per instruction
    constexpr uint32_t UP = 2048 / HD;            // positions of a tile buffer
    extern __shared__ __align__(128) uint8_t smem[];
    // (the bars and uses from MAX_SLOTS on belong to the extra slots that the lm_head has where the cache tiles were)
    __shared__ uint64_t full_bar[MAX_SLOTS + MAX_EXTRA], empty_bar[MAX_SLOTS + MAX_EXTRA], k_bar[NW], v_bar[NW], free_bar, kv_free_bar;
    __shared__ SoloLayer layers_sm[MAX_LAYERS];
    __shared__ Kind kinds[N_KINDS];
    __shared__ SetOff so;
    __shared__ __align__(16) float ss_sm[2][NH][R];   // a norm phase's sums of squares, by epilogue warp
    __shared__ float2 at_ml[2][NW];
    __shared__ Walk walk_sm[NW];
    __shared__ uint32_t units[NW][MAX_UNITS];
    __shared__ uint32_t len_sm[32], by_len[32], pre_sm[33], slot_sm[PARTS > 1 ? 32 : 1];   // slot_sm: the slots of a part's rows
    __shared__ Expiry expiry;
    __shared__ uint32_t failed_sm, flat_sm, live_sm, use_sm[MAX_SLOTS + MAX_EXTRA];   // use_sm: 1 + the number of the use a slot is in (lm_head only)

    const uint32_t tid = threadIdx.x, warp_ = tid >> 5, lane = tid & 31;
    // What tells the parts apart: rows, sets (an offset that set_of() adds), state. (As arguments of their own, chosen by the block, they cost 5 % of a step.)
    const uint32_t part_no = PARTS > 1 && blockIdx.x >= a.sms ? 1u : 0u;
    const uint32_t cta = PARTS > 1 ? blockIdx.x - part_no * a.sms : blockIdx.x;
    State* const state = PARTS > 1 ? a.state + part_no : a.state;
    const uint32_t D = a.dim, F = a.ffn, H = a.heads, L = a.n_layers;
    uint8_t* const kv_sm = smem + slots * SLOT;
    float* const part = reinterpret_cast<float*>(kv_sm + NW * 2 * KV_BUF);        // [NW][TB][R][8]
    float* const at_acc = part + NW * TB * R * 8;                                 // [2][NW][HD]
    float4* const res_sm = reinterpret_cast<float4*>(at_acc + 2 * NW * HD);       // [tile][R][2]: the residual stream of this SM's columns
    float* const gain_sm = reinterpret_cast<float*>(res_sm + TB * R * 2);                // [2 L + 1][tiles][8]: the gains of its columns, by norm
    constexpr uint32_t SPLIT_LEN = unit_len(SPLIT, HD);
    const uint32_t splits = div_up(a.max_len, SPLIT_LEN);

    if (tid == 160) so = SetOff(D, F, H, MT, splits);
    if (tid == 0) {
#pragma unroll 1
        for (uint32_t s = 0; s < MAX_SLOTS + MAX_EXTRA; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], NW); use_sm[s] = 0; }
#pragma unroll 1
        for (uint32_t i = 0; i < NW; i++) { mbar_init(&k_bar[i], 1); mbar_init(&v_bar[i], 1); }
        mbar_init(&free_bar, NH);
        mbar_init(&kv_free_bar, NW);
        expiry.deadline = clock64() + (long long)a.max_cycles;
        expiry.dead = 0;
        failed_sm = *(const volatile uint32_t*)a.status;
        mbar_fence_init();
    }
    if (tid >= 32 && tid < 32 + N_KINDS) make_kind(kinds[tid - 32], tid == 32 ? 3 * D : tid == 34 ? F : tid == 36 ? a.vocab : D, tid == 35 ? F : D, cta, a.sms);
    if (warp_ == 2) {   // the rows' lengths, the rows by length (the longest first), the attention splits of the rows before by that rank
        uint32_t n[PARTS], key[PARTS], rank[PARTS] = {};   // of slot lane + 32 p
#pragma unroll
        for (uint32_t p = 0; p < PARTS; p++) {
            const uint32_t s = lane + 32 * p;
            n[p] = s < a.seqs ? min((uint32_t)max(a.rows ? a.kv_lens[s] : a.lens[s], 0), a.max_len) : 0u;
            key[p] = n[p] << 6 | (63 - s);   // (lengths are below 2^26)
        }
#pragma unroll
        for (uint32_t j = 0; j < 32 * PARTS; j++) {
            const uint32_t o = __shfl_sync(0xffffffffu, key[j / 32], j % 32);
#pragma unroll
            for (uint32_t p = 0; p < PARTS; p++) rank[p] += o > key[p];
        }
#pragma unroll
        for (uint32_t p = 0; p < PARTS; p++) {
            if (PARTS == 1) {
                len_sm[lane] = n[p];
                by_len[rank[p]] = lane;
            } else if (part_of_rank(rank[p]) == part_no) {   // (a part's rows are in order of length)
                const uint32_t row = row_of_rank(rank[p]);
                len_sm[row] = n[p];
                slot_sm[row] = lane + 32 * p;
                by_len[row] = row;
            }
        }
        __syncwarp();
        const uint32_t m = __ballot_sync(0xffffffffu, len_sm[lane] > 0);
        if (lane == 0) live_sm = m;
        const uint32_t mine = div_up(len_sm[by_len[lane]], SPLIT_LEN);
        uint32_t sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= (uint32_t)o) sum += t;
        }
        pre_sm[lane] = sum - mine;
        if (lane == 31) pre_sm[32] = sum;
    }
#pragma unroll 1
    for (uint32_t i = tid; i < L * (uint32_t)(sizeof(SoloLayer) / 8); i += THREADS)
        reinterpret_cast<uint64_t*>(layers_sm)[i] = reinterpret_cast<const uint64_t*>(a.layers)[i];
    const uint32_t e0 = *(const volatile uint32_t*)&state->set;   // (before the block's barrier, so before this SM publishes anything)
    __syncthreads();
    auto report = [&]() {
        atomicExch(a.status, 1u);
        atomicExch(&g_batch_status, 1u);
        if (a.sampled_host) *(volatile uint32_t*)(a.sampled_host + a.seqs) = 1u;
    };
    if (failed_sm) {   // a step before this one failed
        if (tid == 0) report();
        return;
    }
#pragma unroll 1
    for (uint32_t i = tid, n = kinds[OUT].n * 8; i < (2 * L + 1) * n; i += THREADS)
        gain_sm[i] = (i / n == 2 * L ? a.final_norm : i / n & 1 ? layers_sm[i / (2 * n)].norm_2 : layers_sm[i / (2 * n)].norm_1)[kinds[OUT].t0 * 8 + i % n];
    const uint32_t live = live_sm, n_act = __popc(live);
    if (n_act == 0) return;
    __syncthreads();   // the gains

    // The lm_head keeps x where the cache tiles were, and extra slots behind it. Its chunk n is in slot n mod (slots + extra) of the two.
    uint8_t* const extra_sm = kv_sm + D * R * 2;
    const uint32_t extra = min(MAX_EXTRA, (NW * 2 * KV_BUF - D * R * 2) / SLOT), head_slots = slots + extra;
    auto set_of = [&](uint32_t g) { return (g % SETS) * (uint32_t)so.total + (PARTS > 1 ? part_no * a.part_bytes : 0u); };   // byte offset; g = e0: the embedding, e0 + 1 + l: layer l
    auto slot_of = [&](uint32_t r) { return PARTS > 1 ? slot_sm[r] : r; };
    auto row_live = [&](uint32_t r) { return (live >> r) & 1u; };
    auto eight_live = [&](uint32_t e) { return ((live >> (e * 8)) & 0xffu) != 0; };
    const Waiter wt{&expiry};
    const float inv_dim = 1.0f / (float)D;

    if (warp_ < FIRST_COMPUTE) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_FIRST));
    if (warp_ == 0) {
        // ---------------- producer: this SM's weight tiles in the order the compute warps use them, a chunk of a tile by one tensor load (its eight rows as
        // bulk copies of their own took 0.6 us to issue: 3 TB/s over the chip)
        if (lane != 0) return;
        const CUtensorMap* const map = reinterpret_cast<const CUtensorMap*>(a.maps);
        const uint64_t pol = stays_in_l2(step_weight_bytes(2, D, F, L, a.vocab)) ? policy_evict_normal() : policy_evict_first();
        Cursor q;
        uint32_t sent = 0;
        bool ok = true;
        // `ahead` chunks further on, the weights are brought into L2 (a walk of its own over phase, first tile of a pass, chunk, tile of the pass)
        struct { uint32_t i, b, c, t; } pf = {0, 0, 0, 0};
        auto skip_empty = [&]() {
#pragma unroll 1
            while (pf.i < 4 * L && kinds[pf.i & 3].n == 0) pf.i++;
        };
        auto prefetch_next = [&](bool fetch) {
            if (pf.i >= 4 * L) return;
            const Kind& k = kinds[pf.i & 3];
            if (fetch) tma_prefetch_rows(map + pf.i, pf.c * k.pieces, (k.t0 + pf.b + pf.t) * 8);
            if (++pf.t < min(TB, k.n - pf.b)) return;
            pf.t = 0;
            if (++pf.c < k.chunks) return;
            pf.c = 0;
            if ((pf.b += TB) < k.n) return;
            pf.b = 0;
            pf.i++;
            skip_empty();
        };
        if constexpr (CAN_AHEAD) {
            skip_empty();
#pragma unroll 1
            for (uint32_t n = 0; ahead && n < slots + ahead; n++) prefetch_next(n >= slots);
        }
#pragma unroll 1
        for (uint32_t i = 0; i < 4 * L && ok; i++) {
            const Kind& d = kinds[i & 3];
#pragma unroll 1
            for (uint32_t b = 0; b < d.n && ok; b += TB) {
                const uint32_t nt = min(TB, d.n - b);
#pragma unroll 1
                for (uint32_t c = 0; c < d.chunks && ok; c++) {
#pragma unroll 1
                    for (uint32_t t = 0; t < nt; t++) {
                        if (sent >= slots) ok = wait_bar(&empty_bar[q.s], q.ph ^ 1u, expiry);
                        if (!ok) break;
                        mbar_expect_tx(&full_bar[q.s], 8 * d.pitch);
                        tma_load_rows(smem + q.s * SLOT, map + i, c * d.pieces, (d.t0 + b + t) * 8, &full_bar[q.s], pol);
                        sent++;
                        q.advance(1, slots);
                        if (CAN_AHEAD && ahead) prefetch_next(true);
                    }
                }
            }
        }
        uint32_t head_sent = 0;
        {
            const Kind& d = kinds[HEAD];
#pragma unroll 1
            for (uint32_t t = 0, c = 0; t < d.n && ok; c = c + 1 < d.chunks ? c + 1 : 0, t += c == 0) {
                const uint32_t lap = head_sent / head_slots, r = head_sent - lap * head_slots, x = r < slots ? 0 : MAX_SLOTS + r - slots;
                const uint32_t bar = r < slots ? q.s : x;
                if (r < slots) {
                    if (sent >= slots) ok = wait_bar(&empty_bar[bar], q.ph ^ 1u, expiry);
                } else {
                    ok = lap ? wait_bar(&empty_bar[bar], (lap - 1) & 1u, expiry) : wait_bar(&kv_free_bar, 0, expiry);
                }
                if (!ok) break;
                mbar_expect_tx(&full_bar[bar], 8 * d.pitch);
                *(volatile uint32_t*)&use_sm[bar] = 1 + (r < slots ? sent / slots : lap);
                tma_load_rows(r < slots ? smem + bar * SLOT : extra_sm + (r - slots) * SLOT, map + 4 * L, c * d.pieces, (d.t0 + t) * 8, &full_bar[bar], pol);
                head_sent++;
                if (r < slots) {
                    sent++;
                    q.advance(1, slots);
                }
            }
        }
        // leave when every copy has landed: the last use of each slot (q stands on the oldest)
        const uint32_t n = min(sent, slots);
#pragma unroll 1
        for (uint32_t i = 0; i < n; i++) {
            if (sent < slots) { q.s = i; q.ph = 1; }
            mbar_wait(&full_bar[q.s], q.ph ^ 1u);
            q.advance(1, slots);
        }
#pragma unroll 1
        for (uint32_t r = slots; r < min(head_sent, head_slots); r++) mbar_wait(&full_bar[MAX_SLOTS + r - slots], ((head_sent - r - 1) / head_slots) & 1u);
        if (expiry.is_dead()) report();
        return;
    }
    if (warp_ < FIRST_COMPUTE) {
        // ---------------- epilogue: warp e has the e-th tile of a pass. It adds the compute warps' partial sums, applies the norm's factor or
        // adds to the residual stream, and publishes; the compute warps are then already at the next phase. Also the embedding, the sums of
        // squares of the norms, the clearing of exchange sets.
        const uint32_t ht = tid - 32, e = warp_ - 1, h = lane & 1;   // lane: row 16 m + lane / 2, columns 4 h .. 4 h + 3 of the tile
        const uint32_t rl = lane >> 1;
        constexpr uint32_t PB = 12;   // partial sums read together
        auto clear = [&](uint32_t g) {
            uint4* p = reinterpret_cast<uint4*>(a.xch + set_of(g));
            const uint32_t n = (uint32_t)(so.total / 16);
#pragma unroll 1
            for (uint32_t i = cta * NHT + ht; i < n; i += a.sms * NHT) p[i] = make_uint4(EMPTY, EMPTY, EMPTY, EMPTY);
            bar_sync<NHT>(BAR_HELP);
            if (ht == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&state->cleared) : "memory");
        };
        const uint32_t counted = *(const volatile uint32_t*)&state->counted;
        auto wait_cleared = [&](uint32_t clears) {
            if (lane == 0) {
                uint32_t n = 0, v;
                Waiter w = wt;
                do asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&state->cleared) : "memory");
                while ((int32_t)(v - counted - clears * a.sms) < 0 && !w.give_up(n));
            }
            __syncwarp();
        };
        uint32_t nb = 0;
        // 1 / rms of the lane's rows
        auto factors = [&](uint32_t off, float (&f)[MT]) {   // lane (i / Q, i % Q) reads four rows of tile i / Q, + TPL, .. of this warp's
            const uint32_t n = D / 8, step = NH * TPL;
            const uint8_t* const sl = a.xch + off + lane % Q * 16;
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (uint32_t t0 = e * TPL + lane / Q; t0 < n; t0 += 4 * step) {
                uint4 y[4];
                uint32_t polls = 0;
                bool lack;
                Waiter w = wt;
#pragma unroll
                for (uint32_t d = 0; d < 4; d++) y[d].x = y[d].y = y[d].z = y[d].w = t0 + d * step < n ? EMPTY : 0u;
#pragma unroll 1
                do {
#pragma unroll
                    for (uint32_t d = 0; d < 4; d++)
                        if (max(max(y[d].x, y[d].y), max(y[d].z, y[d].w)) == EMPTY) y[d] = xld4(sl + (t0 + d * step) * (R * 4));
                    uint32_t mx = 0;
#pragma unroll
                    for (uint32_t d = 0; d < 4; d++) mx = max(max(mx, max(y[d].x, y[d].y)), max(y[d].z, y[d].w));
                    lack = mx == EMPTY;
                } while (lack && !w.give_up(polls));
#pragma unroll
                for (uint32_t d = 0; d < 4; d++) {
                    sum.x += __uint_as_float(y[d].x); sum.y += __uint_as_float(y[d].y);
                    sum.z += __uint_as_float(y[d].z); sum.w += __uint_as_float(y[d].w);
                }
            }
            __syncwarp();
#pragma unroll
            for (uint32_t o = Q; o < 32; o <<= 1) {
                sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o); sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
                sum.z += __shfl_xor_sync(0xffffffffu, sum.z, o); sum.w += __shfl_xor_sync(0xffffffffu, sum.w, o);
            }
            if (lane < Q) *reinterpret_cast<float4*>(&ss_sm[nb][e][lane * 4]) = sum;
            bar_sync<NHT>(BAR_HELP);
#pragma unroll
            for (uint32_t m = 0; m < MT; m++) {
                const float* const s = &ss_sm[nb][0][m * 16 + rl];
                f[m] = inv_rms((s[0] + s[R] + s[2 * R]) * inv_dim + a.eps);
            }
            nb ^= 1u;
        };
        // publish 8 columns (the vector of a tile) held by two lanes; whole warps
        auto put8 = [&](uint32_t dst, bool eight, const float4& v) {
            const uint32_t w0 = pack2(v.x, v.y), w1 = pack2(v.z, v.w);
            const uint32_t w2 = __shfl_down_sync(0xffffffffu, w0, 1), w3 = __shfl_down_sync(0xffffffffu, w1, 1);
            if (h == 0 && eight) xst4(a.xch + dst, w0, w1, w2, w3);
        };
        // publish the residual stream, multiplied by the next norm's gain, and the sums of squares of whole tiles
        auto put_x = [&](uint32_t xd, uint32_t sd, bool eight, const float4& x, const float4& g) {
            put8(xd, eight, make_float4(x.x * g.x, x.y * g.y, x.z * g.z, x.w * g.w));
            float s = (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (h == 0) xst1(a.xch + sd, word(s));   // (of every row: 0 where there is no sequence)
        };
        if (lane == 0) mbar_arrive(&free_bar);
        // ---- embedding
        if (e < kinds[OUT].n) {
            const uint32_t tile = kinds[OUT].t0 + e;
            const float4 g = *reinterpret_cast<const float4*>(gain_sm + e * 8 + h * 4);
#pragma unroll
            for (uint32_t m = 0; m < MT; m++) {
                const uint32_t row = m * 16 + rl;
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (row_live(row)) {
                    const int32_t ts = a.rows ? a.rows[slot_of(row) * 4] : a.tok_src[slot_of(row)];
                    const uint32_t id = ts >= 0 ? (uint32_t)ts : a.sampled[slot_of(row)];
                    if (id < a.vocab) {
                        const uint2 w = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(a.embedding) + (size_t)id * D + tile * 8 + h * 4);
                        x = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
                    }
                }
                __syncwarp();
                res_sm[(e * R + row) * 2 + h] = x;
                put_x(set_of(e0) + so.x1 + frag<MT>(row, tile), set_of(e0) + so.s1 + (tile * R + row) * 4, eight_live(row >> 3), x, g);
            }
        }
        // Set g may be cleared when everybody has read what there is in it: when ss2 of layer g + 1 is complete, out-proj of layer g + 1 is done, with
        // it attention and qkv of that layer, so ffn-down of layer g (the last readers of set g but for x1 and ss1, which qkv of layer g + 1
        // has read). And it has to be cleared before anybody polls its next content or writes it: see clears_before_out(). The count goes up by a
        // release behind all stores of an SM's epilogue and is awaited with an acquire that the compute warps get with the next free_bar, so
        // the clears are ordered before those polls whatever was read in between. Nothing waits here in earnest: the count is two phases old.
        // The set of the step's embedding stands for a layer. The last layer's set is cleared when the next step starts.
        clear(e0 + SETS - 1);
#pragma unroll 1
        for (uint32_t i = 0; i < 4 * L; i++) {
            const uint32_t l = i >> 2, ph = i & 3, set = set_of(e0 + 1 + l);
            const Kind& d = kinds[ph];
            const uint32_t tiles = d.n;
            const bool norm = ph == QKV || ph == FFN_UP;
            float f[MT];
#pragma unroll
            for (uint32_t m = 0; m < MT; m++) f[m] = 1.0f;
            if (ph == OUT) wait_cleared(clears_before_out(l));
            // A row without a sequence is published as zeros where a row of its eight has one (the consumers look at whole eights only). Here its
            // attention, by the SM with the row's number among its qkv tiles.
            if (ph == QKV) {
#pragma unroll 1
                for (uint32_t r = d.t0; r < min(d.t0 + tiles, R); r++)
                    if (!row_live(r) && eight_live(r >> 3)) {
#pragma unroll 1
                        for (uint32_t v = ht; v < D / 8; v += NHT) xst4(a.xch + set + so.at + frag<MT>(r, v), 0, 0, 0, 0);
                    }
            }
#pragma unroll 1
            for (uint32_t b = 0; b < tiles; b += TB) {
                const bool has = b + e < tiles;
                const uint32_t tile = d.t0 + b + e;
                // all that does not need the sums
                uint32_t dst[MT], sd[MT];
                float4 res[MT], g = make_float4(0.f, 0.f, 0.f, 0.f);
                if (has) {
                    if (!norm) g = *reinterpret_cast<const float4*>(gain_sm + ((2 * l + (ph == OUT ? 1 : 2)) * tiles + e) * 8 + h * 4);
#pragma unroll
                    for (uint32_t m = 0; m < MT; m++) {
                        const uint32_t row = m * 16 + rl;
                        res[m] = make_float4(0.f, 0.f, 0.f, 0.f);
                        sd[m] = 0;
                        if (ph == QKV) dst[m] = set + so.qkv + (row * 3 * D + tile * 8 + h * 4) * 4;
                        else dst[m] = set + (ph == OUT ? so.x2 : ph == FFN_UP ? so.up : so.x1) + frag<MT>(row, tile);
                        if (!norm) {
                            res[m] = res_sm[(e * R + row) * 2 + h];
                            sd[m] = set + (ph == OUT ? so.s2 : so.s1) + (tile * R + row) * 4;
                        }
                    }
                }
                const float* const o = part + e * (R * 8) + lane * 4;
                if (norm && b == 0) factors(ph == QKV ? set_of(e0 + l) + so.s1 : set + so.s2, f);
                bar_sync<NCT + NHT>(BAR_PART);
                if (has) {
#pragma unroll
                    for (uint32_t m = 0; m < MT; m++) {
                        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (uint32_t w0 = 0; w0 < NW; w0 += PB) {
                            float4 y[PB];
#pragma unroll
                            for (uint32_t w = 0; w < PB; w++) y[w] = *reinterpret_cast<const float4*>(o + (w0 + w) * (TB * R * 8) + m * 128);
#pragma unroll
                            for (uint32_t w = 0; w < PB; w += 4) {   // in pairs
                                v.x += (y[w].x + y[w + 1].x) + (y[w + 2].x + y[w + 3].x); v.y += (y[w].y + y[w + 1].y) + (y[w + 2].y + y[w + 3].y);
                                v.z += (y[w].z + y[w + 1].z) + (y[w + 2].z + y[w + 3].z); v.w += (y[w].w + y[w + 1].w) + (y[w + 2].w + y[w + 3].w);
                            }
                        }
                        const uint32_t row = m * 16 + rl;
                        if (!norm) {
                            v.x += res[m].x; v.y += res[m].y; v.z += res[m].z; v.w += res[m].w;
                            put_x(dst[m], sd[m], eight_live(row >> 3), v, g);
                            res_sm[(e * R + row) * 2 + h] = v;
                            continue;
                        }
                        v.x *= f[m]; v.y *= f[m]; v.z *= f[m]; v.w *= f[m];
                        if (ph == QKV) {
                            if (row_live(row)) xst4(a.xch + dst[m], word(v.x), word(v.y), word(v.z), word(v.w));
                            continue;
                        }
                        // SiLU (off by 2^-17 of the value at most, and 0 below about -87: far below the rounding to bf16)
                        v.x = __fdividef(v.x, 1.0f + __expf(-v.x)); v.y = __fdividef(v.y, 1.0f + __expf(-v.y));
                        v.z = __fdividef(v.z, 1.0f + __expf(-v.z)); v.w = __fdividef(v.w, 1.0f + __expf(-v.w));
                        put8(dst[m], eight_live(row >> 3), v);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&free_bar);
            }
            if (ph == FFN_UP) clear(e0 + l);
        }
        // The picks leave out 1 / rms, which changes no order, but for a row whose sum of squares overflowed: there it is 0, and so are all logits.
        if (e == 0 && cta < R && row_live(cta)) {
            float sum = 0.0f;
#pragma unroll 1
            for (uint32_t t = lane; t < D / 8; t += 32) {
                uint32_t y, n = 0;
                Waiter w = wt;
#pragma unroll 1
                do y = xld1(a.xch + set_of(e0 + L) + so.s1 + (t * R + cta) * 4);
                while (y == EMPTY && !w.give_up(n));
                sum += __uint_as_float(y);
            }
            __syncwarp();
            sum = warp_sum(sum);
            if (lane == 0) flat_sm = sum == INFINITY;
            __syncwarp();
            bar_arrive<64>(BAR_FLAT);
        }
        if (lane == 0 && expiry.is_dead()) report();
        return;
    }

    // ---------------- compute warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_COMPUTE));
    const uint32_t cw = warp_ - FIRST_COMPUTE, ct = cw * 32 + lane;
    bool alive = true;   // no wait of this warp for a copy has run out (after the first that did it releases no slot)
    Cursor q;
    const uint32_t frag_lane = (lane & 3) * 8 + (lane >> 2);
    uint32_t part_ph = 0;           // parity of the use of the partial sums
    uint32_t a_live = 0;            // the eights of the rows that have a sequence
#pragma unroll
    for (uint32_t e = 0; e < 2 * MT; e++) a_live |= (eight_live(e) ? 1u : 0u) << e;

    // The warp's share of NT tiles of projection `kind`; x: A fragments. What a phase spends its time on is dependent instructions, ~5 cycles each, and
    // round trips to L2, ~1 us each, so all that can be is done before the activations arrive: the weights are in registers, addresses are known.
    // CPG: chunks of a group (what a warp requests together, as many as there are registers for). With K of one chunk the activations stay
    // in v for the later passes over the same ones (loaded).
    auto pass = [&](auto nt_c, auto cpg_c, uint32_t x, const Kind& kind, auto& v, bool loaded) {
        constexpr uint32_t NT = decltype(nt_c)::value, CPG = decltype(cpg_c)::value, DEPTH = CPG * PPC;
        const uint32_t chunks = kind.chunks, slices = kind.slices, pitch = kind.pitch;
        // the warp's slices cw + NW i, i < nsl
        const uint32_t nsl = cw < slices ? (slices - cw + NW - 1) / NW : 0;
        const uint8_t* xl = a.xch + (x + cw * (MT * 1024) + frag_lane * 16);
        constexpr uint32_t STEP = NW * MT * 1024;
        const uint32_t w_off = (lane >> 2) * pitch + cw * 64 + (lane & 3) * 16;
        float acc[NT][MT][4];
#pragma unroll
        for (uint32_t t = 0; t < NT; t++)
#pragma unroll
            for (uint32_t m = 0; m < MT; m++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[t][m][i] = 0.0f;
        auto issue = [&](uint32_t i0) {
#pragma unroll
            for (uint32_t d = 0; d < DEPTH; d++)
                if (i0 + d < nsl) {
#pragma unroll
                    for (uint32_t e = 0; e < 2 * MT; e++)
                        if (a_live >> e & 1u) v[d][e >> 1][e & 1] = xld4(xl + d * STEP + e * 512);
                }
        };
        uint32_t used = 0;   // slots before q that are not given back yet (a group's)
        auto release = [&]() {
            if (lane < used && alive) {
                const uint32_t back = used - lane;
                mbar_arrive(&empty_bar[q.s >= back ? q.s - back : q.s + slots - back]);
            }
        };
        if (!loaded) {
#pragma unroll
            for (uint32_t d = 0; d < DEPTH; d++)
#pragma unroll
                for (uint32_t e = 0; e < 2 * MT; e++) v[d][e >> 1][e & 1] = make_uint4(0, 0, 0, 0);
            issue(0);
        }
#pragma unroll 1
        for (uint32_t c0 = 0;;) {
            // the group's weights
            used = 0;
            uint4 w[DEPTH][NT];
#pragma unroll
            for (uint32_t cc = 0; cc < CPG; cc++)
                if (cc == 0 || c0 + cc < chunks) {
                    Cursor mine = q;
                    mine.advance(lane < NT ? lane : 0, slots);
                    const bool got = lane >= NT || wait_bar(&full_bar[mine.s], mine.ph, expiry);
                    alive = __all_sync(0xffffffffu, got && alive) != 0;
                    __syncwarp();   // (a vote orders no memory: without this the lanes that do not wait may read before the weights are there)
#pragma unroll
                    for (uint32_t t = 0; t < NT; t++) {
                        const uint32_t at = (q.s + t < slots ? q.s + t : q.s + t - slots) * SLOT + w_off;
#pragma unroll
                        for (uint32_t j = 0; j < PPC; j++)   // (past the end of K: what the slot held, for products that are left out)
                            w[cc * PPC + j][t] = *reinterpret_cast<const uint4*>(smem + at + j * (NW * 64));
                    }
                    q.advance(NT, slots);
                    used += NT;
                }
            // everything there?
            const uint32_t left = nsl - min(nsl, c0 * PPC);
            uint32_t polls = 0;
#pragma unroll 1
            for (;;) {
                uint32_t mx = 0;   // EMPTY is the largest word
#pragma unroll
                for (uint32_t d = 0; d < DEPTH; d++)
                    if (d < left) {
#pragma unroll
                        for (uint32_t e = 0; e < 2 * MT; e++) mx = max(mx, v[d][e >> 1][e & 1].x);
                    }
                Waiter wait = wt;
                if (!__any_sync(0xffffffffu, mx == EMPTY) || __any_sync(0xffffffffu, wait.give_up(polls))) break;
#pragma unroll
                for (uint32_t d = 0; d < DEPTH; d++)
                    if (d < left) {
#pragma unroll
                        for (uint32_t e = 0; e < 2 * MT; e++)
                            if (v[d][e >> 1][e & 1].x == EMPTY) v[d][e >> 1][e & 1] = xld4(xl + d * STEP + e * 512);
                    }
            }
#pragma unroll
            for (uint32_t d = 0; d < DEPTH; d++)
                if (d < left) {
#pragma unroll
                    for (uint32_t t = 0; t < NT; t++)
#pragma unroll
                        for (uint32_t m = 0; m < MT; m++) mma(acc[t][m], v[d][m][0].x, v[d][m][1].x, v[d][m][0].y, v[d][m][1].y, w[d][t].x, w[d][t].y);
#pragma unroll
                    for (uint32_t t = 0; t < NT; t++)
#pragma unroll
                        for (uint32_t m = 0; m < MT; m++) mma(acc[t][m], v[d][m][0].z, v[d][m][1].z, v[d][m][0].w, v[d][m][1].w, w[d][t].z, w[d][t].w);
                }
            c0 += CPG;
            if (c0 >= chunks) break;
            float all = acc[0][0][0];
#pragma unroll
            for (uint32_t t = 1; t < NT; t++) all += acc[t][0][0];
            if (settled(all)) release();
            xl += DEPTH * STEP;
            issue(c0 * PPC);
        }
        wait_block(&free_bar, part_ph, expiry);   // the sums that were there have been read
        part_ph ^= 1u;
        {
            float* const o = part + (cw * TB * R + (lane >> 2)) * 8 + (lane & 3) * 2;
#pragma unroll
            for (uint32_t t = 0; t < NT; t++)
#pragma unroll
                for (uint32_t m = 0; m < MT; m++) {
                    *reinterpret_cast<float2*>(o + (t * R + m * 16) * 8) = make_float2(acc[t][m][0], acc[t][m][1]);
                    *reinterpret_cast<float2*>(o + (t * R + m * 16 + 8) * 8) = make_float2(acc[t][m][2], acc[t][m][3]);
                }
        }
        __syncwarp();
        bar_arrive<NCT + NHT>(BAR_PART);
        release();   // (behind the stores, which waited for the products and so for the weights)
    };
    auto gemm = [&](uint32_t x, const Kind& kind) {
        const uint32_t tiles = kind.n;
        using std::integral_constant;
        constexpr integral_constant<uint32_t, 1> one{};
        uint4 kept[KEEP ? PPC : 1][MT][2];
        const bool keep = KEEP && kind.chunks == 1;
#pragma unroll 1
        for (uint32_t b = 0; b < tiles; b += TB) {
            const uint32_t nt = min(TB, tiles - b);
            auto of = [&](auto nt_c, auto cpg_c) {
                if constexpr (KEEP) {
                    pass(nt_c, one, x, kind, kept, keep && b > 0);
                } else {
                    uint4 v[decltype(cpg_c)::value * PPC][MT][2];
                    pass(nt_c, cpg_c, x, kind, v, false);
                }
            };
            if (nt == 1) of(one, integral_constant<uint32_t, MT == 1 ? 2 : 1>{});
            else if (nt == 2) of(integral_constant<uint32_t, 2>{}, one);
            else of(integral_constant<uint32_t, 3>{}, one);
        }
    };

    uint32_t tiles_done = 0;   // parity of the tiles worked through
    // ---- attention: units of this warp's group. What a warp keeps of it between layers is in shared memory (the projections need the registers).
    // (a multiplication by inv_wpi = 65536 / wpi + 1 divides the small numbers here)
    auto group_of = [&]() { return cw * inv_wpi >> 16; };
    auto in_group = [&](uint32_t i) { return i - (i * inv_wpi >> 16) * wpi; };   // i mod wpi
    auto place_in = [&]() { return in_group(cw); };
    {   // unit j in lane j: row | head << 6 | split << 18
        const uint32_t grp = group_of();
        const uint32_t groups = a.sms * (NW / wpi), gid = grp * a.sms + cta;
        const uint32_t u = lane * groups + ((lane & 1) ? groups - 1 - gid : gid);
        uint32_t unit = EMPTY;
        if (u < pre_sm[32] * H) {
            const uint32_t v = u / H;
            uint32_t lo = 0, hi = 32;   // the rank whose splits hold v
#pragma unroll 1
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (pre_sm[mid] <= v) lo = mid;
                else hi = mid;
            }
            unit = by_len[lo] | ((u % H) << 6) | ((v - pre_sm[lo]) << 18);
        }
        units[cw][lane] = unit;
        const uint32_t n = __popc(__ballot_sync(0xffffffffu, unit != EMPTY));
        if (lane == 0) walk_sm[cw].nu = n;
        __syncwarp();
    }
    // (of two parts a unit's row has the slot above it)
    auto row_in = [&](const Unit& u) { return PARTS > 1 ? u.row & 31u : u.row; };
    auto slot_in = [&](const Unit& u) { return PARTS > 1 ? u.row >> 5 : u.row; };
    auto unit_at = [&](uint32_t j) {
        const uint32_t u = units[cw][j];
        Unit o;
        o.row = u & 63; o.head = (u >> 6) & 0xfff; o.split = u >> 18;
        o.p0 = o.split * SPLIT_LEN;
        o.n = min(SPLIT_LEN, len_sm[o.row] - o.p0);
        o.nb = (o.n + UP - 1) / UP;
        if (PARTS > 1) o.row |= slot_sm[o.row] << 5;
        return o;
    };
    auto look_up = [&]() {   // the pool blocks of the walk's tile (lane 0)
        Walk& k = walk_sm[cw];
        const uint32_t p = k.b * UP;
        const int32_t* bt = a.block_tables + (size_t)slot_in(k.u) * a.max_blocks + (k.u.p0 + p) / 16;
        k.pb0 = (uint32_t)__ldg(bt);
        k.pb1 = UP > 16 && p + 16 < k.u.n ? (uint32_t)__ldg(bt + 1) : EMPTY;
    };
    uint8_t* const kbuf = kv_sm + cw * 2 * KV_BUF;
    uint8_t* const vbuf = kbuf + KV_BUF;
    // Request the keys or the values of the walk's tile; with the values the walk moves on. Called by the whole warp after it has read the buffer;
    // lane 0 does it, with the walk in shared memory.
    auto request = [&](bool values) {
        if (lane == 0 && alive && walk_sm[cw].more) {
            Walk& k = walk_sm[cw];
            const SoloLayer& w = layers_sm[k.l];
            const uint32_t pb0 = k.pb0, pb1 = k.pb1;
            uint64_t* bar = values ? &v_bar[cw] : &k_bar[cw];
            const bf16* pool = reinterpret_cast<const bf16*>(values ? w.v_pool : w.k_pool) + (size_t)k.u.head * (16 * HD);
            uint8_t* dst = values ? vbuf : kbuf;
            constexpr uint32_t TILE = 16 * HD * 2;
            mbar_expect_tx(bar, UP > 16 && pb1 != EMPTY ? 2 * TILE : TILE);
            const uint64_t pol = policy_evict_first();   // (read once a step; the exchange sets and weights stay in L2: 64 sequences 398 instead of 408 us)
            bulk_g2s_hint(dst, pool + (size_t)pb0 * H * (16 * HD), TILE, bar, pol);
            if (UP > 16 && pb1 != EMPTY) bulk_g2s_hint(dst + TILE, pool + (size_t)pb1 * H * (16 * HD), TILE, bar, pol);
            k.asked = !values;
            if (values) {
                k.sent++;
                walk_on(k, wpi, place_in(), L, unit_at, look_up);
            }
        }
        __syncwarp();
    };
    {
        if (lane == 0) {
            Walk& k = walk_sm[cw];
            k.l = k.j = k.more = k.asked = k.sent = 0;
            k.b = place_in();
#pragma unroll 1
            for (uint32_t j = k.nu; j-- > 0;)   // the first unit with a tile for this warp (if there is one there is one in every layer)
                if (place_in() < unit_at(j).nb) { k.more = 1; k.j = j; }
            if (k.more) {
                k.u = unit_at(k.j);
                look_up();
            }
        }
        __syncwarp();
        request(false);
        request(true);
    }

    // publish a head of a row: lane i has its columns DL i .. DL i + DL - 1, to be divided by ls
    constexpr uint32_t DL = HD / 32;
    auto put_at = [&](uint32_t set, uint32_t row, uint32_t head, const float (&o)[DL], float ls) {
        const float r = __fdividef(1.0f, ls);   // (2 ulp, before a rounding to bf16)
        uint32_t w[4];
        w[0] = pack2(o[0] * r, o[1] * r);
        if constexpr (DL == 2) {
#pragma unroll
            for (int i = 1; i < 4; i++) w[i] = __shfl_down_sync(0xffffffffu, w[0], i);
        } else {
            w[1] = pack2(o[DL - 2] * r, o[DL - 1] * r);
            w[2] = __shfl_down_sync(0xffffffffu, w[0], 1);
            w[3] = __shfl_down_sync(0xffffffffu, w[1], 1);
        }
        if (lane % (8 / DL) == 0) {
            uint8_t* const dst = a.xch + set + so.at + frag<MT>(row, (head * HD + lane * DL) >> 3);
            xst4(dst, w[0], w[1], w[2], w[3]);
        }
    };

    auto attention = [&](const SoloLayer& lw, uint32_t set) {
        const uint32_t chunk = lane % CH;
        const uint8_t* const qkv = a.xch + set + so.qkv;
        const uint32_t grp = group_of(), wg = place_in(), nu = walk_sm[cw].nu;
#pragma unroll 1
        for (uint32_t j = 0; j < nu; j++) {
            const Unit u = unit_at(j);
            const uint32_t buf = j & 1, pos = len_sm[row_in(u)] - 1;
            const bool newest = u.p0 + u.n == pos + 1;   // the unit holds the sequence's new position
            constexpr uint32_t KT = UP / 8, NS = HD / 32;   // eights of positions in a tile; k slices of a score
            float m = -INFINITY, l = 0.0f, acc[8];   // this lane's 8 columns, of its share of the positions
#pragma unroll
            for (int e = 0; e < 8; e++) acc[e] = 0.0f;
            if (wg < u.nb) {
                // This lane's 8 columns of the new token's query; of the newest tile's warp also of its key and value, which go to the pools and
                // (below) into the tile. All of it, the rotation's factors and the place in the pools are asked for together.
                const bool owner = newest && wg == in_group(u.nb - 1);
                const uint8_t* const src = qkv + ((size_t)row_in(u) * 3 * D + u.head * HD + chunk * 8) * 4;
                const float4* const rt = reinterpret_cast<const float4*>(a.rope + (size_t)pos * (HD / 2) + chunk * 4);
                const float4 r0 = __ldg(rt), r1 = __ldg(rt + 1);
                const uint32_t pb = owner ? (uint32_t)__ldg(a.block_tables + (size_t)slot_in(u) * a.max_blocks + pos / 16) : 0u;
                uint4 qa[NS], kn = make_uint4(0, 0, 0, 0), vn = kn;
                {
                    uint4 x[6] = {};
                    uint32_t n = 0;
                    Waiter w = wt;
#pragma unroll
                    for (int i = 0; i < 6; i++) x[i].x = i < 2 || owner ? EMPTY : 0u;
                    bool lack;
#pragma unroll 1
                    do {
#pragma unroll
                        for (int i = 0; i < 6; i++)
                            if (x[i].x == EMPTY) x[i] = xld4(src + (size_t)(i >> 1) * D * 4 + (i & 1) * 16);
                        lack = max(max(x[0].x, x[1].x), max(max(x[2].x, x[3].x), max(x[4].x, x[5].x))) == EMPTY;
                    } while (__any_sync(0xffffffffu, lack) && !__any_sync(0xffffffffu, w.give_up(n)));
                    auto packed = [&](const uint4& lo, const uint4& hi, bool rotate) {
                        float o[8] = {__uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(lo.z), __uint_as_float(lo.w),
                                      __uint_as_float(hi.x), __uint_as_float(hi.y), __uint_as_float(hi.z), __uint_as_float(hi.w)};
                        if (rotate) {
                            rope_rotate(o[0], o[1], r0.x, r0.y, o[0], o[1]);
                            rope_rotate(o[2], o[3], r0.z, r0.w, o[2], o[3]);
                            rope_rotate(o[4], o[5], r1.x, r1.y, o[4], o[5]);
                            rope_rotate(o[6], o[7], r1.z, r1.w, o[6], o[7]);
                        }
                        return make_uint4(pack2(o[0], o[1]), pack2(o[2], o[3]), pack2(o[4], o[5]), pack2(o[6], o[7]));
                    };
                    const uint4 qn = packed(x[0], x[1], true);
                    // A fragments: slice s of lane (g, t) is vector 4 s + t, held by the lane of that chunk
#pragma unroll
                    for (uint32_t s = 0; s < NS; s++) {
                        const uint32_t from = s * 4 + (lane & 3);
                        qa[s] = make_uint4(__shfl_sync(0xffffffffu, qn.x, from), __shfl_sync(0xffffffffu, qn.y, from), __shfl_sync(0xffffffffu, qn.z, from),
                                           __shfl_sync(0xffffffffu, qn.w, from));
                    }
                    if (owner) {
                        kn = packed(x[2], x[3], true);
                        vn = packed(x[4], x[5], false);
                        if (lane < CH) {
                            const size_t prow = (((size_t)pb * H + u.head) * 16 + (pos & 15)) * HD + chunk * 8;
                            *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(lw.k_pool) + prow) = kn;
                            *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(lw.v_pool) + prow) = vn;
                        }
                    }
                }
                const float sc = a.scale * 1.44269504088896f;   // scores in units of ln 2
#pragma unroll 1
                for (uint32_t b = wg; b < u.nb; b += wpi) {
                    const uint32_t left = u.n - b * UP;   // positions of the tile that count, if fewer than UP
                    const bool fresh = newest && left <= UP;
                    const uint32_t at = (left - 1) * (HD * 2) + chunk * 16;   // the new position's row in the buffers
                    alive = wait_bar(&k_bar[cw], tiles_done & 1u, expiry) && alive;
                    if (fresh) {
                        if (lane < CH) {
                            *reinterpret_cast<uint4*>(kbuf + at) = kn;
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // before the next tile's copy into the buffer
                        }
                        __syncwarp();
                    }
                    float p[KT][2];   // positions 8 n + 2 t, + 1 (t = lane % 4)
#pragma unroll
                    for (uint32_t n = 0; n < KT; n++) {
                        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (uint32_t s = 0; s < NS; s++) {
                            const uint4 w = *reinterpret_cast<const uint4*>(kbuf + (n * 8 + (lane >> 2)) * (HD * 2) + s * 64 + (lane & 3) * 16);
                            mma(c, qa[s].x, qa[s].x, qa[s].y, qa[s].y, w.x, w.y);
                            mma(c, qa[s].z, qa[s].z, qa[s].w, qa[s].w, w.z, w.w);
                        }
                        p[n][0] = c[0];
                        p[n][1] = c[1];
                    }
                    float mx = -INFINITY;
#pragma unroll
                    for (uint32_t n = 0; n < KT; n++)
#pragma unroll
                        for (uint32_t e = 0; e < 2; e++) {
                            if (n * 8 + (lane & 3) * 2 + e >= left) p[n][e] = -INFINITY;
                            mx = fmaxf(mx, p[n][e]);
                        }
                    const float m2 = fmaxf(m, redux_max(mx) * sc), corr = ex2(m - m2);
                    if (__float_as_uint(m2) != EMPTY) request(false);   // (always, but with all lanes' scores there: see settled)
                    m = m2;
                    l *= corr;
                    // Every four lanes hold all probabilities; lane (g, t) keeps those of positions 8 n + 2 t + (g & 1) to hand out
#pragma unroll
                    for (uint32_t n = 0; n < KT; n++) {
                        p[n][0] = ex2(fmaf(p[n][0], sc, -m2));
                        p[n][1] = ex2(fmaf(p[n][1], sc, -m2));
                        l += p[n][0] + p[n][1];
                        p[n][0] = (lane & 4) ? p[n][1] : p[n][0];
                    }
#pragma unroll
                    for (int e = 0; e < 8; e++) acc[e] *= corr;
                    alive = wait_bar(&v_bar[cw], tiles_done & 1u, expiry) && alive;
                    if (fresh) {   // what lies behind the sequence's end is anything, a NaN even
                        if (lane < CH) *reinterpret_cast<uint4*>(vbuf + at) = vn;
#pragma unroll 1
                        for (uint32_t z = left * CH + lane; z < UP * CH; z += 32) *reinterpret_cast<uint4*>(vbuf + z * 16) = make_uint4(0, 0, 0, 0);
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                    }
                    // values: this lane's vector i is of position PPI i + lane / CH
#pragma unroll
                    for (uint32_t i = 0; i < 8; i++) {
                        const uint32_t r = (i * PPI & 7) + lane / CH;   // of the eight i PPI / 8
                        const float pv = __shfl_sync(0xffffffffu, p[i * PPI / 8][0], (r & 1) * 4 + (r >> 1));
                        float vx[8];
                        unpack8(*reinterpret_cast<const uint4*>(vbuf + i * 512 + lane * 16), vx);
#pragma unroll
                        for (int e = 0; e < 8; e++) acc[e] = fmaf(pv, vx[e], acc[e]);
                    }
                    if (settled(acc[0])) request(true);
                    tiles_done ^= 1u;
                }
            }
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            {   // the warp's sums over its shares of the positions (lanes with the same chunk)
                float* const my_acc = at_acc + (buf * NW + cw) * HD + chunk * 8;
                const bool h16 = lane & 16;
                float t4[4];
#pragma unroll
                for (int i = 0; i < 4; i++) t4[i] = (h16 ? acc[4 + i] : acc[i]) + __shfl_xor_sync(0xffffffffu, h16 ? acc[i] : acc[4 + i], 16);
                if (CH == 8) {
                    const bool h8 = lane & 8;
                    float t2[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) t2[i] = (h8 ? t4[2 + i] : t4[i]) + __shfl_xor_sync(0xffffffffu, h8 ? t4[i] : t4[2 + i], 8);
                    *reinterpret_cast<float2*>(my_acc + (h16 ? 4 : 0) + (h8 ? 2 : 0)) = make_float2(t2[0], t2[1]);
                } else {
                    *reinterpret_cast<float4*>(my_acc + (h16 ? 4 : 0)) = make_float4(t4[0], t4[1], t4[2], t4[3]);
                }
            }
            if (lane == 0) at_ml[buf][cw] = make_float2(m, l);
            bar_sync_n(BAR_GROUP + grp, wpi * 32);
            if (wg == in_group(j)) {   // one warp merges the group's, in warp order
                const float2 ml = lane < wpi ? at_ml[buf][grp * wpi + lane] : make_float2(-INFINITY, 0.0f);
                const float M = redux_max(ml.x), f = ex2(ml.x - M), ls = warp_sum(ml.y * f);
                float o[DL];
#pragma unroll
                for (uint32_t e = 0; e < DL; e++) o[e] = 0.0f;
                const float* src = at_acc + (buf * NW + grp * wpi) * HD + lane * DL;
#pragma unroll 4
                for (uint32_t w = 0; w < wpi; w++) {
                    const float fw = __shfl_sync(0xffffffffu, f, w);
#pragma unroll
                    for (uint32_t e = 0; e < DL; e++) o[e] = fmaf(src[w * HD + e], fw, o[e]);
                }
                if (!SPLIT || len_sm[row_in(u)] <= SPLIT_LEN) {
                    put_at(set, row_in(u), u.head, o, ls);
                } else {
                    uint8_t* dst = a.xch + set + so.part + ((size_t)(row_in(u) * H + u.head) * splits + u.split) * (HD + 4) * 4;
                    if constexpr (DL == 2) xst2(dst + lane * 8, word(o[0]), word(o[1]));
                    else xst4(dst + lane * 16, word(o[0]), word(o[1]), word(o[DL - 2]), word(o[DL - 1]));
                    if (lane == 0) xst2(dst + HD * 4, word(M), word(ls));
                }
            }
        }
        // rows of several splits, each (row, head) by one warp of the chip: after all of its own units, so that nobody waits for a unit behind a merge
        if (SPLIT) {
#pragma unroll 1
            for (uint32_t i = cw * a.sms + cta; i < n_act * H; i += NW * a.sms) {
                const uint32_t row = by_len[i / H], head = i % H, n = len_sm[row], ns = div_up(n, SPLIT_LEN);
                if (ns <= 1) break;   // (longest first)
                const uint8_t* src = a.xch + set + so.part + (size_t)(row * H + head) * splits * (HD + 4) * 4;
                float M = -INFINITY, ls = 0.0f, o[DL];
#pragma unroll
                for (uint32_t e = 0; e < DL; e++) o[e] = 0.0f;
#pragma unroll 1
                for (uint32_t s0 = 0; s0 < ns; s0 += 2) {
                    uint2 ml[2], x[2][DL / 2];
                    auto get = [&](int k) {
                        const uint8_t* p = src + (size_t)(s0 + k) * (HD + 4) * 4;
                        ml[k] = xld2(p + HD * 4);
#pragma unroll
                        for (uint32_t e = 0; e < DL / 2; e++) x[k][e] = xld2(p + lane * (DL * 4) + e * 8);
                    };
                    auto lacks = [&](int k) {
                        bool b = ml[k].x == EMPTY || ml[k].y == EMPTY;
#pragma unroll
                        for (uint32_t e = 0; e < DL / 2; e++) b = b || x[k][e].x == EMPTY || x[k][e].y == EMPTY;
                        return b;
                    };
#pragma unroll
                    for (int k = 0; k < 2; k++)
                        if (s0 + k < ns) get(k);
                    uint32_t tries = 0;
#pragma unroll 1
                    for (;;) {
                        bool again = false;
#pragma unroll
                        for (int k = 0; k < 2; k++)
                            if (s0 + k < ns && lacks(k)) { get(k); again = true; }
                        Waiter w = wt;
                        if (!again || w.give_up(tries)) break;
                    }
#pragma unroll
                    for (int k = 0; k < 2; k++)
                        if (s0 + k < ns) {
                            const float pm = __uint_as_float(ml[k].x), m2 = fmaxf(M, pm), f0 = ex2(M - m2), f1 = ex2(pm - m2);
                            M = m2;
                            ls = ls * f0 + __uint_as_float(ml[k].y) * f1;
#pragma unroll
                            for (uint32_t e = 0; e < DL; e++) o[e] = o[e] * f0 + __uint_as_float(e & 1 ? x[k][e / 2].y : x[k][e / 2].x) * f1;
                        }
                }
                put_at(set, row, head, o, ls);
            }
            __syncwarp();
        }
    };

#pragma unroll 1
    for (uint32_t i = 0; i < 4 * L; i++) {
        const uint32_t l = i >> 2, ph = i & 3, set = set_of(e0 + 1 + l);
        if (ph == OUT) {
            attention(layers_sm[l], set);
            if (l + 1 == L && lane == 0) mbar_arrive(&kv_free_bar);   // (its tiles have been read)
        }
        gemm(ph == QKV ? set_of(e0 + l) + so.x1 : set + (ph == OUT ? so.at : ph == FFN_UP ? so.x2 : so.up), kinds[ph]);
    }
    // ---- lm_head and greedy argmax. The last x goes to shared memory (where the cache tiles were), and a warp has a tile of the weights to itself: no
    // sums across warps. A row's 1 / rms is left out, it does not change which logit is the largest.
    {
        const uint32_t fin = set_of(e0 + L) + so.best, x = set_of(e0 + L) + so.x1;
        const Kind& d = kinds[HEAD];
        uint4* const xs = reinterpret_cast<uint4*>(kv_sm);   // [slice][m][half][lane]
#pragma unroll 1
        for (uint32_t sl = cw; sl < d.slices; sl += NW)
#pragma unroll
            for (uint32_t p = 0; p < 2 * MT; p++) {
                uint4 v = make_uint4(0, 0, 0, 0);
                uint32_t n = 0;
                Waiter w = wt;
                if (a_live >> p & 1u)
#pragma unroll 1
                    do v = xld4(a.xch + x + (sl * (2 * MT) + p) * 512 + frag_lane * 16);
                    while (v.x == EMPTY && !w.give_up(n));
                xs[(sl * (2 * MT) + p) * 32 + lane] = v;
            }
        __syncwarp();
        bar_sync<NCT>(BAR_HEAD);
        float best_v[2 * MT];   // rows 8 p + lane / 4, of this lane's columns
        uint32_t best_i[2 * MT];
#pragma unroll
        for (uint32_t p = 0; p < 2 * MT; p++) { best_v[p] = -INFINITY; best_i[p] = NO_LOGIT; }
        // The chunks of tile t are numbers per t .. of the lm_head's; `base` chunks went through the ring before. Only the tile's warp waits for them, so it
        // looks first whether the slot is in that use at all: a parity alone would take the use before the last for it.
        const uint32_t per = d.chunks, busy = min(NW, max(1u, head_slots / per));   // (more warps than the ring holds tiles would only wait)
        uint32_t base = 0;
#pragma unroll 1
        for (uint32_t k = 0; k < HEAD; k++) base += L * kinds[k].n * kinds[k].chunks;
#pragma unroll 1
        for (uint32_t t = cw; t < d.n && cw < busy; t += busy) {
            float acc[MT][4], odd[MT][4];   // two chains of products
#pragma unroll
            for (uint32_t m = 0; m < MT; m++)
#pragma unroll
                for (int k = 0; k < 4; k++) acc[m][k] = odd[m][k] = 0.0f;
#pragma unroll 1
            for (uint32_t c = 0; c < per; c++) {
                const uint32_t at = t * per + c, lap = at / head_slots, r = at - lap * head_slots, ring = base + lap * slots + r;
                const uint32_t use = r < slots ? ring / slots : lap, bar = r < slots ? ring % slots : MAX_SLOTS + r - slots;
                uint32_t n = 0;
                Waiter wait = wt;
#pragma unroll 1
                while (*(volatile uint32_t*)&use_sm[bar] != use + 1 && !wait.give_up(n)) {}
                __syncwarp();
                alive = __all_sync(0xffffffffu, *(volatile uint32_t*)&use_sm[bar] == use + 1 && wait_bar(&full_bar[bar], use & 1u, expiry) && alive) != 0;
                const uint8_t* const wp = (r < slots ? smem + bar * SLOT : extra_sm + (r - slots) * SLOT) + (lane >> 2) * d.pitch + (lane & 3) * 16;
                const uint4* const xp = xs + c * CHUNK * (2 * MT) * 32 + lane;
                const uint32_t ns = d.count(c);
#pragma unroll 4
                for (uint32_t k = 0; k < ns; k++) {
                    const uint4 w = *reinterpret_cast<const uint4*>(wp + k * 64);
#pragma unroll
                    for (uint32_t m = 0; m < MT; m++) {
                        const uint4 x0 = xp[(k * (2 * MT) + 2 * m) * 32], x1 = xp[(k * (2 * MT) + 2 * m + 1) * 32];
                        mma(acc[m], x0.x, x1.x, x0.y, x1.y, w.x, w.y);
                        mma(odd[m], x0.z, x1.z, x0.w, x1.w, w.z, w.w);
                    }
                }
                if (settled(fmaxf(acc[0][0], odd[0][0])) && lane == 0 && alive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&empty_bar[bar])), "r"(NW) : "memory");
            }
#pragma unroll
            for (uint32_t m = 0; m < MT; m++)
#pragma unroll
                for (int k = 0; k < 4; k++) acc[m][k] += odd[m][k];
            // columns 2 (lane % 4), + 1, in ascending order: the first of the largest stays
            const uint32_t c0 = (d.t0 + t) * 8 + (lane & 3) * 2;
#pragma unroll
            for (uint32_t p = 0; p < 2 * MT; p++)
#pragma unroll
                for (uint32_t k = 0; k < 2; k++)
                    if (c0 + k < a.vocab && acc[p >> 1][(p & 1) * 2 + k] > best_v[p]) { best_v[p] = acc[p >> 1][(p & 1) * 2 + k]; best_i[p] = c0 + k; }
        }
        // this SM's best of each row, then over the SMs, row r by SM r; the lowest index wins ties
        auto better = [](float& v, uint32_t& n, float ov, uint32_t on) { if (ov > v || (ov == v && on < n)) { v = ov; n = on; } };
        uint2* const best_sm = reinterpret_cast<uint2*>(at_acc);   // [R][NW]
#pragma unroll
        for (uint32_t p = 0; p < 2 * MT; p++) {
#pragma unroll
            for (int k = 1; k < 4; k <<= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best_v[p], k);
                const uint32_t on = __shfl_xor_sync(0xffffffffu, best_i[p], k);
                better(best_v[p], best_i[p], ov, on);
            }
            if ((lane & 3) == 0) best_sm[(p * 8 + (lane >> 2)) * NW + cw] = make_uint2(__float_as_uint(best_v[p]), best_i[p]);
        }
        bar_sync<NCT>(BAR_HEAD);
        if (ct < R && row_live(ct)) {
            float v = -INFINITY;
            uint32_t n = NO_LOGIT;
#pragma unroll
            for (uint32_t k = 0; k < NW; k++) {
                const uint2 o = best_sm[ct * NW + k];
                better(v, n, __uint_as_float(o.x), o.y);
            }
            xst2(a.xch + fin + (ct * B200_SMS + cta) * 8, word(v), n);
        }
        if (cta < R && row_live(cta) && cw == 0) {
            __syncwarp();
            float v = -INFINITY;
            uint32_t n = NO_LOGIT;
            constexpr uint32_t PER = (B200_SMS + 31) / 32;
            uint2 o[PER];
            uint32_t polls = 0;
            Waiter w = wt;
            bool lack;
#pragma unroll 1
            do {
                lack = false;
#pragma unroll
                for (uint32_t k = 0; k < PER; k++) o[k] = lane + 32 * k < a.sms ? xld2(a.xch + fin + (cta * B200_SMS + lane + 32 * k) * 8) : make_uint2(0xff800000u, NO_LOGIT);
#pragma unroll
                for (uint32_t k = 0; k < PER; k++) lack = lack || o[k].x == EMPTY || o[k].y == EMPTY;
            } while (lack && !w.give_up(polls));
#pragma unroll
            for (uint32_t k = 0; k < PER; k++) better(v, n, __uint_as_float(o[k].x), o[k].y);
            __syncwarp();
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, v, k);
                const uint32_t on = __shfl_xor_sync(0xffffffffu, n, k);
                better(v, n, ov, on);
            }
            bar_sync<64>(BAR_FLAT);
            if (lane == 0) {
                const uint32_t tok = n < a.vocab && !flat_sm ? n : 0u;   // (no logit above -inf, or all 0: 0)
                a.sampled[slot_of(cta)] = tok;
                if (a.sampled_host) a.sampled_host[slot_of(cta)] = tok;
                if (cta == (uint32_t)__ffs(live) - 1) {   // every SM has published its best, so has read them
                    state->set = (e0 + L + 1) % SETS;
                    state->counted += clears_of_step(L) * a.sms;
                }
            }
        }
    }
    if (expiry.is_dead()) {
        // the latest copy into each buffer may not have been waited for (a copy was only requested when the one before was)
        const uint32_t nv = walk_sm[cw].sent, nk = nv + walk_sm[cw].asked;
        if (nk) mbar_wait(&k_bar[cw], (nk - 1) & 1u);
        if (nv) mbar_wait(&v_bar[cw], (nv - 1) & 1u);
        if (lane == 0) report();
    }
}

template <int HD, int MT, bool SPLIT, int PARTS>
int launch_batch_t(cudaStream_t st, const BatchArgs& a, const Plan& p, uint32_t blocks) {
    {
        static bool attr_set[64] = {};
        int dev = 0;
        AK_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lock(device_cache_mutex());
        if (!attr_set[dev & 63]) {
            AK_CUDA(cudaFuncSetAttribute(batch_kernel<HD, MT, SPLIT, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_DYN_SMEM));
            attr_set[dev & 63] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    AK_CUDA(cudaLaunchKernelEx(&cfg, batch_kernel<HD, MT, SPLIT, PARTS>, a, p.slots, p.wpi, 65536 / p.wpi + 1, ahead_of(a.dim, a.ffn, a.heads, a.part_seqs, a.sms, p.slots)));
    AK_COUNT_LAUNCH();
    return AK_OK;
}

}  // namespace

int batch_maps(void* out, const SoloLayer* layers, const void* lm_head, uint32_t n_layers, uint32_t dim, uint32_t ffn, uint32_t vocab) {
    CUtensorMap* m = reinterpret_cast<CUtensorMap*>(out);
    auto put = [&](const void* w, uint32_t rows, uint32_t k) { return make_tmap_rows(m++, w, rows, k, piece_of(k), chunk_cols(k) / piece_of(k), 8); };
    for (uint32_t l = 0; l < n_layers; l++) {
        AK_TRY(put(layers[l].qkv, 3 * dim, dim));
        AK_TRY(put(layers[l].out, dim, dim));
        AK_TRY(put(layers[l].up, ffn, dim));
        AK_TRY(put(layers[l].down, dim, ffn));
    }
    return put(lm_head, vocab, dim);
}

bool batch_supported(uint32_t dtype, uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers, uint32_t seqs, uint32_t max_len) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    return (uint32_t)sms >= B200_SMS && dtype == AK_BF16 && shape_supported(dim, ffn, heads, n_layers, seqs, max_len);
}

size_t batch_sets_bytes(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t seqs, uint32_t max_len) { return sets_bytes(dim, ffn, heads, seqs, max_len); }

int launch_batch(cudaStream_t st, const BatchArgs& a, uint32_t missing) {
    const uint32_t n = parts_of(a.seqs), blocks = n * a.sms - missing;
    const Plan p = make_plan(a.dim, a.n_layers, a.heads, a.part_seqs, a.max_len, a.sms, n);
    const bool two = m_tiles(a.part_seqs) == 2, split = has_splits(a.max_len, a.dim / a.heads), hd64 = a.dim / a.heads == 64;
    if (n == 2) {   // (17 to 32 rows each)
        if (hd64) return split ? launch_batch_t<64, 2, true, 2>(st, a, p, blocks) : launch_batch_t<64, 2, false, 2>(st, a, p, blocks);
        return split ? launch_batch_t<128, 2, true, 2>(st, a, p, blocks) : launch_batch_t<128, 2, false, 2>(st, a, p, blocks);
    }
    if (hd64) {
        if (split) return two ? launch_batch_t<64, 2, true, 1>(st, a, p, blocks) : launch_batch_t<64, 1, true, 1>(st, a, p, blocks);
        return two ? launch_batch_t<64, 2, false, 1>(st, a, p, blocks) : launch_batch_t<64, 1, false, 1>(st, a, p, blocks);
    }
    if (split) return two ? launch_batch_t<128, 2, true, 1>(st, a, p, blocks) : launch_batch_t<128, 1, true, 1>(st, a, p, blocks);
    return two ? launch_batch_t<128, 2, false, 1>(st, a, p, blocks) : launch_batch_t<128, 1, false, 1>(st, a, p, blocks);
}

int batch_status(unsigned int* out) {
    AK_CUDA(cudaMemcpyFromSymbol(out, g_batch_status, sizeof(unsigned int)));
    return AK_OK;
}

}  // namespace ak
