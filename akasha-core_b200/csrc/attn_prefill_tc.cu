// Causal varlen prefill attention on the 5th-generation tensor cores (bf16 K/V/Q, fp32 softmax):
// the same online-softmax recurrence as the reference's FLASH_ATTENTION kernel
// (src/shaders/cuda.rs:633-685), tiled 128 queries x 128 keys.
//
// An item is one or two 128-query tiles of one (sequence, head). The launch has a block per item; the resident blocks (one per
// SM) are persistent and take over blocks that have not started, so the hardware's queue balances ragged prompts. Warps:
//   * warp 0, TMA: the items' Q tiles and a ring of K and V tiles straight from the paged pools (8 blocks of 16 positions
//     per tile, 128-byte swizzle); looks for the next item between tiles.
//   * warp 1 issues the MMAs. S = Q.K^T: A = Q, B = K tile (both K-major, shared memory), fp32 in TMEM.
//     O += P.V: A = P in TENSOR MEMORY (bf16, written over the S it came from), B = the V tile as loaded (MN-major: V rows
//     are keys, the contiguous direction is head_dim), accumulating in TMEM over all key tiles.
//   * two warpgroups per query tile, two threads <-> query row <-> TMEM lane: each reads 64 scores of the row into registers,
//     causal mask on diagonal and tail tiles only, p = 2^(s * scale * log2 e - m) (one FMA and one ex2 per score), writes P
//     back. The row's reference maximum m moves only when a tile exceeds it by 2^8, so O is almost never rescaled.
// With two query tiles the tensor core computes for one while the other is in its softmax. What bounds it: the chain of a tile
// (softmax ~1900 cycles, P.V and the next S ~1400 of which 1024 are MMA time at head_dim 128), two chains in flight: 3400
// cycles for two tiles, against 2048 of MMA and 2048 of the special-function unit. Taking a quarter of the exponentials to the
// FMA pipe (a degree-5 polynomial) was slower, the issue slots are as scarce.
// 16 prompts of 128 to 3072 tokens, 16 heads of 128: 757 us for the version that ran S, softmax and P.V one after the other,
// P through shared memory; 325 us here. 16 prompts of 3072: 640 us (966 TFLOP/s).
// All mbarrier waits are bounded; on expiry a status word is set and the CTA unwinds.
#include "kernels.h"
#include "tma.h"

namespace ak {

__device__ unsigned int g_prefill_tc_status = 0;

namespace pftc {

constexpr int BQ = 128, BS = 16;

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
// the same with A (M x 16 bf16, two per 32-bit column) in tensor memory
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
#define AK_R32(r) "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), \
    "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), AK_R32(r) : "memory");
}
#undef AK_R32
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
          "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ float ex2(float x) {   // 2^x, hardware approximation (2 ulp), ex2(-inf) = 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// K-major operand, 128-byte swizzle, 128-byte rows; 8-row atoms 1024 bytes apart.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// MN-major operand (the contiguous direction is N): rows of the tile are K (keys), 128-byte swizzle;
// atoms of 8 K-rows are 1024 bytes apart (stride offset), the next 64-column slab along N starts
// `lbo` bytes further (leading offset).
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t addr, uint32_t lbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// kind::f16 instruction descriptor: D f32, A/B bf16, A K-major, B K-major (b_mn = 0) or MN-major (1).
__host__ __device__ constexpr uint32_t idesc(uint32_t m, uint32_t n, uint32_t b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// Keys per tile. A tile is the unit of the online softmax; its boundaries are absolute positions, so a row's arithmetic does
// not depend on which rows share its CTA or launch.
constexpr int BKV = 128;

template <int HD, int QT> struct Cfg {
    static constexpr int HALVES = HD / 64;                 // 64-column (128-byte) slabs per row
    static constexpr int Q_BYTES = BQ * HD * 2;            // one query tile: HALVES slabs of [128 x 64]
    static constexpr int KV_BYTES = BKV * HD * 2;          // a K (or V) tile: HALVES slabs of [128 x 64]
    static constexpr int STAGES = HD == 128 ? 2 : 4;       // K / V ring
    static constexpr int SMEM_BYTES = QT * Q_BYTES + STAGES * 2 * KV_BYTES + 1024;
    static constexpr int TMEM_COLS = 512;                  // S tiles (P overwrites its S) at 0 and 128, O tiles from 256 on
    static constexpr int THREADS = 64 + QT * 256;          // warp 0: TMA, warp 1: MMA; then two softmax warpgroups per query tile
};
// A row keeps the maximum its exponents are taken from until a tile exceeds it by more than this (in powers of two): the
// probabilities then stay below 2^8 and the output tile, which accumulates in TMEM, is almost never rescaled. bf16's relative
// rounding is the same at any size, but under a maximum that always follows the largest probability of a tile is 1, without rounding:
// the output's error against f64 is 1.00 to 1.02 times as large for it (2.01e-3 -> 2.04e-3, 16 prompts of 128 to 3072, head_dim 128),
// 1.07 for scores of standard deviation 4. Following always: 330 -> 349 us on those prompts.
constexpr float RESCALE_LOG2 = 8.0f;

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// What the producer tells the other warps about a piece of work: QT query tiles of one (sequence, head).
struct Item {
    uint32_t q0, h, len, pos0, row0, n0, n1;   // n0, n1: key tiles of query tile 0, 1 (n1 == 0 or >= n0)
    uint32_t valid;                            // 0: no more work
};

// The next block of the grid that has not started, taken over by this one (the launch has a block per item: the resident
// blocks run persistently and the hardware's own queue balances them). The answer arrives in shared memory.
__device__ __forceinline__ void clc_request(uint4* answer, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(answer)), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool clc_answer(const uint4* answer, uint32_t& block) {
    uint32_t got, x;
    asm volatile(
        "{\n.reg .b128 h;\n.reg .pred p;\nld.shared.b128 h, [%2];\nclusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n"
        "selp.u32 %0, 1, 0, p;\nmov.u32 %1, 0;\n@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n}\n"
        : "=r"(got), "=r"(x)
        : "r"(smem_u32(answer))
        : "memory");
    block = x;
    return got != 0;
}

template <int HD, int QT>
__global__ void __launch_bounds__(Cfg<HD, QT>::THREADS, 1)
prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const int32_t* __restrict__ block_tables, uint32_t max_blocks,
                  const int32_t* __restrict__ cu, const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ q_pos0,
                  bf16* __restrict__ out, uint32_t row_base, uint32_t heads, uint32_t n_seqs, uint32_t q_items, uint32_t groups_per_chunk, float scale) {
    using C = Cfg<HD, QT>;
    constexpr int ST = C::STAGES;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t q_full[QT], q_empty[QT], k_full[ST], k_empty[ST], v_full[ST], v_empty[ST], s_full[2], p_ready[2], pv_done, o_full[QT], o_empty[QT], item_full[2],
        item_empty[2], clc_bar, drain;
    __shared__ __align__(16) uint4 clc_resp;
    __shared__ Item items[2];
    __shared__ uint32_t tmem_base_sm, fail_flag;
    __shared__ float row_x[QT][2][2][BQ];   // what the two threads of a row tell each other (alternating by tile): maxima, then sums

    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* const q_sm = smem;
    uint8_t* const kv_sm = q_sm + QT * C::Q_BYTES;   // [stage][K | V]

    if (tid == 0) {
        tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
        for (int s = 0; s < ST; s++) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
        for (int t = 0; t < 2; t++) { mbar_init(&s_full[t], 1); mbar_init(&p_ready[t], 8); mbar_init(&item_full[t], 1); mbar_init(&item_empty[t], 1 + QT * 8); }
        for (int t = 0; t < QT; t++) { mbar_init(&q_full[t], 1); mbar_init(&q_empty[t], 1); mbar_init(&o_full[t], 1); mbar_init(&o_empty[t], 8); }
        mbar_init(&pv_done, 1);
        mbar_init(&clc_bar, 1);
        mbar_init(&drain, 1);
        fail_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) { tmem_alloc(&tmem_base_sm, C::TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Invariant of every TMEM-using kernel of this library: dependents are released only AFTER this CTA holds its
    // TMEM columns. A dependent grid's CTAs allocate TMEM and then block in griddepcontrol.wait until this grid
    // has completed; were they let in first, they could take the columns this CTA still needs and both would wait.
    pdl_trigger();
    pdl_wait();
    const uint32_t tmem = tmem_base_sm;
    auto wait = [](uint64_t* bar, uint32_t ph) { return __all_sync(0xffffffffu, mbar_wait(bar, ph)) != 0; };

    if (warp == 0) {
        // ---------------- TMA producer: fetches an item's Q tiles and its K and V tiles, straight from the paged pools, one lane per
        // 16-position block, and finds the next item meanwhile
        const uint32_t groups = heads * n_seqs;
        uint32_t n_items = 0, cnt = 0;             // items published, key tiles fetched before this item
        uint32_t loads = 0, q_loads[2] = {0, 0};   // K and V tiles asked for: 2 (cnt + t) + (0 | 1); Q tiles asked for
        uint32_t asked = 0;                        // questions to the block queue
        bool ok = true, pending = false, found = false, done = false;
        Item nx;                                   // the next item, if found
        const int32_t* nx_table = nullptr;
        int32_t nx_y = 0;
        auto block_row = [&](const Item& it, const int32_t* table, uint32_t t) -> int32_t {   // pool row of this lane's block of tile t
            const uint32_t pos = t * BKV + lane * BS;
            // blocks past the sequence end are fetched from its first block: finite data, masked out below
            return lane < BKV / BS ? (int32_t)(((uint32_t)table[pos < it.pos0 + it.len ? pos / BS : 0] * heads + it.h) * BS) : 0;
        };
        auto publish = [&](const Item& it) {
            const uint32_t slot = n_items & 1u;
            if (n_items >= 2) ok = wait(&item_empty[slot], ((n_items >> 1) & 1u) ^ 1u);
            if (!ok) return;
            if (lane == 0) { items[slot] = it; mbar_arrive(&item_full[slot]); }
            __syncwarp();
            n_items++;
        };
        auto ask = [&]() {
            if (lane == 0) { mbar_expect_tx(&clc_bar, 16); clc_request(&clc_resp, &clc_bar); }
            __syncwarp();
            asked++;
            pending = true;
        };
        // Block w of the launch. In launch order: chunks of (sequence, head) groups whose K and V fit the L2 together; inside a
        // chunk the last query tiles of all its groups come first, they have the most keys.
        auto decode = [&](uint32_t w) {
            const uint32_t chunk = w / (groups_per_chunk * q_items), rem = w - chunk * groups_per_chunk * q_items;
            const uint32_t in_chunk = min(groups_per_chunk, groups - chunk * groups_per_chunk);
            const uint32_t g = chunk * groups_per_chunk + rem % in_chunk, seq = g / heads;
            nx.h = g - seq * heads;
            nx.q0 = (q_items - 1 - rem / in_chunk) * (QT * BQ);
            // len query rows at positions pos0 .. pos0 + len - 1 (pos0 > 0: a later chunk of a prompt whose first pos0
            // positions are already in the cache); keys are positions 0 .. kv_len - 1
            const uint32_t first = (uint32_t)cu[seq];
            nx.len = (uint32_t)cu[seq + 1] - first;
            if (nx.q0 >= nx.len) return;
            nx.pos0 = q_pos0 ? (uint32_t)q_pos0[seq] : 0u;
            nx.row0 = row_base + first;
            // key tiles of a query tile: up to the position of its last row
            nx.n0 = (nx.pos0 + min(nx.q0 + BQ - 1, nx.len - 1)) / BKV + 1;
            nx.n1 = QT == 2 && nx.q0 + BQ < nx.len ? (nx.pos0 + min(nx.q0 + 2 * BQ - 1, nx.len - 1)) / BKV + 1 : 0u;
            nx.valid = 1;
            nx_table = block_tables + (size_t)seq_slot[seq] * max_blocks;
            nx_y = block_row(nx, nx_table, 0);
            found = true;
            publish(nx);
        };
        // one step of the search for the next item
        auto search = [&](bool block) {
            if (!pending) return;
            const bool here = block ? wait(&clc_bar, (asked - 1) & 1u) : __all_sync(0xffffffffu, mbar_try_wait(&clc_bar, (asked - 1) & 1u)) != 0;
            if (!here) { ok = ok && !block; return; }
            pending = false;
            uint32_t w;
            const bool got = clc_answer(&clc_resp, w);
            fence_async_smem();   // read before the next answer is written
            __syncwarp();
            if (!got) { done = true; publish(Item{}); return; }
            decode(w);
            if (!found) ask();
        };
        decode(blockIdx.x);
        if (!found) ask();
        while (ok) {
            while (ok && !found && !done) search(true);
            if (!ok || !found) break;
            const Item it = nx;
            const int32_t* const table = nx_table;
            int32_t y = nx_y;
            found = false;
            ask();
            const uint32_t n_max = max(it.n0, it.n1);
#pragma unroll
            for (uint32_t t = 0; t < QT; t++) {
                if (!ok || (t && !it.n1)) continue;
                if (q_loads[t]) ok = wait(&q_empty[t], (q_loads[t] - 1) & 1u);   // its S of the item before are done
                if (!ok) continue;
                if (lane == 0) {
                    mbar_expect_tx(&q_full[t], C::Q_BYTES);
#pragma unroll
                    for (int hf = 0; hf < C::HALVES; hf++)
                        tma_load_2d(q_sm + t * C::Q_BYTES + hf * (BQ * 128), &tmQ, (int32_t)(it.h * HD + hf * 64), (int32_t)(it.row0 + it.q0 + t * BQ), &q_full[t]);
                }
                q_loads[t]++;
            }
            for (uint32_t t = 0; t < n_max && ok; t++) {
                const uint32_t c = cnt + t, s = c % ST, ph = (c / ST) & 1u;
                uint8_t* const k_dst = kv_sm + (size_t)s * 2 * C::KV_BYTES;
                const int32_t y_next = t + 1 < n_max ? block_row(it, table, t + 1) : 0;
#pragma unroll
                for (int kv = 0; kv < 2; kv++) {
                    uint64_t* const full = kv ? &v_full[s] : &k_full[s];
                    if (c >= (uint32_t)ST) ok = wait(kv ? &v_empty[s] : &k_empty[s], ph ^ 1u);
                    if (!ok) break;
                    if (lane == 0) mbar_expect_tx(full, C::KV_BYTES);
                    __syncwarp();
                    if (lane < BKV / BS)
#pragma unroll
                        for (int hf = 0; hf < C::HALVES; hf++)
                            tma_load_2d(k_dst + kv * C::KV_BYTES + hf * (BKV * 128) + lane * (BS * 128), kv ? &tmV : &tmK, hf * 64, y, full);
                    loads++;
                }
                y = y_next;
                if (ok) search(false);
            }
            cnt += n_max;
        }
        if (!ok && lane == 0) atomicExch(&fail_flag, 1u);
        // whatever happened, every copy asked for lands before the CTA's memory goes away
        if (pending) mbar_wait(&clc_bar, (asked - 1) & 1u);
#pragma unroll
        for (uint32_t t = 0; t < QT; t++)
            if (q_loads[t]) mbar_wait(&q_full[t], (q_loads[t] - 1) & 1u);
        for (uint32_t i = loads > 2u * ST ? loads - 2u * ST : 0; i < loads; i++) {
            const uint32_t j = i >> 1;
            mbar_wait((i & 1u) ? &v_full[j % ST] : &k_full[j % ST], (j / ST) & 1u);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer. The warp stays converged and the operands are warp-uniform, so that the descriptors live in
        // uniform registers: with a single lane in the branch every MMA cost ~100 cycles to issue, more than it takes to run.
        bool ok = true;
        const uint64_t q_desc = desc_kmajor(smem_u32(q_sm)), k_desc = desc_kmajor(smem_u32(kv_sm)),
                       v_desc = desc_mnmajor(smem_u32(kv_sm + C::KV_BYTES), BKV * 128);
        constexpr uint32_t STAGE_STEP = 2 * C::KV_BYTES / 16;   // (descriptor addresses count 16 bytes)
        // S of query tile t against the key tile in stage st, into TMEM buffer b
        auto issue_s = [&](uint32_t t, uint32_t st, uint32_t b) {
            const uint64_t qd = q_desc + t * (C::Q_BYTES / 16), kd = k_desc + st * STAGE_STEP;
#pragma unroll
            for (int kk = 0; kk < HD / 16; kk++)
                tc_mma(tmem + b * BKV, qd + (kk / 4) * (BQ * 128 / 16) + (kk % 4) * 2, kd + (kk / 4) * (BKV * 128 / 16) + (kk % 4) * 2, idesc(BQ, BKV, 0),
                       kk != 0);
            tc_commit(&s_full[b]);
        };
        // O of query tile t (+)= P . V of the key tile in stage st; P (bf16, two per column) lies in TMEM over the S of buffer b, V is
        // the MN-major B operand as loaded
        auto issue_pv = [&](uint32_t t, uint32_t st, uint32_t b, bool add) {
            const uint64_t vd = v_desc + st * STAGE_STEP;
#pragma unroll
            for (int kk = 0; kk < BKV / 16; kk++)
                tc_mma_ts(tmem + 256 + t * HD, tmem + b * BKV + kk * 8, vd + kk * (16 * 128 / 16), idesc(BQ, HD, 1), (add || kk != 0) ? 1u : 0u);
        };
        uint32_t cnt = 0, cp[2] = {0, 0}, ci[2] = {0, 0};   // key tiles before the item; P tiles and items of each query tile
        uint32_t n0 = 0, n1 = 0, k = 0;                     // the item's key tiles; items begun
        // the next item: its first S of query tile 0 (key tile number `first`). The S and P buffers need no wait: the P.V that
        // read them last was issued before, and MMAs run in order.
        uint32_t next0 = 0, next1 = 0, next_valid = 0;
        auto begin = [&](uint32_t first) {
            ok = wait(&item_full[k & 1u], (k >> 1) & 1u);
            if (!ok) return;
            next0 = items[k & 1u].n0; next1 = items[k & 1u].n1; next_valid = items[k & 1u].valid;
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_empty[k & 1u]);
            k++;
            if (!next_valid) return;
            ok = wait(&q_full[0], (k - 1) & 1u) && wait(&k_full[first % ST], (first / ST) & 1u);
            tc_fence_after();
            if (ok && elect_one()) {
                issue_s(0, first % ST, QT == 1 ? (cp[0] ^ (k > 1)) & 1u : 0u);
                if (QT == 1) tc_commit(&k_empty[first % ST]);
                if (next0 == 1) tc_commit(&q_empty[0]);
            }
            __syncwarp();
        };
        begin(0);
        while (ok && next_valid) {
            n0 = next0; n1 = next1;
            const uint32_t n_max = max(n0, n1);
            bool begun = false;   // the item after this one
            if (QT == 2) {
                if (n1) ok = wait(&q_full[QT - 1], ci[1] & 1u);
                tc_fence_after();
                if (ok && elect_one()) {
                    if (n1) {
                        issue_s(1, cnt % ST, 1);
                        if (n1 == 1) tc_commit(&q_empty[QT - 1]);
                    }
                    tc_commit(&k_empty[cnt % ST]);
                }
                __syncwarp();
            }
            for (uint32_t j = 0; j < n_max && ok; j++) {
                const uint32_t c = cnt + j, s = c % ST, s1 = (c + 1) % ST;
                const bool more = j + 1 < n_max;
                if (more) ok = wait(&k_full[s1], ((c + 1) / ST) & 1u);
                if (!ok) break;
                if (QT == 1) {
                    // S alternates between two buffers: the S of the next tile is computed while this one is in its softmax
                    const uint32_t b = cp[0] & 1u;
                    tc_fence_after();
                    if (more && elect_one()) {
                        issue_s(0, s1, b ^ 1u);
                        tc_commit(&k_empty[s1]);
                        if (j + 2 == n_max) tc_commit(&q_empty[0]);
                    }
                    __syncwarp();
                    if (!more) { begin(cnt + n_max); begun = true; }
                    ok = ok && wait(&v_full[s], (c / ST) & 1u) && wait(&p_ready[b], (cp[0] >> 1) & 1u);
                    if (ok && j == 0 && ci[0]) ok = wait(&o_empty[0], (ci[0] - 1) & 1u);   // the output before has been read
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        issue_pv(0, s, b, j != 0);
                        tc_commit(&v_empty[s]);
                        tc_commit(&pv_done);
                        if (!more) tc_commit(&o_full[0]);
                    }
                    __syncwarp();
                    cp[0]++;
                } else {
                    // two query tiles take turns: one is in its softmax while the tensor core works for the other
                    ok = wait(&v_full[s], (c / ST) & 1u);
#pragma unroll
                    for (uint32_t t = 0; t < 2; t++) {
                        const uint32_t nt = t ? n1 : n0;
                        if (!ok) continue;
                        if (j >= nt) {   // tile 0 has one key tile less: it starts on the next item while tile 1 has its last one
                            if (t == 0) { begin(cnt + n_max); begun = true; }
                            continue;
                        }
                        ok = wait(&p_ready[t], cp[t] & 1u);
                        if (ok && j == 0 && ci[t]) ok = wait(&o_empty[t], (ci[t] - 1) & 1u);
                        if (!ok) continue;
                        tc_fence_after();
                        if (elect_one()) {
                            issue_pv(t, s, t, j != 0);
                            if (j + 1 < nt) {
                                issue_s(t, s1, t);
                                if (j + 2 == nt) tc_commit(&q_empty[t]);
                            } else {
                                tc_commit(&o_full[t]);
                            }
                        }
                        __syncwarp();
                        cp[t]++;
                    }
                    if (!ok) break;
                    if (elect_one()) {
                        tc_commit(&v_empty[s]);
                        if (more) tc_commit(&k_empty[s1]);
                    }
                    __syncwarp();
                }
            }
            cnt += n_max;
            ci[0]++;
            if (n1) ci[1]++;
            if (ok && !begun) begin(cnt);
        }
        // every MMA issued ends before the CTA's memory goes away
        if (elect_one()) {
            if (!ok) atomicExch(&fail_flag, 2u);
            tc_commit(&drain);
        }
        __syncwarp();
        mbar_wait(&drain, 0);
    } else {
        // ---------------- two softmax warpgroups per query tile: a row (a TMEM lane) belongs to two threads, one per 64 keys of a
        // tile. (One thread per row left two warps per scheduler: the tile's serial chain, not a pipe, set the time.)
        const uint32_t qt = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1u, r = (warp & 3u) * 32 + lane;
        const uint32_t lane_addr = ((warp & 3u) * 32u) << 16;
        const float sl2 = scale * 1.4426950408889634f;           // base 2: p = 2^(s * scale * log2 e - m)
        constexpr int HK = BKV / 2, HO = HD / 2;                 // this thread's keys of a tile, and its columns of the output
        auto tile_sync = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + qt) : "memory"); };   // the 256 threads of the tile
        auto tile_all = [&](bool v) -> bool {                    // the same with a vote
            uint32_t r;
            asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.and.pred q, %2, 256, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                         : "=r"(r) : "r"((uint32_t)v), "r"(1 + qt) : "memory");
            return r != 0;
        };
        uint32_t cnt = 0, cs = 0, ci = 0, rx = 0;   // key tiles of all items before; S tiles and items of this query tile; uses of row_x
        bool ok = true;
        for (uint32_t k = 0;; k++) {
            // A warp whose wait ran out goes on without waiting, so that the tile's barriers stay whole; the tile's warps leave
            // together, here.
            if (ok) ok = wait(&item_full[k & 1u], (k >> 1) & 1u);
            if (!tile_all(ok)) break;
            const Item it = items[k & 1u];
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_empty[k & 1u]);
            if (!it.valid) break;
            const uint32_t n = qt ? it.n1 : it.n0, qf = it.q0 + qt * BQ, kv_len = it.pos0 + it.len;   // qf: first query row of the tile
            const uint32_t qi = it.pos0 + qf + r;                                                     // this thread's query position
            float m_ref = 0.0f, l_run = 0.0f;
            for (uint32_t j = 0; j < n; j++, cs++) {
                const uint32_t b = QT == 1 ? (cs & 1u) : qt, ph = QT == 1 ? (cs >> 1) & 1u : cs & 1u;
                const uint32_t s_addr = tmem + b * BKV + lane_addr;
                if (ok) ok = wait(&s_full[b], ph);
                tc_fence_after();
                const uint32_t k0 = j * BKV, kh = k0 + half * HK;
                float s[HK];
#pragma unroll
                for (int c = 0; c < HK; c += 32) tmem_ld32(s_addr + half * HK + c, reinterpret_cast<uint32_t*>(s) + c);
                tmem_ld_wait();
                // Keys this thread's row sees, of its 64; only the warps whose rows do not all see all of them need the mask (the
                // diagonal and the end of the sequence).
                const uint32_t vis = min(qi + 1, kv_len);   // keys 0 .. vis - 1
                if (kh + HK > min(it.pos0 + qf + (warp & 3u) * 32 + 1, kv_len)) {
                    const uint32_t seen = vis > kh ? vis - kh : 0u;
#pragma unroll
                    for (int c = 0; c < HK; c += 32) {
                        const uint32_t bits = seen >= c + 32u ? 0xffffffffu : seen > (uint32_t)c ? (1u << (seen - c)) - 1u : 0u;
#pragma unroll
                        for (int i = 0; i < 32; i++)
                            if (!(bits & (1u << i))) s[c + i] = -INFINITY;
                    }
                }
                float mx0 = s[0], mx1 = s[1], mx2 = s[2], mx3 = s[3];
#pragma unroll
                for (int i = 4; i + 8 <= HK; i += 8) {
                    mx0 = fmaxf(fmaxf(mx0, s[i]), s[i + 1]); mx1 = fmaxf(fmaxf(mx1, s[i + 2]), s[i + 3]);
                    mx2 = fmaxf(fmaxf(mx2, s[i + 4]), s[i + 5]); mx3 = fmaxf(fmaxf(mx3, s[i + 6]), s[i + 7]);
                }
#pragma unroll
                for (int i = HK - 4; i < HK; i++) mx0 = fmaxf(mx0, s[i]);
                const float m_h = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
                row_x[qt][rx & 1u][half][r] = m_h;
                tc_fence_before();
                tile_sync();   // (after it nobody reads this tile's S: P may overwrite it)
                tc_fence_after();
                const float m_t = fmaxf(m_h, row_x[qt][rx & 1u][half ^ 1u][r]) * sl2;   // (scale > 0)
                rx++;
                if (j == 0) {
                    m_ref = m_t;   // every row sees position 0
                } else {
                    const bool grow = m_t > m_ref + RESCALE_LOG2;
                    if (__any_sync(0xffffffffu, grow)) {
                        // rare: bring this row's output and sum to the new maximum (factor 1 for the rows that keep theirs)
                        const float f = grow ? ex2(m_ref - m_t) : 1.0f;
                        if (grow) m_ref = m_t;
                        l_run *= f;
                        if (QT == 1) {   // (with two query tiles this tile's S was issued behind the P.V of the last one)
                            if (ok) ok = wait(&pv_done, (cs - 1) & 1u);
                            tc_fence_after();
                        }
                        const uint32_t o_addr = tmem + 256 + qt * HD + half * HO + lane_addr;
#pragma unroll 1
                        for (int c = 0; c < HO; c += 16) {
                            uint32_t o[16];
                            tmem_ld16(o_addr + c, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                            tmem_st16(o_addr + c, o);
                        }
                    }
                }
                // P = 2^(s * sl2 - m_ref) in bf16 over the S just read; the running sum adds the ROUNDED probabilities, the ones
                // the tensor core multiplies
                uint64_t rs = 0;
                const uint64_t nm = pack2(-m_ref, -m_ref), sc = pack2(sl2, sl2);
#pragma unroll
                for (int c = 0; c < HK; c += 32) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const uint64_t x = fma2(pack2(s[c + i], s[c + i + 1]), sc, nm);
                        float p0, p1;
                        unpack2(x, p0, p1);
                        p0 = ex2(p0);
                        p1 = ex2(p1);
                        const bf162 v2 = __floats2bfloat162_rn(p0, p1);
                        const uint32_t u = *reinterpret_cast<const uint32_t*>(&v2);
                        rs = add2(rs, pack2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)));
                        pk[i / 2] = u;
                    }
                    tmem_st16(s_addr + (half * HK + c) / 2, pk);
                }
                float rs0, rs1;
                unpack2(rs, rs0, rs1);
                l_run += rs0 + rs1;
                if (k0 + BKV > kv_len) {
                    // Tile rows past the sequence end hold whatever the pool held (possibly non-finite): their probabilities
                    // are 0, but 0 * NaN would poison P.V, so clear those V rows (whole 128-byte rows, the swizzle permutes
                    // within a row only).
                    const uint32_t st = (cnt + j) % ST;
                    if (ok) ok = wait(&v_full[st], ((cnt + j) / ST) & 1u);
                    uint8_t* const v_sm = kv_sm + (size_t)st * 2 * C::KV_BYTES + C::KV_BYTES;
                    const uint32_t first = kv_len - k0, chunks = (BKV - first) * 8;
                    for (int hf = 0; hf < C::HALVES; hf++)
                        for (uint32_t i = half * 128 + r; i < chunks; i += 256)
                            *reinterpret_cast<uint4*>(v_sm + hf * (BKV * 128) + (first + i / 8) * 128 + (i % 8) * 16) = make_uint4(0, 0, 0, 0);
                    fence_async_smem();
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[b]);
            }
            cnt += max(it.n0, it.n1);
            if (n == 0) continue;
            if (ok) ok = wait(&o_full[qt], ci & 1u);
            ci++;
            tc_fence_after();
            row_x[qt][rx & 1u][half][r] = l_run;
            uint32_t o[HO];
#pragma unroll
            for (int c = 0; c < HO; c += 32) tmem_ld32(tmem + 256 + qt * HD + half * HO + lane_addr + c, o + c);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_empty[qt]);
            tile_sync();
            const float inv = 1.0f / (row_x[qt][rx & 1u][0][r] + row_x[qt][rx & 1u][1][r]);
            // A lane holds HO columns of one row, NP 16-byte pieces. Exchanged among NP lanes (a butterfly), a store of the warp covers
            // 32 / NP rows whole instead of 16 bytes of 32 rows, which went out one row per cycle.
            constexpr int NP = HO / 8;
            uint32_t pk[NP][4];
#pragma unroll
            for (int d = 0; d < HO; d += 2) {
                const bf162 v2 = __floats2bfloat162_rn(__uint_as_float(o[d]) * inv, __uint_as_float(o[d + 1]) * inv);
                pk[d / 8][(d % 8) / 2] = *reinterpret_cast<const uint32_t*>(&v2);
            }
#pragma unroll
            for (int x = 1; x < NP; x *= 2)
#pragma unroll
                for (int a = 0; a < NP; a++)
                    if (!(a & x))
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const uint32_t give = (lane & x) ? pk[a][e] : pk[a | x][e], got = __shfl_xor_sync(0xffffffffu, give, x);
                            if (lane & x) pk[a][e] = got; else pk[a | x][e] = got;
                        }
            const uint32_t lane0 = lane & ~(uint32_t)(NP - 1), piece = lane & (NP - 1);   // pk[a]: this lane's piece of the row of lane0 + a
            const uint32_t rw = qf + (warp & 3u) * 32 + lane0;
            bf16* const dst = out + (size_t)(it.row0 + rw) * (heads * HD) + (size_t)it.h * HD + half * HO + piece * 8;
#pragma unroll
            for (int a = 0; a < NP; a++)
                if (ok && rw + a < it.len) *reinterpret_cast<uint4*>(dst + (size_t)a * (heads * HD)) = make_uint4(pk[a][0], pk[a][1], pk[a][2], pk[a][3]);
            rx++;   // (it alternates: a warp may be in the next item's first tile while another still reads these sums)
        }
        if (!ok && lane == 0) atomicExch(&fail_flag, 3u);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && fail_flag) atomicExch(&g_prefill_tc_status, fail_flag);
    if (warp == 1) {
        __syncwarp();
        tmem_dealloc(tmem, C::TMEM_COLS);
    }
}

template <int HD, int QT>
static int launch(cudaStream_t st, const void* q, uint64_t q_rows, const void* k_pool, const void* v_pool, uint64_t pool_rows,
                  const int32_t* bt, uint32_t max_blocks, const int32_t* cu, const int32_t* seq_slot, const int32_t* pos0, void* out, uint32_t n_seqs,
                  uint32_t max_len, uint32_t row_base, uint32_t heads, float scale) {
    using C = Cfg<HD, QT>;
    CUtensorMap tmQ, tmK, tmV;
    const uint64_t dim = (uint64_t)heads * HD;
    AK_TRY(make_tmap_2d(&tmQ, q, 2, dim, q_rows, dim * 2, 64, BQ, TMA_SWIZZLE_128B));
    AK_TRY(make_tmap_2d(&tmK, k_pool, 2, HD, pool_rows, (uint64_t)HD * 2, 64, BS, TMA_SWIZZLE_128B));
    AK_TRY(make_tmap_2d(&tmV, v_pool, 2, HD, pool_rows, (uint64_t)HD * 2, 64, BS, TMA_SWIZZLE_128B));
    {
        static bool attr_set[64] = {};
        int dev = 0;
        AK_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lock(device_cache_mutex());
        if (!attr_set[dev & 63]) {
            AK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<HD, QT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
            attr_set[dev & 63] = true;
        }
    }
    // K and V of the (sequence, head) groups of a chunk stay within half of the L2, so that their query tiles read them from there
    const uint32_t q_items = cdiv(max_len, QT * BQ), groups = heads * n_seqs;
    uint32_t per_chunk = (uint32_t)((64u << 20) / ((uint64_t)max_len * HD * 4));
    if (per_chunk < 1) per_chunk = 1;
    if (per_chunk > groups) per_chunk = groups;
    return launch_k(prefill_tc_kernel<HD, QT>, dim3(groups * q_items), dim3(C::THREADS), C::SMEM_BYTES, st, NO_CLUSTER, tmQ, tmK, tmV, bt, max_blocks, cu,
                    seq_slot, pos0, (bf16*)out, row_base, heads, n_seqs, q_items, per_chunk, scale);
}

}  // namespace pftc

int launch_attn_prefill_tc(cudaStream_t st, const void* q, uint64_t q_rows, const void* k_pool, const void* v_pool,
                           uint64_t pool_blocks, const int32_t* block_tables, uint32_t max_blocks_per_seq, const int32_t* cu,
                           const int32_t* seq_slot, const int32_t* pos0, void* out, uint32_t n_seqs, uint32_t max_len, uint32_t row_base, uint32_t heads,
                           uint32_t head_dim, float scale) {
    if (n_seqs == 0 || max_len == 0) return AK_OK;
    const uint64_t pool_rows = pool_blocks * heads * pftc::BS;
    // Two query tiles per CTA keep the tensor core busy through the softmax, one makes twice as many CTAs: below a wave of
    // pairs (a prompt or two joining a decode batch) the grid is what counts. The same arithmetic per row either way.
    const bool two = (uint64_t)cdiv(max_len, 2 * pftc::BQ) * heads * n_seqs >= B200_SMS;
#define AK_PF_ARGS st, q, q_rows, k_pool, v_pool, pool_rows, block_tables, max_blocks_per_seq, cu, seq_slot, pos0, out, n_seqs, max_len, row_base, heads, scale
    if (head_dim == 64) return two ? pftc::launch<64, 2>(AK_PF_ARGS) : pftc::launch<64, 1>(AK_PF_ARGS);
    AK_REQUIRE(head_dim == 128, AK_ERR_UNSUPPORTED, "prefill attention (tensor cores): head_dim must be 64 or 128");
    return two ? pftc::launch<128, 2>(AK_PF_ARGS) : pftc::launch<128, 1>(AK_PF_ARGS);
#undef AK_PF_ARGS
}

int prefill_tc_status(unsigned int* out) {
    AK_CUDA(cudaMemcpyFromSymbol(out, g_prefill_tc_status, sizeof(unsigned int)));
    return AK_OK;
}

}  // namespace ak
