// f32 product on the tensor cores: C[m,n] (op)= A[m,k] @ Wt[n,k]^T, f32 operands, f32-accurate sums.
//
// Every operand is split, on its way into shared memory, into three bf16 pieces x = x0 + x1 + x2 (each the rounding of what is left: 3 x 8 bits hold
// the 24 of an f32 exactly, unless it is so small that the third piece falls below bf16's smallest numbers: x is off by 2^-134 at most, 1e-7 of it at 2^-111,
// 1e-4 at 2^-121), and six of the nine products are taken: x0 y0, and x0 y1 + x1 y0 + x1 y1 + x0 y2 + x2 y0. What is left out, x1 y2 + x2 y1 + x2 y2, is
// at most about 2^-24 of a product and of either sign. The large products and the others have accumulators of their own in tensor memory. The tensor core's
// additions cut instead of rounding, so the large products' accumulator is fresh for every K block of 64 (4 MMAs) and is added in registers
// with ordinary f32 additions; the others', at most 2^-7 of it, runs through a segment.
//
// What bounded the FMA kernel it replaces is the FMA pipe and the shared-memory words that feed it (a 512-token prefill of the 162M model ran at 40 % of
// 74 TFLOP/s). Here a K block of a 128 x 128 tile takes 1.9 us: 24 MMAs of 64 cycles (1536), and about 3300 cycles of shared memory, which both operands
// go through as f32, as pieces, and as what the MMAs read; the split and the additions have warps of their own and as many issue slots as the MMAs have
// cycles. A 128 x 64 tile asks for half as much again per product and ran at 0.6 of the rate. A launch costs about 7 us beside its blocks (its
// shared memory leaves the next one no room to start early). m x n x k 512 x 2304 x 768: 52 -> 20 us, 512 x 768 x 3072 60 -> 26, 64 x 3072 x 768 17.7 ->
// 11.4, 64 x 768 x 768 9.6 -> 10.8; 512-token prompts of small models see launch_gemm_f32_nt(). It spills 64 bytes, behind its loops. Error against 64 bits (2-norm), normal operands, at k = 768 1.85e-7 -> 0.88e-7, 3072 3.6e-7 -> 1.0e-7. With operands
// all of one sign, whose sums rounding hardly touches, cutting shows: k = 320 0.66e-7 -> 0.84e-7, 768 0.73e-7 -> 0.85e-7, 3072 1.17e-7 -> 0.86e-7.
//
// The order of a row's sum is a function of (n, k) alone: K is cut into segments of `per` blocks; a segment's blocks are added in order, h segments make
// a group, of which there are two, and the groups are added. Who does it depends on m: one CTA (many rows), a cluster of two CTAs with a group each,
// or of a CTA for each segment (few rows); the partial tiles are read through distributed shared memory.
//
// A result that is not finite (infinite or NaN operands and those that round to an infinite piece, or sums past the largest f32) is computed again with FMAs,
// by a warp for each (a thread for each before): 512 x 768 x 3072, 26 us, with a NaN in one column of the weights 710 -> 53 us, in one row of the activations
// 1160 -> 32, everywhere 6340 -> 52; with an infinity in one row 1160 -> 370, in every row 6340 -> 1480.
#include "kernels.h"
#include "tcgen05.cuh"
#include "tma.h"

#include <type_traits>

namespace ak {

__device__ unsigned int g_gemm_f32_status = 0;

namespace {

constexpr uint32_t TM = 128, TN = 128, TK = 64;
constexpr uint32_t HALF = 32;                             // K columns of a staged tile (one 128-byte row), and of what is split and multiplied at a time
constexpr uint32_t STG = 128 * HALF * 4, STAGE = 2 * STG, STAGES = 4;   // f32: A, B
constexpr uint32_t PL = 128 * TK * 2, OPS = 6 * PL;       // the bf16 pieces of a K block: three tiles of A, three of B, both halves side by side
constexpr uint32_t SMEM = 1024 + STAGES * STAGE + OPS;
constexpr uint32_t ACC_LOW = 2 * TN, ACC_TOT = 3 * TN, TMEM_COLS = 4 * TN;   // columns: large products (two buffers), the others, sum of the groups
constexpr uint32_t NCW = 8, NPW = 8;                      // warps that split, warps that add
constexpr uint32_t THREADS = 128 + 32 * (NCW + NPW);
constexpr int REGS_FIRST = 64, REGS_SPLIT = 64, REGS_ADD = 144;   // of 640 x 96 at launch
static_assert(REGS_FIRST * 128 + REGS_SPLIT * 32 * NCW + REGS_ADD * 32 * NPW <= THREADS * 96, "the split draws on the registers of the launch");
constexpr uint32_t MAX_SEGS = 6;

// the pair (x, y) as three bf16 pairs
__device__ __forceinline__ void split2(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    uint64_t v, minus;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    asm("mov.b64 %0, {%1, %1};" : "=l"(minus) : "f"(-1.0f));
    auto cut = [&]() {   // the rounding of v; v becomes the (exact) rest
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        const bf162 r = __floats2bfloat162_rn(a, b);
        const uint32_t u = *reinterpret_cast<const uint32_t*>(&r);
        uint64_t e;
        asm("mov.b64 %0, {%1, %2};" : "=l"(e) : "r"(u << 16), "r"(u & 0xffff0000u));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(e), "l"(minus));
        return u;
    };
    p0 = cut();
    p1 = cut();
    p2 = cut();
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "f"(v[0]), "f"(v[1]),
        "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
        : "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// A warp's row of A times the columns of W that are marked in its lanes (col .. col + 3, a bit each), with FMAs and all lanes on one lane's columns at a
// time. Once a lane's sum is NaN, so is the whole; a row with a NaN has no other results. x: the columns' results as they are.
__device__ __forceinline__ float4 again(const float* ar, const float* w, uint32_t k, uint32_t col, uint32_t bad, float4 x) {
    const uint32_t lane = threadIdx.x & 31;
    auto rounds = [&](auto f) {   // f(z): of this lane's four values of k from z on, whether they settle the matter
        for (uint32_t z0 = 0; z0 < k; z0 += 512) {
            bool done = false;
#pragma unroll
            for (uint32_t z = z0 + lane * 4, i = 0; i < 4; i++, z += 128)
                if (z < k) done = f(z) || done;
            if (__any_sync(0xffffffffu, done)) return true;
        }
        return false;
    };
    const bool none = rounds([&](uint32_t z) {
        const float4 v = *reinterpret_cast<const float4*>(ar + z);
        return isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w);
    });
    for (uint32_t lanes = __ballot_sync(0xffffffffu, bad); lanes; lanes &= lanes - 1) {
        const uint32_t l = __ffs(lanes) - 1, bits = __shfl_sync(0xffffffffu, bad, l);
        const float* const wr = w + (size_t)__shfl_sync(0xffffffffu, col, l) * k;
        float s[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) s[i] = none || !(bits >> i & 1u) ? NAN : 0.0f;
        if (!none)
            rounds([&](uint32_t z) {
                const float4 u = *reinterpret_cast<const float4*>(ar + z);
#pragma unroll
                for (uint32_t i = 0; i < 4; i++)
                    if (bits >> i & 1u) {
                        const float4 v = *reinterpret_cast<const float4*>(wr + (size_t)i * k + z);
                        s[i] = fmaf(u.w, v.w, fmaf(u.z, v.z, fmaf(u.y, v.y, fmaf(u.x, v.x, s[i]))));
                    }
                return isnan(s[0]) && isnan(s[1]) && isnan(s[2]) && isnan(s[3]);
            });
#pragma unroll
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; i++) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
        if (lane == l) {
            if (bits & 1u) x.x = s[0];
            if (bits & 2u) x.y = s[1];
            if (bits & 4u) x.z = s[2];
            if (bits & 8u) x.w = s[3];
        }
    }
    return x;
}

struct Cut {
    uint32_t per, h, segs;   // K blocks of a segment, segments of a group, segments
};

__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const float* a, const float* w, float* c, uint32_t m,
                   uint32_t n, uint32_t k, uint32_t flags, const Cut cut, uint32_t a_box) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t stg_full[STAGES], stg_empty[STAGES], op_full[2], op_empty[2], acc_full[2], acc_empty[2], low_empty;   // op: by half
    __shared__ uint32_t tmem_base_sm, fail_flag;
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* const stg = smem + OPS;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const uint32_t cs = gridDim.z, rank = blockIdx.z;   // CTAs of the cluster: 1, groups or segments
    const uint32_t kb_total = (k + TK - 1) / TK, mine = (cs == 1 ? cut.segs : cs == cut.segs ? 1 : cut.h) * cut.per;
    const uint32_t kb0 = min(rank * mine, kb_total), nkb = min(kb0 + mine, kb_total) - kb0;

    const uint32_t halves = 2 * nkb, pre = min(halves, STAGES), tx = (a_box * HALF + TN * HALF) * 4;
    auto load_a = [&](uint32_t s, uint32_t j) { tma_load_2d(stg + s * STAGE, &tmA, (int32_t)((2 * kb0 + j) * HALF), (int32_t)m0, &stg_full[s]); };
    auto load_b = [&](uint32_t s, uint32_t j) { tma_load_2d(stg + s * STAGE + STG, &tmB, (int32_t)((2 * kb0 + j) * HALF), (int32_t)n0, &stg_full[s]); };

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < STAGES; s++) { mbar_init(&stg_full[s], 1); mbar_init(&stg_empty[s], NCW); }
        for (uint32_t b = 0; b < 2; b++) {
            mbar_init(&op_full[b], NCW);
            mbar_init(&op_empty[b], 1);
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], NPW);
        }
        mbar_init(&low_empty, NPW);
        fail_flag = 0;
        mbar_fence_init();
        for (uint32_t j = 0; j < pre; j++) {   // (the weights do not depend on the preceding kernel)
            mbar_expect_tx(&stg_full[j], tx);
            load_b(j, j);
        }
        tma_prefetch_desc(&tmA);
    }
    if (warp == 2) {
        tmem_alloc(&tmem_base_sm, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sm;
    pdl_trigger();

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_FIRST));
        if (warp == 0 && lane == 0) {
            // ---------------- producer: half K blocks of both operands as f32
            pdl_wait();
            for (uint32_t j = 0; j < pre; j++) load_a(j, j);
            uint32_t s = 0, ph = 1, j = pre;
            for (; j < halves; j++) {
                if (!mbar_wait(&stg_empty[s], ph ^ 1u)) { atomicExch(&fail_flag, 1u); break; }
                mbar_expect_tx(&stg_full[s], tx);
                load_a(s, j);
                load_b(s, j);
                if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
            // every copy has landed before this CTA's memory goes away: the last use of each stage
            for (uint32_t x = j > STAGES ? j - STAGES : 0; x < j; x++) mbar_wait(&stg_full[x % STAGES], x / STAGES & 1u);
        } else if (warp == 1) {
            // ---------------- MMA issuer (a converged warp, see the bf16 kernel)
            constexpr uint32_t idesc = make_idesc(TM, TN);
            const uint64_t da = make_smem_desc(smem_u32(smem)), db = da + (3 * PL >> 4);
            constexpr uint32_t P = PL >> 4;
            uint32_t in_seg = 0, segs = 0;
            for (uint32_t j = 0; j < 2 * nkb; j++) {
                const uint32_t i = j >> 1, half = j & 1u, b = i & 1u;
                bool got = mbar_wait(&op_full[half], i & 1u);
                if (!half) {
                    got = mbar_wait(&acc_empty[b], (i >> 1 & 1u) ^ 1u) && got;
                    if (in_seg == 0 && segs) got = mbar_wait(&low_empty, (segs - 1) & 1u) && got;
                }
                if (!__all_sync(0xffffffffu, got)) { if (lane == 0) atomicExch(&fail_flag, 2u); break; }
                tc_fence_after();
                const uint32_t acc = tmem + b * TN, low = tmem + ACC_LOW, on = half * 4;   // a half: 32 bf16 = 64 bytes inside the swizzle row
                if (elect_one()) {
#pragma unroll
                    for (uint32_t kk = 0; kk < HALF / 16; kk++) {
                        const uint64_t a0 = da + on + kk * 2, b0 = db + on + kk * 2;
                        const uint32_t more = half || kk;
                        tc_mma_f16(acc, a0, b0, idesc, more);
                        tc_mma_f16(low, a0, b0 + P, idesc, more || in_seg);
                        tc_mma_f16(low, a0 + P, b0, idesc, 1u);
                        tc_mma_f16(low, a0 + P, b0 + P, idesc, 1u);
                        tc_mma_f16(low, a0, b0 + 2 * P, idesc, 1u);
                        tc_mma_f16(low, a0 + 2 * P, b0, idesc, 1u);
                    }
                    tc_commit(&op_empty[half]);
                    if (half) tc_commit(&acc_full[b]);
                }
                __syncwarp();
                if (half && ++in_seg == cut.per) { in_seg = 0; segs++; }
            }
        }
    } else if (warp < 4 + NCW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_SPLIT));
        // ---------------- split: a thread takes 8 columns of a row at a time. The eight lanes of a shared-memory phase are at four pieces of rows r and
        // r + 4: the f32 loads (halves in turn) and the stores into the swizzled bf16 tiles are free of bank conflicts.
        const uint32_t cw = warp - 4, q = lane & 3, hs = lane >> 2 & 1, r8 = hs * 4 + (lane >> 3);
        uint32_t s = 0, sph = 0;
        for (uint32_t j = 0; j < 2 * nkb; j++) {
            const uint32_t half = j & 1u;
            bool got = mbar_wait(&stg_full[s], sph);
            got = mbar_wait(&op_empty[half], (j >> 1 & 1u) ^ 1u) && got;
            if (!__all_sync(0xffffffffu, got)) { if (lane == 0) atomicExch(&fail_flag, 4u); break; }
            __syncwarp();
            auto piece = [&](const uint8_t* src, uint8_t* dst, uint32_t row) {
                const uint8_t* const p = src + row * 128 + q * 32;
                const float4 u = *reinterpret_cast<const float4*>(p + hs * 16), v = *reinterpret_cast<const float4*>(p + (hs ^ 1u) * 16);
                const float4 lo = hs ? v : u, hi = hs ? u : v;
                uint4 o[3];
                split2(lo.x, lo.y, o[0].x, o[1].x, o[2].x);
                split2(lo.z, lo.w, o[0].y, o[1].y, o[2].y);
                split2(hi.x, hi.y, o[0].z, o[1].z, o[2].z);
                split2(hi.z, hi.w, o[0].w, o[1].w, o[2].w);
                uint8_t* const d = dst + row * 128 + (((half * 4 + q) ^ (row & 7)) << 4);
#pragma unroll
                for (int e = 0; e < 3; e++) *reinterpret_cast<uint4*>(d + e * PL) = o[e];
            };
            const uint8_t* const st = stg + s * STAGE;
#pragma unroll
            for (uint32_t i = 0; i < 2; i++) piece(st + STG, smem + 3 * PL, (cw + NCW * i) * 8 + r8);
#pragma unroll
            for (uint32_t i = 0; i < 2; i++)
                if ((cw + NCW * i) * 8 < a_box) piece(st, smem, (cw + NCW * i) * 8 + r8);
            tma_store_fence();   // (generic writes before the tensor core's reads)
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&stg_empty[s]);
                mbar_arrive(&op_full[half]);
            }
            if (++s == STAGES) { s = 0; sph ^= 1u; }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_ADD));
        // ---------------- add: a thread has 64 columns of a row
        constexpr uint32_t CW = TN / 2;
        const uint32_t pw = warp - 4 - NCW, col = (pw >> 2) * CW;
        const uint32_t taddr = tmem + (((warp & 3u) * 32) << 16) + col;
        const uint32_t h = cs == cut.segs ? 1u : cut.h;
        float seg[CW], grp[CW];
#pragma unroll
        for (uint32_t e = 0; e < CW; e++) seg[e] = grp[e] = 0.0f;
        uint32_t in_seg = 0, in_grp = 0, grps = 0;
        auto add16 = [&](uint32_t at, float* to) {
            uint32_t v[16];
            tmem_ld16(at, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; e++) to[e] += __uint_as_float(v[e]);
        };
        for (uint32_t i = 0; i < nkb; i++) {
            const uint32_t b = i & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[b], i >> 1 & 1u))) { if (lane == 0) atomicExch(&fail_flag, 8u); break; }
            tc_fence_after();
            const bool seg_end = ++in_seg == cut.per || i + 1 == nkb;
#pragma unroll
            for (uint32_t x = 0; x < CW; x += 16) add16(taddr + b * TN + x, seg + x);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
            if (!seg_end) continue;
            in_seg = 0;
#pragma unroll
            for (uint32_t x = 0; x < CW; x += 16) add16(taddr + ACC_LOW + x, seg + x);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&low_empty);
#pragma unroll
            for (uint32_t e = 0; e < CW; e++) { grp[e] += seg[e]; seg[e] = 0.0f; }
            if (++in_grp != h && i + 1 != nkb) continue;
            in_grp = 0;
            // the sum of the groups waits in tensor memory, but for the last
            if (grps++)
#pragma unroll
                for (uint32_t x = 0; x < CW; x += 16) add16(taddr + ACC_TOT + x, grp + x);
            if (i + 1 == nkb) break;
#pragma unroll
            for (uint32_t x = 0; x < CW; x += 16) tmem_st16(taddr + ACC_TOT + x, grp + x);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
            for (uint32_t e = 0; e < CW; e++) grp[e] = 0.0f;
        }
        // the CTA's tile, where the pieces were (every MMA has completed): 512 bytes a row, the 16-byte vectors swizzled
        const uint32_t row = (warp & 3u) * 32 + lane;
#pragma unroll
        for (uint32_t x = 0; x < CW / 4; x++)
            *reinterpret_cast<float4*>(smem + row * (TN * 4) + (((col / 4 + x) ^ (row & 7u)) << 4)) = make_float4(grp[4 * x], grp[4 * x + 1], grp[4 * x + 2], grp[4 * x + 3]);
    }
    if (cs > 1) cluster_sync_all();
    else __syncthreads();
    if (warp >= 4 + NCW) {
        pdl_wait();   // (C is read and written)
        const uint32_t rows = min(TM, m - m0), rows_per = (rows + cs - 1) / cs, h = cs == cut.segs ? cut.h : 1u;
        const uint32_t base = smem_u32(smem);
        // A warp has a row at a time, a lane four columns of it. Rows with results that are not finite wait for a second pass (AGAIN).
        const uint32_t col = n0 + lane * 4, pw = warp - (4 + NCW);
        uint32_t later = 0;   // a bit per row of the warp
        auto store_rows = [&](auto again_c) {
            constexpr bool AGAIN = decltype(again_c)::value;
#pragma unroll 1
            for (uint32_t r0 = pw; r0 < rows_per; r0 += NPW) {
                const uint32_t row = rank * rows_per + r0, off = base + row * (TN * 4) + ((lane ^ (row & 7u)) << 4);
                if (row >= rows) break;
                if (AGAIN && !(later >> r0 / NPW & 1u)) continue;
                float4 p[MAX_SEGS];
#pragma unroll
                for (uint32_t r = 0; r < MAX_SEGS; r++)
                    if (r < cs) p[r] = ld_cluster(map_to_cta(off, r));
                float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t in_grp = 0;
#pragma unroll
                for (uint32_t r = 0; r < MAX_SEGS; r++)
                    if (r < cs) {
                        y[0] += p[r].x; y[1] += p[r].y; y[2] += p[r].z; y[3] += p[r].w;
                        if (++in_grp == h || r + 1 == cs) {
                            in_grp = 0;
#pragma unroll
                            for (int i = 0; i < 4; i++) { x[i] += y[i]; y[i] = 0.0f; }
                        }
                    }
                uint32_t bad = 0;
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) bad |= (col + i < n && !(fabsf(x[i]) < INFINITY) ? 1u : 0u) << i;
                if constexpr (AGAIN) {
                    const float4 v = again(a + (size_t)(m0 + row) * k, w, k, col, bad, make_float4(x[0], x[1], x[2], x[3]));
                    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
                } else if (__any_sync(0xffffffffu, bad)) {
                    later |= 1u << r0 / NPW;
                    continue;
                }
                if (col >= n) continue;
                if (flags & GEMM_SILU)
#pragma unroll
                    for (int i = 0; i < 4; i++) x[i] = x[i] / (1.0f + expf(-x[i]));
                float* const d = c + (size_t)(m0 + row) * n + col;
                if ((n & 3u) == 0 && ((uintptr_t)c & 15u) == 0) {
                    if (flags & GEMM_ADD) {
                        const float4 o = *reinterpret_cast<const float4*>(d);
                        x[0] = o.x + x[0]; x[1] = o.y + x[1]; x[2] = o.z + x[2]; x[3] = o.w + x[3];
                    }
                    *reinterpret_cast<float4*>(d) = make_float4(x[0], x[1], x[2], x[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (col + i < n) d[i] = (flags & GEMM_ADD) ? d[i] + x[i] : x[i];
                }
            }
        };
        store_rows(std::false_type{});
        if (later) store_rows(std::true_type{});
    }
    tc_fence_before();
    if (cs > 1) cluster_sync_all();   // nobody leaves while a peer may still read its tile
    else __syncthreads();
    tc_fence_after();
    if (warp == 2) tmem_dealloc(tmem, TMEM_COLS);
    if (threadIdx.x == 0 && fail_flag) atomicExch(&g_gemm_f32_status, fail_flag);
}

}  // namespace

// CTAs of clusters of `cs` that run at a time (a GPC holds whole clusters only, so fewer than the SMs); 0: not known
static uint32_t resident_ctas(uint32_t cs) {
    static uint32_t known[64][MAX_SEGS + 1] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(device_cache_mutex());
    uint32_t& v = known[dev & 63][cs];
    if (v) return v;
    if (cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, cs);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = cs;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_tc_kernel, &cfg) != cudaSuccess || n < 1) return 0;
    return v = (uint32_t)n * cs;
}

// 16-byte rows (k % 4 == 0) and aligned operands, see launch_gemm_f32_nt()
int launch_gemm_f32_tc(cudaStream_t st, const float* a, const float* wt, float* c, uint32_t m, uint32_t n, uint32_t k, uint32_t flags) {
    const uint32_t tn = cdiv(n, TN), tm = cdiv(m, TM), kb = cdiv(k, TK), a_box = m < TM ? m : TM;
    // Segments: as many as let one row tile occupy the SMs, at most five, or six where K or n is small and a K block more is a good part of the
    // launch: 4 x 1536 x 384 8.3 -> 6.8 us, the four products of a layer of a 384-wide model with 4, 128 and 512 rows 37.7, 51.4, 63.2 -> 33.3, 44.7, 57.2. (With
    // six everywhere, clusters of which only 22 run at a time: 512 x 768 x 768 12.6 -> 20.6, 512 x 768 x 3072 25.7 -> 42.5; with eight, and partial
    // tiles of as many to add, everything is 1 to 3 % slower.) Five segments are groups of three and two, so that a cluster of two can take more than
    // the one wave that clusters of five have: 512 x 960 x 320 17.6 -> 13.8 us, a prompt of 480 tokens of the 320-wide model 1270 -> 1007.
    const uint32_t most = k <= 384 || n <= 256 ? MAX_SEGS : 5;
    uint32_t segs = B200_SMS / tn;
    if (segs > most) segs = most;
    if (segs > kb) segs = kb;
    if (segs < 1) segs = 1;
    Cut cut;
    cut.per = cdiv(kb, segs);
    cut.segs = cdiv(kb, cut.per);
    cut.h = cdiv(cut.segs, 2);
    // Who adds them: the choice with the shortest way to the end, a CTA per SM at a time. In 0.1 us: 9 for a K block, up to 10 more for the split
    // of its activations, 65 for the rest of a tile, 10 more in a cluster.
    uint32_t cs = 0, best = 0;
    for (uint32_t o : {1u, cut.segs > 2 ? 2u : 1u, cut.segs}) {
        const uint32_t room = resident_ctas(o);
        AK_REQUIRE(room || o > 1, AK_ERR_CUDA, "f32 product: the kernel does not fit an SM");
        if (!room) continue;
        const uint32_t cost = cdiv(tn * tm * o, room) * ((o == 1 ? cut.segs : o == cut.segs ? 1 : cut.h) * cut.per * (9 + 10 * a_box / TM) + 65 + (o > 1 ? 10 : 0));
        if (!cs || cost < best) { cs = o; best = cost; }
    }
    CUtensorMap tmA, tmB;
    AK_TRY(make_tmap_2d(&tmA, a, 4, k, m, (uint64_t)k * 4, HALF, a_box, TMA_SWIZZLE_NONE));
    AK_TRY(make_tmap_2d(&tmB, wt, 4, k, n, (uint64_t)k * 4, HALF, TN, TMA_SWIZZLE_NONE));
    const dim3 grid(tn, tm, cs), cluster(1, 1, cs);
    return launch_k(gemm_f32_tc_kernel, grid, dim3(THREADS), SMEM, st, cs > 1 ? cluster : NO_CLUSTER, tmA, tmB, a, wt, c, m, n, k, flags, cut, a_box);
}

int gemm_f32_tc_status(unsigned int* out) {
    AK_CUDA(cudaMemcpyFromSymbol(out, g_gemm_f32_status, sizeof(unsigned int)));
    return AK_OK;
}

}  // namespace ak
