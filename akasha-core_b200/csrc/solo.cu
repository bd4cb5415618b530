// One decode step of ONE sequence (batch 1) as a single persistent kernel: embedding, every layer, lm_head, greedy argmax.
//
// What bounds it. A step streams every weight once (162M model: 494 MB f32 = 75 us at the measured HBM rate, 247 MB bf16 =
// 38 us), but as a chain of ~88 launches it took 0.37-0.45 ms: each launch is a boundary of ~2 us plus the latencies of
// its first loads, for 0.1-1 us of streaming. Here the two things are taken apart:
//   * the weight stream never stops: a producer thread per SM walks the SM's weight rows of ALL phases of all layers in
//     order and keeps a ~144 KB shared-memory ring of bulk copies full, whatever the other warps wait for;
//   * between phases only the activations cross the chip (a vector of dim .. ffn values), and each value travels with its
//     own flag: a 64-bit store {value, step number} that the consumers poll in L2. No grid barrier, no fence, one
//     one-way latency per phase.
// A layer has five phases: qkv rows -> attention (head, split of the positions) -> out-proj rows -> ffn-up rows ->
// ffn-down rows. The rows of a phase are dealt evenly over the 148 SMs. Inside an SM the K range is cut into slices of 64
// that belong to the 12 compute warps: a warp polls, normalises and multiplies its own slice only (the whole vector read
// by every warp cost more shared-memory bandwidth than the weights), for up to 24 rows at a time, and one reducer warp adds the
// 12 partial sums of each row, in warp order, and publishes it. The RMS norm's 1 / rms is a factor of the row sums, so its
// sum of squares travels with the partials and nothing waits for it. Every SM holds the residual stream, sliced the same
// way, in shared memory and adds every projection to it itself: no reduction across SMs.
// Every exchange buffer is written once per launch (they are per layer), so nothing is ever overwritten while a slow SM
// may still read it; the step number in the flags makes clearing them unnecessary.
//
// The grid is launched cooperatively (its blocks wait on one another): one block per SM, all resident. Every wait is
// bounded: on expiry a status word is set, later waits of the block return at once, and the block reports the failure where it
// would report its best logit, so that the step's done word says STEP_FAILED instead of a token. A warp whose wait for
// a chunk ran out releases no more chunks, so no slot is written again, and the producer leaves only when every copy it started has landed.
//
// Arithmetic: f32 products and sums of f32 or bf16 weights with f32 activations (the multi-launch bf16 path rounds the
// activations to bf16 for the tensor core; here they stay f32), keys and values rounded to the cache type.
// Nothing may spill: local memory is poison here (the ring leaves the L1 cache a few KB, every reload goes to L2; a 17-warp
// version with 96 registers took 0.67 ms per step, and 44 bytes of spills at 128 registers cost 20 us).
#include "solo.h"
#include "solo_plan.h"

namespace ak {

__device__ unsigned int g_solo_status = 0;

namespace {

using namespace solo;
static_assert(CTAS == B200_SMS, "a block per SM");
constexpr int NC = (NW + 1) * 32;        // threads of the compute and reducer warps (the block barrier's count)
// Four warpgroups: the first holds the producer (warp 0) and the reducer (warp 1), the others the compute warps. 512 threads
// launch with 128 registers each; the first group gives 48 of them to the others.
constexpr int THREADS = 512, FIRST_COMPUTE = 4;
constexpr int REGS_FIRST = 80, REGS_COMPUTE = 144;
static_assert(REGS_FIRST * 128 + REGS_COMPUTE * 384 <= 65536, "the split draws on the registers of the launch");
constexpr uint32_t BLOCK_FAILED = 0xfffffffeu;   // in the place of the index of a block's best logit (0xffffffff: it has none)
// Copies of every exchanged value: an SM polls copy (SM mod copies), which spreads the polls over the L2. Since an SM asks only for what is missing, a copy
// more costs about what it gives: bf16, 201 positions, 160.7 / 161.5 / 163.1 us a step with 1 / 2 / 4; f32 182.4 / 180.7 / 179.5, at 20 to 84 positions
// (64 tokens generated) 13.24 / 13.19 / 13.29 ms.
constexpr uint32_t MAX_REPLICAS = 2;
template <typename T> __device__ constexpr uint32_t replicas() { return sizeof(T) == 4 ? MAX_REPLICAS : 1; }

// ---- flagged exchange: {value, step} in one 64-bit word
template <uint32_t N> __device__ __forceinline__ void ll_put(uint64_t* p, size_t copy_stride, float v, uint32_t ep) {
    const uint64_t word = (uint64_t)__float_as_uint(v) | ((uint64_t)ep << 32);
#pragma unroll
    for (uint32_t c = 0; c < N; c++) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p + c * copy_stride), "l"(word) : "memory");
}
__device__ __forceinline__ void ll_ld2(const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool ll_ok(uint64_t v, uint32_t ep) { return (uint32_t)(v >> 32) == ep; }
__device__ __forceinline__ float ll_val(uint64_t v) { return __uint_as_float((uint32_t)v); }

struct Waiter {   // bounds the polling of one thread; `dead` is sticky for the block
    uint32_t* dead;
    __device__ __forceinline__ bool give_up(uint32_t& n, long long& t0) {
        if (n == 0) t0 = clock64();
        n++;
        if ((n & 63u) == 0) {
            if (*(volatile uint32_t*)dead) return true;
            if (clock64() - t0 > AK_WAIT_MAX_CYCLES) {
                *(volatile uint32_t*)dead = 1u;
                atomicExch(&g_solo_status, 1u);
                return true;
            }
        }
        return false;
    }
};
// n <= N value pairs at p, p + stride, ... (in words), all requested at once and then again as long as they are missing
template <int N>
__device__ __forceinline__ void poll_pairs(const uint64_t* p, uint32_t stride, uint32_t n, uint32_t ep, Waiter w, float2 (&v)[N]) {
    uint64_t a[N], b[N];
    uint32_t tries = 0;
    long long t0 = 0;
#pragma unroll
    for (int i = 0; i < N; i++) a[i] = b[i] = 0;   // (step 0 is none)
    for (;;) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; i++)   // what is not there yet (the polls of 148 SMs hold up each other and the stores they wait for)
            if ((uint32_t)i < n && !(ll_ok(a[i], ep) && ll_ok(b[i], ep))) ll_ld2(p + (size_t)i * stride, a[i], b[i]);
#pragma unroll
        for (int i = 0; i < N; i++)
            if ((uint32_t)i < n) ok = ok && ll_ok(a[i], ep) && ll_ok(b[i], ep);
        if (ok || w.give_up(tries, t0)) break;
    }
#pragma unroll
    for (int i = 0; i < N; i++)
        if ((uint32_t)i < n) v[i] = make_float2(ll_val(a[i]), ll_val(b[i]));
}
// one or two attention splits: the pair at p and the pair `ml` words on, the same `stride` further for the second split
__device__ __forceinline__ void poll_splits(const uint64_t* p, uint32_t ml, uint32_t stride, bool two, uint32_t ep, Waiter w, float2 (&v)[4]) {
    uint64_t a[4], b[4];
    uint32_t tries = 0;
    long long t0 = 0;
    for (;;) {
        ll_ld2(p, a[0], b[0]);
        ll_ld2(p + ml, a[1], b[1]);
        bool ok = ll_ok(a[0], ep) && ll_ok(b[0], ep) && ll_ok(a[1], ep) && ll_ok(b[1], ep);
        if (two) {
            ll_ld2(p + stride, a[2], b[2]);
            ll_ld2(p + stride + ml, a[3], b[3]);
            ok = ok && ll_ok(a[2], ep) && ll_ok(b[2], ep) && ll_ok(a[3], ep) && ll_ok(b[3], ep);
        }
        if (ok || w.give_up(tries, t0)) break;
    }
    v[0] = make_float2(ll_val(a[0]), ll_val(b[0]));
    v[1] = make_float2(ll_val(a[1]), ll_val(b[1]));
    if (two) {
        v[2] = make_float2(ll_val(a[2]), ll_val(b[2]));
        v[3] = make_float2(ll_val(a[3]), ll_val(b[3]));
    }
}
__device__ __forceinline__ bool wait_full(uint64_t* bar, uint32_t parity, uint32_t* dead) {
    if (mbar_try_wait(bar, parity)) return true;
    uint32_t n = 0;
    long long t0 = 0;
    Waiter w{dead};
    while (!mbar_try_wait(bar, parity))
        if (w.give_up(n, t0)) return false;
    return true;
}

__device__ __forceinline__ void bar_block() { asm volatile("bar.sync 1, %0;" ::"n"(NC) : "memory"); }
// the sums of squares of a norm phase are in shared memory: arrived at by the compute warps, waited for by the reducer
__device__ __forceinline__ void bar_ss_arrive() { asm volatile("bar.arrive 2, %0;" ::"n"(NC) : "memory"); }
__device__ __forceinline__ void bar_ss_wait() { asm volatile("bar.sync 2, %0;" ::"n"(NC) : "memory"); }

__device__ __forceinline__ void bulk_g2s_stream(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t pol) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
                 : "memory");
}

template <typename T> struct Vec;   // a 16-byte vector of weights / cache elements
template <> struct Vec<float> {
    static constexpr int N = 4;
    __device__ static __forceinline__ void get(const uint4& r, float* o) {
        o[0] = __uint_as_float(r.x); o[1] = __uint_as_float(r.y); o[2] = __uint_as_float(r.z); o[3] = __uint_as_float(r.w);
    }
    __device__ static __forceinline__ uint4 put(const float* v) {
        return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
    }
};
template <> struct Vec<bf16> {
    static constexpr int N = 8;
    __device__ static __forceinline__ void get(const uint4& r, float* o) {
        o[0] = __uint_as_float(r.x << 16); o[1] = __uint_as_float(r.x & 0xffff0000u);
        o[2] = __uint_as_float(r.y << 16); o[3] = __uint_as_float(r.y & 0xffff0000u);
        o[4] = __uint_as_float(r.z << 16); o[5] = __uint_as_float(r.z & 0xffff0000u);
        o[6] = __uint_as_float(r.w << 16); o[7] = __uint_as_float(r.w & 0xffff0000u);
    }
    __device__ static __forceinline__ uint4 put(const float* v) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const bf162 p = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
            o[e] = *reinterpret_cast<const uint32_t*>(&p);
        }
        return make_uint4(o[0], o[1], o[2], o[3]);
    }
};

__device__ __forceinline__ float redux_max(float v) {   // of the warp (a NaN is left out)
    float m;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}
// 1 / sqrt(m): the hardware's approximation and one Newton step (below 1 ulp). The step has no value where m is 0 or infinite (a
// residual stream whose squares overflow): there the approximation is exact.
__device__ __forceinline__ float inv_rms(float m) {
    const float y = rsqrtf(m);
    return y > 0.0f && y < INFINITY ? y * fmaf(-0.5f * m * y, y, 1.5f) : y;
}

struct Ring {
    uint8_t* base;
    uint64_t *full, *empty;
    uint32_t n;       // slots
};
struct Cursor {   // a place in the ring: slot and the parity of its current use
    uint32_t s = 0, ph = 0;
    __device__ __forceinline__ void advance(uint32_t by, uint32_t n) {   // by <= n
        s += by;
        if (s >= n) { s -= n; ph ^= 1u; }
    }
    __device__ __forceinline__ void retreat(uint32_t by, uint32_t n) {   // by <= n
        if (s < by) { s += n; ph ^= 1u; }
        s -= by;
    }
};

// Producer: this SM's rows of w, chunk by chunk. Returns false when a wait ran out.
template <typename T>
__device__ __forceinline__ bool stream_rows(const Ring& rg, Cursor& q, uint32_t& sent, const T* w, const Kind& d, uint64_t pol, uint32_t* dead) {
    const T* src = w + (size_t)d.r0 * d.k;
    uint32_t left = d.rows * d.k, in_row = 0;   // elements still to send; position inside the row (rows sent in pieces)
    const uint32_t whole = d.rpc * d.k;
    while (left) {
        if (sent >= rg.n && !wait_full(&rg.empty[q.s], q.ph ^ 1u, dead)) return false;
        uint32_t elems;
        if (d.ppr > 1) {
            elems = min(d.piece, d.k - in_row);
            in_row += elems;
            if (in_row == d.k) in_row = 0;
        } else {
            elems = min(whole, left);
        }
        const uint32_t bytes = elems * (uint32_t)sizeof(T);
        mbar_expect_tx(&rg.full[q.s], bytes);
        bulk_g2s_stream(rg.base + (size_t)q.s * SLOT, src, bytes, &rg.full[q.s], pol);
        src += elems;
        left -= elems;
        sent++;
        q.advance(1, rg.n);
    }
    return true;
}

// Compute warp: the partial sums of up to BLK rows of kind d over the warp's K slices. Lane (r, kq) = (lane / 8, lane % 8) works
// on rows r, r + 4, ... and 8 of a slice's 64 elements. The ring is ahead of the activations, so a block's first weights are
// moved into registers (fetch) while the activations are still under way: what is left on the path from the last
// activation to the row sums is the multiplications.
template <typename T> struct Block {
    static constexpr bool F32 = sizeof(T) == 4;
    static constexpr int WP = F32 ? 2 : 1;            // 16-byte pieces per row and slice
    static constexpr int PQ = 6;                      // rows per lane taken ahead
    uint4 w[PQ * WP];                                 // PQ rows of slice 0, or (n <= 8) two rows of slices 0 .. PQ / 2 - 1
    float acc[8];
    uint32_t base;                                    // ring byte of the block's first chunk

    // byte offset of slice sl inside a row, in the ring
    __device__ static __forceinline__ uint32_t slice_off(const Kind& d, uint32_t sl) {
        const uint32_t pc = d.ppr > 1 ? div_inv(sl, d.inv_pslices) : 0;
        return pc * SLOT + (sl * SLICE - pc * d.piece) * (uint32_t)sizeof(T);
    }
    // rows r + 4 i0, r + 4 (i0 + 1), ... (N of them) of slice sl
    template <int N>
    __device__ __forceinline__ void load(const Ring& rg, const Kind& d, uint32_t n, uint32_t sl, int i0, uint32_t lane, uint4* o) {
        const uint32_t r = lane >> 3, kq = lane & 7, ring = rg.n * SLOT;
        const uint32_t so = base + slice_off(d, sl) + kq * 16;
        // elements of lane kq in a slice: bf16 8 * kq .. + 7 (16 bytes); f32 4 * kq .. + 3 and 32 + 4 * kq .. + 3
        const bool in0 = sl * SLICE + kq * (F32 ? 4 : 8) < d.k, in1 = sl * SLICE + 32 + kq * 4 < d.k;
#pragma unroll
        for (int i = 0; i < N; i++) {
            uint32_t off = so + d.row_off[r][i0 + i];
            if (off >= ring) off -= ring;
            const bool ok = r + 4 * (i0 + i) < n;
            o[i * WP] = make_uint4(0, 0, 0, 0);
            if (ok && in0) o[i * WP] = *reinterpret_cast<const uint4*>(rg.base + off);
            if (F32) {
                o[i * WP + WP - 1] = make_uint4(0, 0, 0, 0);
                if (ok && in1) o[i * WP + WP - 1] = *reinterpret_cast<const uint4*>(rg.base + off + 128);
            }
        }
    }
    __device__ __forceinline__ static float dot(const uint4* o, const float (&x)[8], float acc) {
        float w[8];
        if (F32) {
            Vec<float>::get(o[0], w);
            Vec<float>::get(o[WP - 1], w + 4);
        } else {
            Vec<bf16>::get(o[0], w);
        }
        float t0 = fmaf(x[0], w[0], acc), t1 = x[4] * w[4];
        t0 = fmaf(x[1], w[1], t0); t1 = fmaf(x[5], w[5], t1);
        t0 = fmaf(x[2], w[2], t0); t1 = fmaf(x[6], w[6], t1);
        t0 = fmaf(x[3], w[3], t0); t1 = fmaf(x[7], w[7], t1);
        return t0 + t1;
    }
    // a slice of the activations, held as one pair per lane (elements 2 * lane, 2 * lane + 1), as this lane's 8 elements
    __device__ static __forceinline__ void spread(const float2& v, uint32_t lane, float (&x)[8]) {
        const uint32_t kq = lane & 7;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t src = F32 ? (j >> 1) * 16 + kq * 2 + (j & 1) : kq * 4 + j;
            x[2 * j] = __shfl_sync(0xffffffffu, v.x, src);
            x[2 * j + 1] = __shfl_sync(0xffffffffu, v.y, src);
        }
    }

    // wait for the block's chunks (from q on), take the first weights; false: a wait ran out
    __device__ __forceinline__ bool fetch(const Ring& rg, const Cursor& q, const Kind& d, uint32_t n, uint32_t chunks, uint32_t warp, uint32_t lane, uint32_t* dead) {
        base = q.s * SLOT;
        bool got = true;
        if (lane < chunks) {
            Cursor mine = q;
            mine.advance(lane, rg.n);
            got = wait_full(&rg.full[mine.s], mine.ph, dead);
        }
        got = __all_sync(0xffffffffu, got) != 0;
        __syncwarp();   // (a vote orders no memory: without this the lanes that do not wait might read before the weights are there)
        if (n <= 8) {
#pragma unroll
            for (int s = 0; s < PQ / 2; s++) load<2>(rg, d, n, warp + NW * s, 0, lane, w + 2 * s * WP);
        } else {
            load<PQ>(rg, d, n, warp, 0, lane, w);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = 0.0f;
        return got;
    }
    // add the warp's slice S (S == ANY: slice s > 0, nothing of it in registers), activations v
    static constexpr int ANY = 99;
    template <int S>
    __device__ __forceinline__ void add(const Ring& rg, const Kind& d, uint32_t n, uint32_t s, const float2& v, uint32_t warp, uint32_t lane) {
        float x[8];
        spread(v, lane, x);
        const uint32_t sl = warp + NW * (S == ANY ? s : (uint32_t)S);
        if (n <= 8) {
            if constexpr (2 * S + 1 < PQ) {
#pragma unroll
                for (int i = 0; i < 2; i++) acc[i] = dot(w + (2 * S + i) * WP, x, acc[i]);
            } else {
                uint4 o[2 * WP];
                load<2>(rg, d, n, sl, 0, lane, o);
#pragma unroll
                for (int i = 0; i < 2; i++) acc[i] = dot(o + i * WP, x, acc[i]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < (int)NQ; i += 2) {
                if (S == 0 && i + 1 < PQ) {
                    acc[i] = dot(w + i * WP, x, acc[i]);
                    acc[i + 1] = dot(w + (i + 1) * WP, x, acc[i + 1]);
                } else if ((uint32_t)(4 * i) < n) {
                    uint4 o[2 * WP];
                    load<2>(rg, d, n, sl, i, lane, o);
                    acc[i] = dot(o, x, acc[i]);
                    acc[i + 1] = dot(o + WP, x, acc[i + 1]);
                }
            }
        }
    }
    // slice s > 0 of a block whose slices come one by one
    __device__ __forceinline__ void add_slice(const Ring& rg, const Kind& d, uint32_t n, uint32_t s, const float2& v, uint32_t warp, uint32_t lane) {
        add<ANY>(rg, d, n, s, v, warp, lane);
    }
    // Lane (r, kq) gets the sum of row r + 4 * (4 (kq & 1) + 2 (kq >> 1 & 1) + (kq >> 2)) over the warp's slices (rows past n: zero).
    // The 8 lanes of a row group trade 4 + 2 + 1 values, each keeping one row.
    __device__ __forceinline__ float reduce(uint32_t lane) {
        const bool h1 = lane & 1, h2 = lane & 2, h4 = lane & 4;
        float b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) b[i] = (h1 ? acc[4 + i] : acc[i]) + __shfl_xor_sync(0xffffffffu, h1 ? acc[i] : acc[4 + i], 1);
        float c[2];
#pragma unroll
        for (int i = 0; i < 2; i++) c[i] = (h2 ? b[2 + i] : b[i]) + __shfl_xor_sync(0xffffffffu, h2 ? b[i] : b[2 + i], 2);
        return (h4 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h4 ? c[0] : c[1], 4);
    }
};

struct XchOff {   // word offsets inside a layer's exchange region
    uint32_t qkv, att, hid1, up, hid2, total;
    __host__ __device__ XchOff(uint32_t dim, uint32_t ffn, uint32_t heads) {
        qkv = 0;
        att = qkv + 3 * dim;                                   // per split: dim accumulator values, then (max, sum) per head
        hid1 = att + SOLO_MAX_SPLITS * (dim + 2 * heads);
        up = hid1 + dim;
        hid2 = up + ffn;
        total = hid2 + dim;
    }
};

template <typename T, int HD>
__global__ void __launch_bounds__(THREADS, 1) solo_kernel(const __grid_constant__ SoloArgs a, const uint32_t slots) {
    constexpr uint32_t REPLICAS = replicas<T>();
    constexpr int EPV = Vec<T>::N;
    constexpr int VR = HD / EPV;             // 16-byte vectors per cache row
    constexpr int RPI = 32 / VR;             // rows a warp loads per instruction
    constexpr int UP = 1024 / HD;            // positions of a warp's unit
    constexpr uint32_t KV_TILE = 1024 * sizeof(T);   // its keys (and its values): 1024 elements, contiguous in the pool
    constexpr int NL = KV_TILE / 512;        // loads per lane and tile
    constexpr uint32_t NA = att_warps(sizeof(T));    // compute warps with an attention unit
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full_bar[MAX_SLOTS], empty_bar[MAX_SLOTS], kv_full[NW], kv_empty[NW];
    __shared__ float part[2][NW][32], part_ss[NW];   // partial row sums of two blocks; sums of squares
    __shared__ float p_m[NW], p_l[NW], p_acc[NW][HD];
    __shared__ SoloLayer layers_sm[MAX_LAYERS];
    __shared__ Kind kinds[N_KINDS];
    __shared__ float best_v[NW];
    __shared__ uint32_t best_i[NW];
    __shared__ uint32_t dead;

    const uint32_t tid = threadIdx.x, warp_ = tid >> 5, lane_ = tid & 31;
    const uint32_t cta = blockIdx.x, ctas = gridDim.x;
    const uint32_t D = a.dim, F = a.ffn, H = a.heads, V = a.vocab, L = a.n_layers, ep = a.step;
    const Ring rg{smem, full_bar, empty_bar, slots};
    uint8_t* const kv_sm = smem + slots * SLOT;   // per compute warp: a unit of keys, a unit of values
    const XchOff xo(D, F, H);

    if (tid == 0) {
        for (uint32_t s = 0; s < slots; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], NW); }
        for (uint32_t i = 0; i < NW; i++) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
        dead = 0;
        mbar_fence_init();
    }
    if (tid >= 32 && tid < 32 + N_KINDS) {
        const uint32_t i = tid - 32;
        make_kind(kinds[i], i == 0 ? 3 * D : (i == 2 ? F : (i == 4 ? V : D)), i == 3 ? F : D, sizeof(T), slots, cta, ctas);
    }
    for (uint32_t i = tid; i < NW * HD; i += THREADS) p_acc[i / HD][i % HD] = 0.0f;
    if (tid < NW) { p_m[tid] = -INFINITY; p_l[tid] = 0.0f; }
    for (uint32_t i = tid; i < L * (uint32_t)(sizeof(SoloLayer) / 8); i += THREADS)
        reinterpret_cast<uint64_t*>(layers_sm)[i] = reinterpret_cast<const uint64_t*>(a.layers)[i];
    __syncthreads();

    const Waiter wt{&dead};
    const uint32_t n_pos = a.pos + 1, n_units = (n_pos + UP - 1) / UP;
    const uint32_t want = (n_units + NA - 1) / NA;
    uint32_t splits = want < SOLO_MAX_SPLITS ? want : SOLO_MAX_SPLITS;
    while (splits > 1 && splits * H > ctas) splits--;
    const uint32_t ups = (n_units + splits - 1) / splits;
    const uint32_t head = cta % H, split = cta / H;
    const bool attends = cta < splits * H;
    const uint32_t u_begin = split * ups, u_end = min(u_begin + ups, n_units), n_u = attends && u_end > u_begin ? u_end - u_begin : 0, rounds = (n_u + NA - 1) / NA;

    if (warp_ < FIRST_COMPUTE) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_FIRST));
    if (warp_ == 0) {
        // ---------------- producer: this SM's weight rows, in the order the compute warps use them (lane 0), and the cache
        // tiles of its attention share (lane i: those of compute warp i)
        const uint64_t pol = stays_in_l2(step_weight_bytes(sizeof(T), D, F, L, V)) ? policy_evict_normal() : policy_evict_first();
        Cursor q;
        uint32_t sent = 0, kv_sent = 0;
        bool ok = true;
        // round r of a layer's attention: units u_begin + NA r ..
        auto stream_kv = [&](const SoloLayer& w, uint32_t r) {
            const uint32_t u = u_begin + r * NA + lane_;
            if (lane_ >= NA || u >= u_end || !ok) return;
            const uint32_t p0 = u * UP;
            const size_t o = (((size_t)(p0 >> 4) * H + head) * 16 + (p0 & 15)) * HD;
            if (kv_sent > 0 && !wait_full(&kv_empty[lane_], (kv_sent - 1) & 1u, &dead)) { ok = false; return; }
            uint8_t* const dst = kv_sm + lane_ * 2 * KV_TILE;
            mbar_expect_tx(&kv_full[lane_], 2 * KV_TILE);
            bulk_g2s(dst, reinterpret_cast<const T*>(w.k_pool) + o, KV_TILE, &kv_full[lane_]);
            bulk_g2s(dst + KV_TILE, reinterpret_cast<const T*>(w.v_pool) + o, KV_TILE, &kv_full[lane_]);
            kv_sent++;
        };
#pragma unroll 1
        for (uint32_t i = 0; i <= 4 * L; i++) {
            const SoloLayer& w = layers_sm[i < 4 * L ? i >> 2 : 0];
            const void* const m = i == 4 * L ? a.lm_head : (i & 3) == 0 ? w.qkv : (i & 3) == 1 ? w.out : (i & 3) == 2 ? w.up : w.down;
            if (lane_ == 0 && ok) ok = stream_rows<T>(rg, q, sent, (const T*)m, kinds[i == 4 * L ? 4 : i & 3], pol, &dead);
            __syncwarp();
            // the first round's tiles right behind the qkv weights; later rounds, which wait for earlier ones to be used, behind
            // the out-proj's weights if those fit the ring (they cannot leave it before the attention is done), else before
            const bool late = kinds[1].chunks <= slots;
            if (i < 4 * L && (i & 3) == 0 && rounds) stream_kv(w, 0);
            if (i < 4 * L && (i & 3) == (late ? 1u : 0u))
#pragma unroll 1
                for (uint32_t r = 1; r < rounds; r++) stream_kv(w, r);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
        }
        // every copy lands before the block's memory goes away: a slot is only written again when its last copy was waited for, so
        // the latest one of each is enough
        if (lane_ < NA && kv_sent > 0) mbar_wait(&kv_full[lane_], (kv_sent - 1) & 1u);
        if (lane_ == 0)
            for (uint32_t i = 0; i < min(sent, slots); i++) {
                q.retreat(1, slots);
                mbar_wait(&full_bar[q.s], q.ph);
            }
        return;
    }

    // softmax in base e for f32 (parity mode: expf), base 2 otherwise
    const float sc = sizeof(T) == 4 ? a.scale : a.scale * 1.4426950408889634f;
    auto ex = [](float v) -> float { if constexpr (sizeof(T) == 4) return expf(v); else return exp2f(v); };
    uint32_t buf = 0;

    if (warp_ == 1) {
        const uint32_t lane = lane_;
        // ---------------- reducer: adds the warps' partial sums in warp order and publishes the rows, a lane per row
        const float inv_d = 1.0f / (float)D;
        const size_t copy = (size_t)L * xo.total + 2 * B200_SMS;   // words of one copy
#pragma unroll 1
        for (uint32_t it = 0; it < 4 * L; it++) {
            const uint32_t ph = it & 3;
            uint64_t* const xl = a.xch + (size_t)(it >> 2) * xo.total;
            if (ph == 1 && attends) {
                bar_block();
                // warps without a unit left max = -inf, sum = 0, accumulator 0
                float f[NA], M, ls = 0.0f, o[HD / 32];
                if constexpr (sizeof(T) == 4) {   // (an expf is long: lane i finds warp i's factor. With exponentials of the hardware that is no gain)
                    const float pm = lane < NA ? p_m[lane] : -INFINITY;
                    M = redux_max(pm);
                    const float fl = ex(pm - M);
#pragma unroll
                    for (int i = 0; i < (int)NA; i++) f[i] = __shfl_sync(0xffffffffu, fl, i);
                } else {
                    M = p_m[0];
#pragma unroll
                    for (int i = 1; i < (int)NA; i++) M = fmaxf(M, p_m[i]);
#pragma unroll
                    for (int i = 0; i < (int)NA; i++) f[i] = ex(p_m[i] - M);
                }
#pragma unroll
                for (int e = 0; e < HD / 32; e++) o[e] = 0.0f;
#pragma unroll
                for (int i = 0; i < (int)NA; i++) {
                    ls = fmaf(p_l[i], f[i], ls);
#pragma unroll
                    for (int e = 0; e < HD / 32; e++) o[e] = fmaf(p_acc[i][e * 32 + lane], f[i], o[e]);
                }
                uint64_t* const out = xl + xo.att + (size_t)split * (D + 2 * H);
#pragma unroll
                for (int e = 0; e < HD / 32; e++) ll_put<REPLICAS>(out + head * HD + e * 32 + lane, copy, splits == 1 ? o[e] / ls : o[e], ep);
                if (splits > 1 && lane < 2) ll_put<REPLICAS>(out + D + 2 * head + lane, copy, lane == 0 ? M : ls, ep);
            }
            const Kind& d = kinds[ph];
            uint64_t* const out = xl + (ph == 0 ? xo.qkv : ph == 1 ? xo.hid1 : ph == 2 ? xo.up : xo.hid2) + d.r0;
            float rs = 1.0f;
            if ((ph & 1) == 0) {   // the norm's factor, while the compute warps multiply
                bar_ss_wait();
                float u[NW];
#pragma unroll
                for (int i = 0; i < NW; i++) u[i] = part_ss[i];
#pragma unroll
                for (int i = 0; i < NW / 4; i++) u[i] = (u[4 * i] + u[4 * i + 1]) + (u[4 * i + 2] + u[4 * i + 3]);
                rs = inv_rms(((u[0] + u[1]) + u[2]) * inv_d + a.eps);
            }
#pragma unroll 1
            for (uint32_t j0 = 0; j0 < d.rows; j0 += d.blk, buf ^= 1u) {
                const bool mine = lane < min(d.blk, d.rows - j0);
                uint64_t* const dst = out + j0 + lane;
                bar_block();
                float t[NW];
#pragma unroll
                for (int i = 0; i < NW; i++) t[i] = part[buf][i][lane];
#pragma unroll
                for (int i = 0; i < NW / 4; i++) t[i] = (t[4 * i] + t[4 * i + 1]) + (t[4 * i + 2] + t[4 * i + 3]);
                float v = ((t[0] + t[1]) + t[2]) * rs;
                if (mine) {
                    // (bf16 weights: off by 2^-17 of the value at most, and 0 below about -87)
                    if (ph == 2) v = sizeof(T) == 4 ? v / (1.0f + expf(-v)) : __fdividef(v, 1.0f + __expf(-v));
                    ll_put<REPLICAS>(dst, copy, v, ep);
                }
            }
        }
        // ---- greedy argmax: this SM's best, then block 0's over all SMs; the lowest index wins ties
        auto better = [](float& v, uint32_t& i, float ov, uint32_t oi) { if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; } };
        auto warp_best = [&](float& v, uint32_t& i) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, v, o);
                const uint32_t oi = __shfl_xor_sync(0xffffffffu, i, o);
                better(v, i, ov, oi);
            }
        };
        bar_ss_wait();   // (the lm_head's sums of squares are the compute warps' own business)
        bar_block();     // logits and every warp's best are in shared memory
        float bv = lane < NW ? best_v[lane] : -INFINITY;
        uint32_t bi = lane < NW ? best_i[lane] : 0xffffffffu;
        warp_best(bv, bi);
        if (a.logits_host) bar_block();   // the logits are on the host
        uint64_t* const fin = a.xch + (size_t)L * xo.total;
        if (lane == 0) {
            ll_put<REPLICAS>(fin + 2 * cta, copy, bv, ep);
            ll_put<REPLICAS>(fin + 2 * cta + 1, copy, __uint_as_float(*(volatile uint32_t*)&dead ? BLOCK_FAILED : bi), ep);
        }
        if (cta != 0) return;
        bv = -INFINITY;
        bi = 0xffffffffu;
        bool failed = false;
        for (uint32_t c = lane; c < ctas; c += 32) {
            float2 p[1];
            poll_pairs(fin + 2 * c, 0, 1, ep, wt, p);
            failed = failed || __float_as_uint(p[0].y) == BLOCK_FAILED;
            better(bv, bi, p[0].x, __float_as_uint(p[0].y));
        }
        warp_best(bv, bi);
        failed = __any_sync(0xffffffffu, failed || *(volatile uint32_t*)&dead);
        if (lane == 0) {
            const uint32_t tok = bi < V ? bi : 0u;   // (no logit above -inf: 0)
            *a.sampled = tok;
            if (a.done_host) {
                __threadfence_system();
                *(volatile uint64_t*)a.done_host = (uint64_t)(failed ? STEP_FAILED : tok) | ((uint64_t)ep << 32);
            }
        }
        return;
    }

    // ---------------- compute warps. Slice i of a warp is slice warp + 12 i of the vector, a pair of elements per lane.
    if (warp_ < FIRST_COMPUTE) return;   // warps 2 and 3 fill the warpgroup
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_COMPUTE));
    const uint32_t warp = warp_ - FIRST_COMPUTE, lane = lane_;
    const uint32_t max_d = (D / SLICE + NW - 1) / NW, max_f = ((F + SLICE - 1) / SLICE + NW - 1) / NW;
    const uint32_t nsl_d = (D / SLICE + NW - 1 - warp) / NW, nsl_f = ((F + SLICE - 1) / SLICE + NW - 1 - warp) / NW;
    float2* const hid = reinterpret_cast<float2*>(kv_sm + NA * 2 * KV_TILE) + (size_t)warp * (max_d + max_f) * 32 + lane;   // residual stream: [slice][lane]
    float2* const xs = hid + max_d * 32;    // a phase's activations, for the row blocks after the first
    const uint32_t part_i = (lane >> 3) + ((lane & 1) << 4) + ((lane & 2) << 2) + (lane & 4);   // row of a block this lane ends up with
    {
        const uint32_t id = a.tok_src >= 0 ? (uint32_t)a.tok_src : *a.sampled;
        const T* row = reinterpret_cast<const T*>(a.embedding) + (size_t)(id < V ? id : 0) * D;
        for (uint32_t i = 0; i < nsl_d; i++) {
            const uint32_t e = (warp + NW * i) * SLICE + 2 * lane;
            hid[i * 32] = id < V ? make_float2(Cvt<T>::to_f(row[e]), Cvt<T>::to_f(row[e + 1])) : make_float2(0.f, 0.f);
        }
    }
    const uint64_t* const xch = a.xch + (size_t)(cta % REPLICAS) * ((size_t)L * xo.total + 2 * B200_SMS);   // the copy this SM polls
    Cursor q;   // the next chunk
    uint32_t kv_use = 0;

    // A phase's first block: release the previous block's chunks (only now: the partial sums before were on the critical path,
    // this is in the shadow of the reducer and the exchange), then wait for and take the first weights. In this order: the
    // two blocks together may be more than the ring.
    uint32_t to_release = 0;   // chunks before q that this warp is done with
    bool alive = true;         // no wait of this warp for a copy has run out. After the first that did it releases nothing any more: a later
                               // wait may take an old phase for its own, and the slot's copy may still be under way
    auto release = [&]() {
        if (lane < to_release) {
            Cursor c = q;
            c.retreat(to_release - lane, rg.n);
            mbar_arrive(&rg.empty[c.s]);
        }
        to_release = 0;
    };
    auto begin = [&](Block<T>& blk, const Kind& d) {
        release();
        alive = blk.fetch(rg, q, d, d.n0, d.chunks0, warp, lane, &dead) && alive;
    };
    // After the first block's activations have been added: publish its partial sums, then work through the other row
    // blocks, activations from xs. A kind without rows on this SM has no block (and no barrier).
    auto finish = [&](Block<T>& blk, const Kind& d, uint32_t nsl) {
        if (d.rows == 0) return;
        uint32_t chunks = d.chunks0, j0 = d.n0;
        for (;;) {
            part[buf][warp][part_i] = blk.reduce(lane);
            bar_block();
            buf ^= 1u;
            q.advance(chunks, rg.n);
            to_release = alive ? chunks : 0;
            if (j0 >= d.rows) break;
            release();
            const uint32_t n = min(d.blk, d.rows - j0);
            chunks = d.ppr > 1 ? n * d.ppr : div_inv(n + d.rpc - 1, d.inv_rpc);
            j0 += n;
            alive = blk.fetch(rg, q, d, n, chunks, warp, lane, &dead) && alive;
            if (nsl) blk.template add<0>(rg, d, n, 0, xs[0], warp, lane);
#pragma unroll 1
            for (uint32_t i = 1; i < nsl; i++) blk.add_slice(rg, d, n, i, xs[i * 32], warp, lane);
        }
    };
    // norm phases (qkv, ffn-up, lm_head): residual += src (nullptr: nothing), activations = residual * gain
    auto norm_phase = [&](const Kind& d, const float* gain, const uint64_t* src) {
        const bool more = d.rows > d.n0 || nsl_d > 1;   // the activations are needed again
        Block<T> blk;
        begin(blk, d);
        // the warp's slices: all polled first, then the sum of squares goes to the reducer, then the products
        float ss = 0.0f;
        float2 x0 = make_float2(0.f, 0.f);
#pragma unroll 1
        for (uint32_t i = 0; i < nsl_d; i++) {
            const uint32_t e = (warp + NW * i) * SLICE + 2 * lane;
            const float2 g = __ldg(reinterpret_cast<const float2*>(gain + e));
            float2 h = hid[i * 32], v[1];
            if (src) {
                poll_pairs(src + e, 0, 1, ep, wt, v);
                h.x += v[0].x;
                h.y += v[0].y;
            }
            const float2 x = make_float2(h.x * g.x, h.y * g.y);
            ss += h.x * h.x + h.y * h.y;
            hid[i * 32] = h;
            if (i == 0) x0 = x;
            if (more) xs[i * 32] = x;
        }
        ss = warp_sum(ss);
        if (lane == 0) part_ss[warp] = ss;
        __syncwarp();
        bar_ss_arrive();
        if (nsl_d) blk.template add<0>(rg, d, d.n0, 0, x0, warp, lane);
#pragma unroll 1
        for (uint32_t i = 1; i < nsl_d; i++) blk.add_slice(rg, d, d.n0, i, xs[i * 32], warp, lane);
        finish(blk, d, nsl_d);
    };

    // ---- lm_head: many rows and no one waiting for the single row, so a warp takes whole rows (row warp + 12 i), with its share
    // of the activations in registers: a third of the instructions per weight of the sliced form
    auto lm_head = [&](const uint64_t* src) {
        constexpr int NV = 1024 / (32 * EPV);   // 16-byte vectors a lane holds: rows of up to 1024
        const Kind& d = kinds[4];
        release();
        float ss = 0.0f;
        for (uint32_t i = 0; i < nsl_d; i++) {
            const uint32_t e = (warp + NW * i) * SLICE + 2 * lane;
            const float2 g = __ldg(reinterpret_cast<const float2*>(a.final_norm + e));
            float2 h = hid[i * 32], v[1];
            if (src) {
                poll_pairs(src + e, 0, 1, ep, wt, v);
                h.x += v[0].x;
                h.y += v[0].y;
            }
            ss += h.x * h.x + h.y * h.y;
            xs[i * 32] = make_float2(h.x * g.x, h.y * g.y);
        }
        ss = warp_sum(ss);
        if (lane == 0) part_ss[warp] = ss;
        asm volatile("bar.sync 3, %0;" ::"n"(NW * 32) : "memory");   // the compute warps' activations and sums are in shared memory
        bar_ss_arrive();
        ss = 0.0f;
#pragma unroll
        for (int i = 0; i < NW; i++) ss += part_ss[i];
        const float rs = inv_rms(ss / (float)D + a.eps);
        const float* const x_all = reinterpret_cast<const float*>(kv_sm + NA * 2 * KV_TILE);
        float* const logit_sm = reinterpret_cast<float*>(kv_sm);   // (no cache tile is in use any more)
        float bv = -INFINITY;
        uint32_t bi = 0xffffffffu, rel = 0;   // chunks released
        Cursor cur = q;                        // chunk number rel
        auto release_to = [&](uint32_t c) {    // a chunk is waited for even where this warp has no row in it: only then is every arrival of the slot's last use in
            __syncwarp();
            for (; rel < c; rel++, cur.advance(1, rg.n)) {
                alive = __all_sync(0xffffffffu, wait_full(&rg.full[cur.s], cur.ph, &dead)) && alive;
                if (alive && lane == 0) mbar_arrive(&rg.empty[cur.s]);
            }
        };
        const bool in_regs = D <= 32 * EPV * NV;
        float xr[NV * EPV];
        auto load_x = [&](uint32_t v, float* o) {   // vector v of this lane: elements (32 v + lane) * EPV ..
            const uint32_t e = (v * 32 + lane) * EPV, sl = e / SLICE;
            const float* p = x_all + ((sl % NW) * (max_d + max_f) + max_d + sl / NW) * SLICE + e % SLICE;
#pragma unroll
            for (int j = 0; j < EPV; j += 4) {
                const float4 t = e < D ? *reinterpret_cast<const float4*>(p + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                o[j] = t.x; o[j + 1] = t.y; o[j + 2] = t.z; o[j + 3] = t.w;
            }
        };
#pragma unroll
        for (int v = 0; v < NV; v++) load_x(v, xr + v * EPV);
#pragma unroll 1
        for (uint32_t j = warp; j < d.rows; j += NW) {
            const uint32_t c = div_inv(j, d.inv_rpc);
            release_to(c);
            wait_full(&rg.full[cur.s], cur.ph, &dead);
            const uint8_t* const wp = rg.base + cur.s * SLOT + (j - c * d.rpc) * D * (uint32_t)sizeof(T) + lane * 16;
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int v = 0; v < NV; v++) {
                float wv[EPV];
                Vec<T>::get((v * 32 + lane) * EPV < D ? *reinterpret_cast<const uint4*>(wp + v * 512) : make_uint4(0, 0, 0, 0), wv);
#pragma unroll
                for (int e = 0; e < EPV; e++) acc[e & 3] = fmaf(xr[v * EPV + e], wv[e], acc[e & 3]);
            }
            if (!in_regs)
#pragma unroll 1
                for (uint32_t v = NV; v * 32 * EPV < D; v++) {
                    float wv[EPV], xv[EPV];
                    load_x(v, xv);
                    Vec<T>::get((v * 32 + lane) * EPV < D ? *reinterpret_cast<const uint4*>(wp + v * 512) : make_uint4(0, 0, 0, 0), wv);
#pragma unroll
                    for (int e = 0; e < EPV; e++) acc[e & 3] = fmaf(xv[e], wv[e], acc[e & 3]);
                }
            const float logit = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3])) * rs;
            if (logit > bv) { bv = logit; bi = d.r0 + j; }
            if (lane == 0) logit_sm[j] = logit;
        }
        release_to((d.rows + d.rpc - 1) / d.rpc);
        if (lane == 0) { best_v[warp] = bv; best_i[warp] = bi; }
        bar_block();
        if (a.logits)
            for (uint32_t j = warp * 32 + lane; j < d.rows; j += NW * 32) a.logits[d.r0 + j] = logit_sm[j];
        if (a.logits_host) {
            for (uint32_t j = warp * 32 + lane; j < d.rows; j += NW * 32) a.logits_host[d.r0 + j] = logit_sm[j];
            __threadfence_system();   // on the host before this SM reports its best, and so before the step is done
            bar_block();
        }
    };

    auto attend = [&](const SoloLayer& w, const uint64_t* xl) {
        const uint32_t lv = lane % VR, sub = lane / VR;
        const uint32_t u0 = u_begin + warp;
        if (warp < NA && u0 < u_end) {
            // the new token's q, k, v: elements 2 * lane, 2 * lane + 1 (+ 64 j) here, rotated, then traded into 16-byte vectors
            const bool has_new = (n_units - 1 - u0) % NA == 0 && n_units <= u_end;   // this warp's last unit holds the new position
            float2 nv[3][HD / 64];
            {
                float2 cs[HD / 64];
#pragma unroll
                for (int j = 0; j < HD / 64; j++) cs[j] = __ldg(a.rope + (size_t)a.pos * (HD / 2) + j * 32 + lane);
#pragma unroll
                for (int j = 0; j < HD / 64; j++) {
                    float2 v[3];
                    poll_pairs(xl + xo.qkv + head * HD + j * 64 + 2 * lane, D, has_new ? 3 : 1, ep, wt, v);
                    if (!has_new) v[1] = v[2] = make_float2(0.f, 0.f);
                    rope_rotate(v[0].x, v[0].y, cs[j].x, cs[j].y, nv[0][j].x, nv[0][j].y);
                    rope_rotate(v[1].x, v[1].y, cs[j].x, cs[j].y, nv[1][j].x, nv[1][j].y);
                    nv[2][j] = v[2];
                }
            }
            auto vec_of = [&](int which, float (&o)[EPV]) {
#pragma unroll
                for (int e = 0; e < EPV; e += 2) {
                    const uint32_t el = lv * EPV + e;
                    float2 r = make_float2(__shfl_sync(0xffffffffu, nv[which][0].x, (el >> 1) & 31), __shfl_sync(0xffffffffu, nv[which][0].y, (el >> 1) & 31));
                    if (HD == 128) {
                        const float2 r1 = make_float2(__shfl_sync(0xffffffffu, nv[which][HD / 64 - 1].x, (el >> 1) & 31),
                                                      __shfl_sync(0xffffffffu, nv[which][HD / 64 - 1].y, (el >> 1) & 31));
                        if (el >= 64) r = r1;
                    }
                    o[e] = r.x;
                    o[e + 1] = r.y;
                }
            };
            float qv[EPV];
            vec_of(0, qv);
            uint4 kn = make_uint4(0, 0, 0, 0), vn = kn;
            if (has_new) {   // (warp-uniform) its key and value go to the pools
                float t[EPV];
                vec_of(1, t);
                kn = Vec<T>::put(t);
                vec_of(2, t);
                vn = Vec<T>::put(t);
                if (sub == 0) {
                    const size_t o = (((size_t)(a.pos >> 4) * H + head) * 16 + (a.pos & 15)) * HD + lv * EPV;
                    *reinterpret_cast<uint4*>(reinterpret_cast<T*>(w.k_pool) + o) = kn;
                    *reinterpret_cast<uint4*>(reinterpret_cast<T*>(w.v_pool) + o) = vn;
                }
            }
            float m_run = -INFINITY, l_run = 0.0f, acc[EPV];
#pragma unroll
            for (int e = 0; e < EPV; e++) acc[e] = 0.0f;
            const uint8_t* const ks = kv_sm + warp * 2 * KV_TILE + lane * 16;
#pragma unroll 1
            for (uint32_t u = u0; u < u_end; u += NA, kv_use++) {
                const uint32_t newest = a.pos - u * UP;   // the new position's row in this unit (>= UP: not here)
                const bool got = wait_full(&kv_full[warp], kv_use & 1u, &dead);
                float s[NL], mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    uint4 raw = *reinterpret_cast<const uint4*>(ks + i * 512);
                    if (i * RPI + sub == newest) raw = kn;
                    float kf[EPV], t = 0.0f;
                    Vec<T>::get(raw, kf);
#pragma unroll
                    for (int e = 0; e < EPV; e++) t = fmaf(qv[e], kf[e], t);
                    s[i] = t;
                }
#pragma unroll
                for (int o = VR / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < NL; i++) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    s[i] = (uint32_t)(i * RPI) + sub <= newest ? s[i] * sc : -INFINITY;
                    mx = fmaxf(mx, s[i]);
                }
#pragma unroll
                for (int o = VR; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m_run, mx), corr = ex(m_run - m_new);
                float ls = 0.0f;
#pragma unroll
                for (int e = 0; e < EPV; e++) acc[e] *= corr;
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    const float p = ex(s[i] - m_new);
                    ls += p;
                    const uint32_t row = i * RPI + sub;
                    uint4 raw = *reinterpret_cast<const uint4*>(ks + KV_TILE + i * 512);
                    if (row >= newest) raw = row == newest ? vn : make_uint4(0, 0, 0, 0);   // rows past the sequence may hold anything
                    float vf[EPV];
                    Vec<T>::get(raw, vf);
#pragma unroll
                    for (int e = 0; e < EPV; e++) acc[e] = fmaf(p, vf[e], acc[e]);
                }
                l_run = l_run * corr + ls;
                m_run = m_new;
                // The buffer goes back behind a value that all of this tile's loads went into, in every lane: a load from shared memory and a later
                // arrival on a barrier are not in order by themselves (the comparison is true of every sum: a NaN comes out as 0x7fffffff).
                alive = __all_sync(0xffffffffu, got && __float_as_uint(acc[0]) != 0xffffffffu) && alive;
                if (alive && lane == 0) mbar_arrive(&kv_empty[warp]);
            }
#pragma unroll
            for (int o = VR; o < 32; o <<= 1) {
                l_run += __shfl_xor_sync(0xffffffffu, l_run, o);
#pragma unroll
                for (int e = 0; e < EPV; e++) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
            }
            if (sub == 0) {
#pragma unroll
                for (int e = 0; e < EPV; e++) p_acc[warp][lv * EPV + e] = acc[e];
            }
            if (lane == 0) { p_m[warp] = m_run; p_l[warp] = l_run; }
        }
        bar_block();
    };

#pragma unroll 1
    for (uint32_t l = 0;; l++) {
        const uint64_t* const xl = xch + (size_t)l * xo.total;
        const bool last = l == L;
        const SoloLayer& w = layers_sm[last ? 0 : l];
        const uint64_t* const src = l ? xl - xo.total + xo.hid2 : nullptr;
        if (last) { lm_head(src); break; }
        norm_phase(kinds[0], w.norm_1, src);
        if (attends) {
            release();   // (the copies of the coming phases go on meanwhile)
            attend(w, xl);
        }
        {   // ---- out-proj: merge the heads' splits, in split order
            const Kind& d = kinds[1];
            const bool more = d.rows > d.n0;
            Block<T> blk;
            begin(blk, d);
#pragma unroll 1
            for (uint32_t i = 0; i < nsl_d; i++) {
                const uint32_t e = (warp + NW * i) * SLICE + 2 * lane;
                const uint64_t* p = xl + xo.att;
                float2 v;
                if (splits == 1) {
                    float2 o[1];
                    poll_pairs(p + e, 0, 1, ep, wt, o);
                    v = o[0];
                } else {
                    float M = -INFINITY, ls = 0.0f;
                    v = make_float2(0.f, 0.f);
                    const uint32_t ml = D + 2 * (e / HD) - e;   // a split's max and sum behind its accumulator
#pragma unroll 1
                    for (uint32_t s = 0; s < splits; s += 2, p += 2 * (D + 2 * H)) {
                        float2 o[4];   // accumulator pair, (max, sum) of two splits
                        const bool two = s + 1 < splits;
                        poll_splits(p + e, ml, D + 2 * H, two, ep, wt, o);
                        if (!two) { o[2] = make_float2(0.f, 0.f); o[3] = make_float2(-INFINITY, 0.0f); }
                        const float m2 = fmaxf(fmaxf(M, o[1].x), o[3].x), f0 = ex(M - m2), f1 = ex(o[1].x - m2), f2 = ex(o[3].x - m2);
                        ls = fmaf(o[3].y, f2, fmaf(o[1].y, f1, ls * f0));
                        v.x = fmaf(o[2].x, f2, fmaf(o[0].x, f1, v.x * f0));
                        v.y = fmaf(o[2].y, f2, fmaf(o[0].y, f1, v.y * f0));
                        M = m2;
                    }
                    v.x /= ls;
                    v.y /= ls;
                }
                if (i == 0) blk.template add<0>(rg, d, d.n0, 0, v, warp, lane);
                else blk.add_slice(rg, d, d.n0, i, v, warp, lane);
                if (more) xs[i * 32] = v;
            }
            finish(blk, d, nsl_d);
        }
        norm_phase(kinds[2], w.norm_2, xl + xo.hid1);
        {   // ---- ffn-down
            constexpr uint32_t PN = sizeof(T) == 4 ? 2 : 4;   // slices polled at once (registers)
            const Kind& d = kinds[3];
            const bool more = d.rows > d.n0;
            Block<T> blk;
            begin(blk, d);
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < nsl_f; i0 += PN) {
                float2 v[PN];
                const uint32_t n = min(PN, nsl_f - i0), e = (warp + NW * i0) * SLICE + 2 * lane;
                // the vector's last slice may be short: pairs past its end count for nothing
                const uint32_t np = e + (n - 1) * NW * SLICE < F ? n : n - 1;
#pragma unroll
                for (int i = 0; i < (int)PN; i++) v[i] = make_float2(0.f, 0.f);
                poll_pairs(xl + xo.up + e, NW * SLICE, np, ep, wt, v);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < (int)PN; i++)
                    if (more && (uint32_t)i < n) xs[(i0 + i) * 32] = v[i];
                if (i0 == 0) {
                    blk.template add<0>(rg, d, d.n0, 0, v[0], warp, lane);
                    if (n > 1) blk.template add<1>(rg, d, d.n0, 1, v[1], warp, lane);
                    if (PN > 2 && n > 2) blk.template add<2>(rg, d, d.n0, 2, v[PN - 2], warp, lane);
                    if (PN > 2 && n > 3) blk.template add<3>(rg, d, d.n0, 3, v[PN - 1], warp, lane);
                } else {
#pragma unroll
                    for (int i = 0; i < (int)PN; i++)
                        if ((uint32_t)i < n) blk.add_slice(rg, d, d.n0, i0 + i, v[i], warp, lane);
                }
            }
            finish(blk, d, nsl_f);
        }
    }
}

}  // namespace

bool solo_supported(uint32_t dtype, uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers, uint32_t vocab) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    return (uint32_t)sms >= B200_SMS && shape_supported(dtype == AK_F32 ? 4 : 2, dim, ffn, heads, n_layers, vocab);
}

size_t solo_xch_words(uint32_t dim, uint32_t ffn, uint32_t heads, uint32_t n_layers) {
    return MAX_REPLICAS * ((size_t)n_layers * XchOff(dim, ffn, heads).total + 2 * B200_SMS);
}

template <typename T, int HD>
static int launch_solo_t(cudaStream_t st, const SoloArgs& a) {
    Plan p;
    AK_REQUIRE(make_plan(sizeof(T), a.dim, a.ffn, p), AK_ERR_UNSUPPORTED, "solo step: model does not fit the kernel's shared memory");
    {
        static bool attr_set[64] = {};
        int dev = 0;
        AK_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lock(device_cache_mutex());
        if (!attr_set[dev & 63]) {
            AK_CUDA(cudaFuncSetAttribute(solo_kernel<T, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_DYN_SMEM));
            attr_set[dev & 63] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B200_SMS);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    AK_CUDA(cudaLaunchKernelEx(&cfg, solo_kernel<T, HD>, a, p.slots));
    AK_COUNT_LAUNCH();
    return AK_OK;
}

int launch_solo(cudaStream_t st, uint32_t dtype, const SoloArgs& a) {
    const uint32_t hd = a.dim / a.heads;
    if (dtype == AK_F32) return hd == 64 ? launch_solo_t<float, 64>(st, a) : launch_solo_t<float, 128>(st, a);
    return hd == 64 ? launch_solo_t<bf16, 64>(st, a) : launch_solo_t<bf16, 128>(st, a);
}

int solo_status(unsigned int* out) {
    AK_CUDA(cudaMemcpyFromSymbol(out, g_solo_status, sizeof(unsigned int)));
    return AK_OK;
}

}  // namespace ak
