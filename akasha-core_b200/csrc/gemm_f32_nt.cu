// True-fp32 product with the weight matrix K-major: C[m,n] (op)= A[m,k] @ Wt[n,k]^T, the layout the runner keeps its f32 projections
// in (each output column's weights contiguous, so that a batch-1 step streams whole rows).
//
// GEMM: gemm_f32_tc.cu where rows and operands are 16-byte aligned and (n, k) is not small. Else on the FMA pipe: 64 x 128 tile per CTA, 128 threads, 8 x 8
// outputs per thread as packed pairs (fma.rn.f32x2: two IEEE fused multiply-adds per instruction), K blocks of 16 double-buffered in shared memory with
// the next block's global loads in flight; K is split over a thread-block cluster and the partial tiles are added through distributed
// shared memory in rank order. Either way the order of a sum is a function of (n, k) only: it does not depend on how many rows share the launch.
// GEMV: a warp per output, the weights streamed once with 128-bit loads. Its order of sums is another one, so it is only for rows that
// never share a launch (GEMM_ALONE: the decode row of a runner with one slot).
#include <cooperative_groups.h>

#include "kernels.h"

namespace cg = cooperative_groups;

namespace ak {
namespace ntf32 {

constexpr int BM = 64, BN = 128, BK = 16, THREADS = 128;

// Row k of a tile starts 8 (k / 4) floats late: the transposing stores of 8 rows x 4 k groups fall into 32 banks.
__device__ __host__ constexpr uint32_t at(uint32_t k, uint32_t width) { return k * width + 8 * (k >> 2); }
struct Tiles {
    float a[2][at(BK, BM)];
    float b[2][at(BK, BN)];
};
union Smem {
    Tiles t;
    float red[BM][BN];   // a CTA's partial tile (split K)
};

__device__ __forceinline__ void ffma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint64_t dup2(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}

// 4 consecutive k of one row; k % 4 == 0 and 16-byte rows unless SCALAR
template <bool SCALAR>
__device__ __forceinline__ float4 load4(const float* __restrict__ p, uint32_t row, uint32_t rows, uint32_t k0, uint32_t k_end, uint32_t ld) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= rows) return v;
    const float* s = p + (size_t)row * ld + k0;
    if (!SCALAR) {
        if (k0 < k_end) v = *reinterpret_cast<const float4*>(s);
    } else {
        if (k0 < k_end) v.x = s[0];
        if (k0 + 1 < k_end) v.y = s[1];
        if (k0 + 2 < k_end) v.z = s[2];
        if (k0 + 3 < k_end) v.w = s[3];
    }
    return v;
}

template <bool SCALAR>
__global__ void __launch_bounds__(THREADS, 3)
gemm_kernel(const float* __restrict__ a, const float* __restrict__ w, float* __restrict__ c, uint32_t m, uint32_t n, uint32_t k, uint32_t flags) {
    __shared__ __align__(16) Smem sm;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t ks = gridDim.z, rank = blockIdx.z;
    const uint32_t t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const uint32_t m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const uint32_t per = ((k + BK - 1) / BK + ks - 1) / ks * BK;
    const uint32_t k_begin = min(rank * per, k), k_end = min(k_begin + per, k);

    // Four lanes read the 64 bytes of a row that a K block has (a lane per row instead: 32 sectors per load, and the L1 was busier
    // than the FMA pipe). The tiles are K-major.
    const uint32_t lr = t >> 2, lq = t & 3;
    float4 ra[2], rb[4];
    auto fetch_b = [&](uint32_t k0) {
#pragma unroll
        for (int i = 0; i < 4; i++) rb[i] = load4<SCALAR>(w, n0 + lr + 32 * i, n, k0 + 4 * lq, k_end, k);
    };
    auto fetch_a = [&](uint32_t k0) {
#pragma unroll
        for (int i = 0; i < 2; i++) ra[i] = load4<SCALAR>(a, m0 + lr + 32 * i, m, k0 + 4 * lq, k_end, k);
    };
    auto put = [&](uint32_t buf) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float* d = &sm.t.a[buf][at(4 * lq, BM) + lr + 32 * i];
            d[0] = ra[i].x; d[BM] = ra[i].y; d[2 * BM] = ra[i].z; d[3 * BM] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float* d = &sm.t.b[buf][at(4 * lq, BN) + lr + 32 * i];
            d[0] = rb[i].x; d[BN] = rb[i].y; d[2 * BN] = rb[i].z; d[3 * BN] = rb[i].w;
        }
    };

    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0;

    fetch_b(k_begin);   // the weights do not depend on the preceding kernel
    pdl_wait();
    pdl_trigger();
    fetch_a(k_begin);
    put(0);
    __syncthreads();
    uint32_t buf = 0;
    for (uint32_t k0 = k_begin; k0 < k_end; k0 += BK) {
        const bool more = k0 + BK < k_end;
        if (more) { fetch_a(k0 + BK); fetch_b(k0 + BK); }
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float* const ar = &sm.t.a[buf][at(kk, BM) + ty * 8];
            const float* const br = &sm.t.b[buf][at(kk, BN) + tx * 4];
            const float4 a0 = *reinterpret_cast<const float4*>(ar), a1 = *reinterpret_cast<const float4*>(ar + 4);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(br), b1 = *reinterpret_cast<const ulonglong2*>(br + 64);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint64_t a2 = dup2(av[i]);
                ffma2(acc[i][0], a2, b0.x);
                ffma2(acc[i][1], a2, b0.y);
                ffma2(acc[i][2], a2, b1.x);
                ffma2(acc[i][3], a2, b1.y);
            }
        }
        if (more) put(buf ^ 1u);
        __syncthreads();
        buf ^= 1u;
    }

    auto out4 = [&](uint32_t row, uint32_t col, float4 v) {
        if (row >= m || col >= n) return;
        float* p = c + (size_t)row * n + col;
        float x[4] = {v.x, v.y, v.z, v.w};
        const bool vec = (n & 3u) == 0 && ((uintptr_t)c & 15u) == 0;
        if (flags & GEMM_SILU)
#pragma unroll
            for (int e = 0; e < 4; e++) x[e] = x[e] / (1.0f + expf(-x[e]));
        if (vec) {
            if (flags & GEMM_ADD) {
                const float4 o = *reinterpret_cast<const float4*>(p);
                x[0] = o.x + x[0]; x[1] = o.y + x[1]; x[2] = o.z + x[2]; x[3] = o.w + x[3];
            }
            *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (col + e < n) p[e] = (flags & GEMM_ADD) ? p[e] + x[e] : x[e];
        }
    };
    auto pair = [](uint64_t v) { return make_float2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32))); };
    if (ks == 1) {
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float2 lo = pair(acc[i][2 * h]), hi = pair(acc[i][2 * h + 1]);
                out4(m0 + ty * 8 + i, n0 + h * 64 + tx * 4, make_float4(lo.x, lo.y, hi.x, hi.y));
            }
        return;
    }
    // the loop's last barrier has let every thread finish reading the tiles the partial overwrites
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 lo = pair(acc[i][2 * h]), hi = pair(acc[i][2 * h + 1]);
            *reinterpret_cast<float4*>(&sm.red[ty * 8 + i][h * 64 + tx * 4]) = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    cluster.sync();
    const uint32_t rows_per = (BM + ks - 1) / ks;
    for (uint32_t e = t; e < rows_per * (BN / 4); e += THREADS) {
        const uint32_t row = rank * rows_per + e / (BN / 4), col = (e % (BN / 4)) * 4;
        if (row >= BM || m0 + row >= m) break;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t r = 0; r < ks; r++) {
            const float4 p = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&sm.red[row][col], r));
            s.x += p.x; s.y += p.y; s.z += p.z; s.w += p.w;
        }
        out4(m0 + row, n0 + col, s);
    }
    cluster.sync();   // nobody leaves while a peer may still read its partial
}

// ---- m == 1
constexpr int GV_WARPS = 8;
__global__ void __launch_bounds__(GV_WARPS * 32)
gemv_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, uint32_t n, uint32_t k, uint32_t flags, uint32_t vec) {
    pdl_wait();
    pdl_trigger();
    const uint32_t lane = threadIdx.x & 31, n_warps = gridDim.x * GV_WARPS;
    for (uint32_t r = blockIdx.x * GV_WARPS + (threadIdx.x >> 5); r < n; r += n_warps) {
        const float* p = w + (size_t)r * k;
        float s = 0.0f;
        if (vec) {
#pragma unroll 8
            for (uint32_t i = lane * 4; i < k; i += 128) {
                const float4 a = __ldcs(reinterpret_cast<const float4*>(p + i)), b = __ldg(reinterpret_cast<const float4*>(x + i));
                s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
            }
        } else {
            for (uint32_t i = lane; i < k; i += 32) s = fmaf(p[i], x[i], s);
        }
        s = warp_sum(s);
        if (lane == 0) {
            if (flags & GEMM_SILU) s = s / (1.0f + expf(-s));
            y[r] = (flags & GEMM_ADD) ? y[r] + s : s;
        }
    }
}

}  // namespace ntf32

int launch_gemm_f32_nt(cudaStream_t st, const float* a, const float* wt, float* c, uint32_t m, uint32_t n, uint32_t k, uint32_t flags) {
    using namespace ntf32;
    if (m == 0 || n == 0) return AK_OK;
    const bool vec = (k & 3u) == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)wt % 16 == 0;
    if (m == 1 && (flags & GEMM_ALONE)) {
        const uint32_t ctas = cdiv(n, GV_WARPS), room = B200_SMS * 8;
        return launch_k(gemv_kernel, dim3(ctas < room ? ctas : room), dim3(GV_WARPS * 32), 0, st, NO_CLUSTER, a, wt, c, n, k, flags, (uint32_t)vec);
    }
    // Where a launch is short anyway the FMA pipe is quicker to the end of it (an SM's whole shared and tensor memory are set up for nothing). Four products of a
    // layer, this kernel / tensor cores, us, with 4, 128 and 1024 rows: 64-wide model 26 / 25, 32 / 43, 33 / 45; 128-wide 26.7 / 30.0, 38.5 / 42.7, 43.1 / 44.0
    // (2048 rows 57 / 45); 256-wide, of which only 256 x 256 is small, 30.5 / 29.8, 37.3 / 39.5, 72 / 50. Steps of a 128-wide model of 2 layers with
    // 8 sequences 88 / 101.
    const bool small = k <= 128 || (uint64_t)n * k <= 65536;
    if (vec && !small) return launch_gemm_f32_tc(st, a, wt, c, m, n, k, flags);
    // K is split so that one row tile occupies every SM, at most eight ways (a portable cluster), never less than 64 of K per CTA
    const uint32_t tn = cdiv(n, BN);
    uint32_t ks = B200_SMS / tn;
    if (ks > 8) ks = 8;
    if (ks > k / 64) ks = k / 64;
    if (ks < 1) ks = 1;
    const dim3 grid(tn, cdiv(m, BM), ks), cluster(1, 1, ks);
    if (vec) return launch_k(gemm_kernel<false>, grid, dim3(THREADS), 0, st, cluster, a, wt, c, m, n, k, flags);
    return launch_k(gemm_kernel<true>, grid, dim3(THREADS), 0, st, cluster, a, wt, c, m, n, k, flags);
}

}  // namespace ak
