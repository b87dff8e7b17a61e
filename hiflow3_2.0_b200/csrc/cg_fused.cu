// cg_fused.cu -- a whole CG solve in one cooperative launch, for structured
// operators whose vectors fit the registers of one CTA per SM.
//
// Three launches per iteration (product, update, direction) cost about 15 us
// at any small size: launches and reduction tails, with the operator and the
// vectors in L1 and L2.  Here the CTAs keep their rows' x, r, p and Jacobi
// scaling in registers for the whole solve and meet twice per iteration in a
// grid sum (grid_gather.cuh): p.Ap, then ||r||^2 and r.z.  No third meeting and
// no fence is needed for the vector exchange: a row's owner writes z with the
// epoch of the sum behind it as one 16-byte word, a reader polls the words it
// gathers, and forms p_new = beta p + z at each of them from its own copy of p
// there, with the same rounding as the owner (cg_direction's).  Where those
// copies do not fit the registers (3-D, four rows per thread) the owner sends
// p_new instead, one L2 round trip later.
//   Rows are dealt out in 32-row chunks, E per warp; a chunk gathers one word
// per band and lane, the two columns beyond the chunk of all bands come in one
// load (lane b the left one of band b, lane 16 + b the right one).  Values stay
// in registers where they fit, else they are re-read through L1, which holds
// up to about 33 MB of them over the GPU.
//   Bound by the two grid sums and one L2 round trip of the gathers.  Per
// iteration, launch per step -> here: 2-D 33^2 15.1 -> 3.4 us (up to 7 where the device
// spreads its three CTAs), 256^2 16.5 -> 7-8, 512^2 19.8 -> 11; 3-D 41^3 17.2 -> 9.7,
// 64^3 23.4 -> 16.7 (FP32 19.3 -> 14.5).
#include "b200la.h"
#include "b200la_internal.h"
#include "grid_gather.cuh"
#include "spmv_rows.cuh"

#include <algorithm>
#include <cstdlib>

using namespace b200;

namespace {

constexpr int kCgThreads = 512;
constexpr int kCgMaxRows = 4;   // rows per thread
constexpr int kCgStream = -1;   // (instead of a number of rows) the vectors stay in memory

struct CgFusedArgs {
    const void *val;          // st_val, or sh_val (half layout)
    const unsigned *mask;     // half layout: identity rows
    int cen[kMaxBands];
    int n;
    const void *b, *invd;     // invd null: no preconditioner
    void *x;
    unsigned char *rows;      // a 16-byte word per row
    // vectors in memory (cg_stream_kernel)
    void *r, *p;
    int per_warp, r_shared, l2hint;
    int maxits, hist_len;
    double abstol, reltol, divtol;
    double *hist;
    DevState *out;            // host mirror: the final state; pad0 set if a wait ran out
    unsigned char *gmem;
    int *err;
    int first;   // number of a wait's first poll (gather_first)
};

// The 3 NB values of row 32 c + lane in (band, column) order.
template <typename T, int NB, bool HALF>
__device__ __forceinline__ void row_values(const CgFusedArgs &a, int c, int lane, T (&v)[3 * NB])
{
    if constexpr (sizeof(T) == 4) {
        constexpr int G = (3 * NB + 3) / 4;
        const float4 *q = static_cast<const float4 *>(a.val) + (size_t)c * (32 * G) + lane;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float4 w = __ldg(q + 32 * g);
            const float e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (4 * g + k < 3 * NB) v[4 * g + k] = e[k];
        }
    } else if constexpr (!HALF) {
        const double *q = static_cast<const double *>(a.val) + (size_t)c * (32 * 3 * NB) + lane;
#pragma unroll
        for (int k = 0; k < 3 * NB; ++k) v[k] = __ldg(q + 32 * k);
    } else {
        // diagonal, +1 and upper bands of the row; the lower half from the rows
        // that own it; identity rows keep their diagonal alone
        constexpr int U = (NB - 1) / 2, H = half_positions(NB);
        const double *hv = static_cast<const double *>(a.val), *own = hv + (size_t)c * H * 32 + lane;
        const int r = (c << 5) + lane;
        const bool ident = (__ldg(a.mask + c) >> lane) & 1u;
        auto at = [&](int q, int p) -> double {
            return q >= 0 && !ident ? __ldg(hv + ((size_t)(q >> 5) * H + p) * 32 + (q & 31)) : 0.0;
        };
#pragma unroll
        for (int b = 0; b < U; ++b) {
            const int q = r + a.cen[b], p = 2 + 3 * (U - 1 - b);
            v[3 * b] = at(q - 1, p + 2);
            v[3 * b + 1] = at(q, p + 1);
            v[3 * b + 2] = at(q + 1, p);
        }
        v[3 * U] = at(r - 1, 1);
        v[3 * U + 1] = __ldg(own);
        v[3 * U + 2] = ident ? 0.0 : __ldg(own + 32);
#pragma unroll
        for (int k = 0; k < 3 * U; ++k) v[3 * (U + 1) + k] = ident ? 0.0 : __ldg(own + 32 * (2 + k));
    }
}

// sum_j a_ij g(j) of the warp's chunk, products in column order; w[b] holds g
// at the band centres of the lane's row and h the lane's column beyond the chunk.
template <typename T, int NB>
__device__ __forceinline__ T row_sum(const T (&v)[3 * NB], const T (&w)[NB], T h, int lane)
{
    T s = T(0);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        T left = __shfl_up_sync(0xffffffffu, w[b], 1), right = __shfl_down_sync(0xffffffffu, w[b], 1);
        const T hl = __shfl_sync(0xffffffffu, h, b), hr = __shfl_sync(0xffffffffu, h, 16 + b);
        if (lane == 0) left = hl;
        if (lane == 31) right = hr;
        s += v[3 * b] * left;
        s += v[3 * b + 1] * w[b];
        s += v[3 * b + 2] * right;
    }
    return s;
}

template <typename T, int NB, bool HALF, int E>
__global__ void __launch_bounds__(kCgThreads, 1) cg_fused_kernel(CgFusedArgs a)
{
    constexpr bool kKeep = E * 3 * NB * (int)sizeof(T) <= 144;   // the values stay in registers
    constexpr bool kTrack = E * (NB + 1) * (int)sizeof(T) <= 160;   // and p at the gathered columns
    __shared__ typename GridGather<kCgThreads>::Shared sh;
    GridGather<kCgThreads> gg(a.gmem, sh, a.err, a.first);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = a.n, last = n - 1, nch = (n + 31) >> 5;
    const int c0 = (blockIdx.x * (kCgThreads / 32) + warp) * E;   // the warp's chunks
    const T *b = static_cast<const T *>(a.b), *invd = static_cast<const T *>(a.invd);
    T *x = static_cast<T *>(a.x);
    // the column beyond the chunk that this lane loads
    int beyond = 0;
#pragma unroll
    for (int q = 0; q < NB; ++q)
        if ((lane & 15) == q) beyond = a.cen[q] + (lane < 16 ? -1 : 32);
    auto clamp = [&](int j) { return min(max(j, 0), last); };
    T xr[E], rr[E], pr[E], dr[E], keep[kKeep ? E : 1][3 * NB];
    auto values = [&](int e, T (&v)[3 * NB]) {
        if constexpr (kKeep) {
#pragma unroll
            for (int k = 0; k < 3 * NB; ++k) v[k] = keep[e][k];
        } else {
            row_values<T, NB, HALF>(a, c0 + e, lane, v);
        }
    };
    // the words of the columns that chunk c gathers, once they carry `epoch`
    auto gather = [&](int c, T (&w)[NB], T &h) {
        const int r = 32 * c + lane;
        for (long long i = gg.first;; ++i) {
            bool ready = true;
#pragma unroll
            for (int q = 0; q <= NB; ++q) {
                double v;
                unsigned long long t;
                ld_word(a.rows + 16 * (size_t)clamp(q < NB ? r + a.cen[q] : 32 * c + beyond), v, t);
                (q < NB ? w[q < NB ? q : 0] : h) = (T)v;
                ready &= t == gg.epoch;
            }
            if (__all_sync(0xffffffffu, ready) || __any_sync(0xffffffffu, gg.stop(i))) return;
        }
    };
    T pc[kTrack ? E : 1][NB + 1];   // p at the gathered columns
    // r = b - A x, z = M^-1 r (cg.cc:200-214)
    double sum[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int c = c0 + e, r = 32 * c + lane;
        xr[e] = rr[e] = pr[e] = dr[e] = T(0);
        if constexpr (kTrack) {
#pragma unroll
            for (int q = 0; q <= NB; ++q) pc[e][q] = T(0);
        }
        if (c >= nch) continue;
        T v[3 * NB], w[NB];
        row_values<T, NB, HALF>(a, c, lane, v);
        if constexpr (kKeep) {
#pragma unroll
            for (int k = 0; k < 3 * NB; ++k) keep[e][k] = v[k];
        }
#pragma unroll
        for (int q = 0; q < NB; ++q) w[q] = x[clamp(r + a.cen[q])];
        const T s = row_sum<T, NB>(v, w, x[clamp(32 * c + beyond)], lane);
        if (r < n) {
            xr[e] = x[r];
            rr[e] = b[r] - s;
            dr[e] = invd ? invd[r] : T(1);
            const T z = rr[e] * dr[e];
            if constexpr (kTrack) st_word(a.rows + 16 * (size_t)r, (double)z, gg.epoch + 1);
            sum[0] += (double)(rr[e] * rr[e]);
            sum[1] += (double)(rr[e] * z);
        }
    }
    gg.template publish<2>(sum);
    gg.template total<2>(sum);
    // IterateControl::Check (iterate_control.cc:84-110); every CTA decides alike
    const double res0 = sqrt(sum[0]);
    auto check = [&](int step, double v) -> int {
        if (v < a.abstol) return kSuccessAbs;
        if (v < a.reltol * res0) return kSuccessRel;
        if (v > a.divtol * res0) return kFailDiv;
        if (step >= a.maxits) return kFailMaxits;
        return kIterate;
    };
    const bool scribe = blockIdx.x == 0 && threadIdx.x == 0;
    int it = 0, status = check(0, res0);
    double res = res0, rho = sum[1], beta = 0.0, alpha = 0.0;
    if (scribe && a.hist && a.hist_len > 0) a.hist[0] = res0;
    while (status == kIterate) {
        // p = beta p + z; Ap; p.Ap (cg.cc:241, 219-220)
        const T bt = (T)beta;
        T ap[E];
        double pap[1] = {0.0};
        if constexpr (!kTrack) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int r = 32 * (c0 + e) + lane;
                pr[e] = fma(bt, pr[e], rr[e] * dr[e]);
                if (r < n) st_word(a.rows + 16 * (size_t)r, (double)pr[e], gg.epoch);
            }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int c = c0 + e, r = 32 * c + lane;
            ap[e] = T(0);
            if (c >= nch) continue;
            T v[3 * NB], w[NB], h;
            gather(c, w, h);
            values(e, v);
            if constexpr (kTrack) {
#pragma unroll
                for (int q = 0; q < NB; ++q) w[q] = pc[e][q] = fma(bt, pc[e][q], w[q]);
                h = pc[e][NB] = fma(bt, pc[e][NB], h);
                pr[e] = fma(bt, pr[e], rr[e] * dr[e]);
            }
            ap[e] = row_sum<T, NB>(v, w, h, lane);
            if (r < n) pap[0] += (double)(pr[e] * ap[e]);
        }
        gg.template publish<1>(pap);
        gg.template total<1>(pap);
        alpha = rho / pap[0];
        const T al = (T)alpha;
        // x += alpha p; r -= alpha Ap; ||r||, r.z (cg.cc:221-240)
        double v[2] = {0.0, 0.0};
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int r = 32 * (c0 + e) + lane;
            if (r >= n) continue;
            xr[e] += al * pr[e];
            rr[e] -= al * ap[e];
            const T z = rr[e] * dr[e];
            if constexpr (kTrack) st_word(a.rows + 16 * (size_t)r, (double)z, gg.epoch + 1);
            v[0] += (double)(rr[e] * rr[e]);
            v[1] += (double)(rr[e] * z);
        }
        gg.template publish<2>(v);
        gg.template total<2>(v);
        ++it;
        res = sqrt(v[0]);
        status = check(it, res);
        if (scribe && a.hist && it < a.hist_len) a.hist[it] = res;
        beta = v[1] / rho;
        rho = v[1];
    }
    gg.close();
    if (gg.failed() && threadIdx.x == 0) a.out->pad0 = 1.0;   // by whichever CTA gave up
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int r = 32 * (c0 + e) + lane;
        if (r < n) x[r] = xr[e];
    }
    if (scribe) {
        a.out->iter = it;
        a.out->status = status;
        a.out->res = res;
        a.out->res0 = res0;
        a.out->rr = res * res;
        a.out->rho = rho;
        a.out->beta = beta;
        a.out->alpha = alpha;
    }
}

// The same solve for operators beyond the registers: a persistent grid of one
// 1,024-thread CTA per SM whose warps own every grid-stride chunk of 32 rows.
// A p (and r, where both fit) stay in shared memory between the phases, so an
// iteration reads the operator, p, the scaling and x once each beside the gathers,
// and writes x and p; the CTAs meet in two grid sums and, before p is gathered, a
// grid barrier.  With a launch per step the same product left 15-23 us an
// iteration to the two vector kernels, their reduction tails and the gaps between
// launches.  Per iteration, launch per step -> here, in one call: 2-D 600^2 FP64
// 20.2 -> 13.8 us, 1000^2 29.4 -> 20.4; 3-D 70^3 25.2 -> 21.2, 100^3 50.5 -> 44.6 (FP32
// 35.4 -> 25.9), 108^3 59.1 -> 57.7, 128^3 88.5 -> 88.7 (FP32 57.2 -> 50.5).
constexpr int kStreamThreads = 1024;
constexpr size_t kStreamSmem = 160 * 1024;   // the rest of the 228 KB is L1 for the gathers
constexpr size_t kStreamAp = 128 * 1024;     // A p beyond this: launch per step (no gain left at 2.4 million FP64 rows)

template <typename T, int NB, bool HALF>
__global__ void __launch_bounds__(kStreamThreads, 1) cg_stream_kernel(CgFusedArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ typename GridGather<kStreamThreads>::Shared sh;
    GridGather<kStreamThreads> gg(a.gmem, sh, a.err, a.first);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = a.n, last = n - 1, nch = (n + 31) >> 5;
    const int K = a.per_warp, c0 = blockIdx.x * (kStreamThreads / 32) + warp, cs = gridDim.x * (kStreamThreads / 32);
    const T *b = static_cast<const T *>(a.b), *invd = static_cast<const T *>(a.invd);
    T *x = static_cast<T *>(a.x), *p = static_cast<T *>(a.p);
    T *aps = reinterpret_cast<T *>(s_raw) + tid;                          // A p of the thread's k-th row at 1024 k
    T *rs = a.r_shared ? aps + (size_t)K * kStreamThreads : nullptr;      // r likewise
    auto r_at = [&](int k, int r) -> T & { return rs ? rs[(size_t)k * kStreamThreads] : static_cast<T *>(a.r)[r]; };
    const uint64_t pol = l2_policy(0), pol_v = l2_policy(a.l2hint & 4 ? 1 : 0), pol_own = l2_policy(a.l2hint & 8 ? 1 : 0);
    int cen[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) cen[q] = a.cen[q];
    auto product = [&](int c, const T *v) -> T {
        auto gx = [&](int j) -> T { return v[j]; };
        if constexpr (HALF)
            return half_row<NB>(static_cast<const double *>(a.val), a.mask, cen, c, lane, last, pol, pol_own,
                                (a.l2hint & 16) != 0, gx);
        else
            return stencil_row<T, NB>(static_cast<const typename StencilVec<T, stencil_group<T>()>::type *>(a.val), cen, c,
                                      lane, last, pol_v, gx);
    };
    // The value lines of the warp's first two chunks come into L2 while the CTAs
    // wait for one another before the product (FP32 100^3 29.0 -> 26.1 us an
    // iteration, 128^3 52.8 -> 50.7, in one call).  Not those of the half layout, whose second
    // readings they push out of L2 (FP64 128^3 89 -> 97 us).
    constexpr int kGroup = stencil_group<T>();
    constexpr int kChunkBytes = 32 * (int)sizeof(T) * kGroup * ((3 * NB + kGroup - 1) / kGroup);
    auto ahead = [&](int k) {
        const int c = c0 + k * cs;
        if (HALF || c >= nch) return;
        const char *q = static_cast<const char *>(a.val) + (size_t)c * kChunkBytes;
        for (int o = 128 * lane; o < kChunkBytes; o += 128 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + o));
    };
    // r = b - A x, p = z = M^-1 r (cg.cc:200-214)
    double sum[2] = {0.0, 0.0};
    for (int k = 0, c = c0; c < nch; ++k, c += cs) {
        const int r = 32 * c + lane;
        const T s = product(c, x);
        if (r >= n) continue;
        const T rv = b[r] - s, z = invd ? rv * invd[r] : rv;
        r_at(k, r) = rv;
        p[r] = z;
        sum[0] += (double)(rv * rv);
        sum[1] += (double)(rv * z);
    }
    gg.template publish<2>(sum);
    gg.template total<2>(sum);
    const double res0 = sqrt(sum[0]);
    auto check = [&](int step, double v) -> int {
        if (v < a.abstol) return kSuccessAbs;
        if (v < a.reltol * res0) return kSuccessRel;
        if (v > a.divtol * res0) return kFailDiv;
        if (step >= a.maxits) return kFailMaxits;
        return kIterate;
    };
    const bool scribe = blockIdx.x == 0 && tid == 0;
    int it = 0, status = check(0, res0);
    double res = res0, rho = sum[1], beta = 0.0, alpha = 0.0;
    if (scribe && a.hist && a.hist_len > 0) a.hist[0] = res0;
    while (status == kIterate) {
        ahead(1);
        gg.sync();   // p
        // Ap = A p; alpha = rho / p.Ap (cg.cc:219-220)
        double pap[1] = {0.0};
        for (int k = 0, c = c0; c < nch; ++k, c += cs) {
            const int r = 32 * c + lane;
            const T s = product(c, p);
            aps[(size_t)k * kStreamThreads] = s;
            if (r < n) pap[0] += (double)(p[r] * s);
        }
        gg.template publish<1>(pap);
        gg.template total<1>(pap);
        alpha = rho / pap[0];
        const T al = (T)alpha;
        // r -= alpha Ap; ||r||, r.z (cg.cc:222-240)
        double v[2] = {0.0, 0.0};
#pragma unroll 4
        for (int k = 0; k < K; ++k) {
            const int r = 32 * (c0 + k * cs) + lane;
            if (r >= n) continue;
            const T rv = r_at(k, r) - al * aps[(size_t)k * kStreamThreads], z = invd ? rv * __ldg(invd + r) : rv;
            r_at(k, r) = rv;
            v[0] += (double)(rv * rv);
            v[1] += (double)(rv * z);
        }
        gg.template publish<2>(v);
        // x += alpha p (cg.cc:221) while the sums travel
#pragma unroll 4
        for (int k = 0; k < K; ++k) {
            const int r = 32 * (c0 + k * cs) + lane;
            if (r < n) x[r] += al * p[r];
        }
        ahead(0);
        gg.template total<2>(v);
        ++it;
        res = sqrt(v[0]);
        status = check(it, res);
        if (scribe && a.hist && it < a.hist_len) a.hist[it] = res;
        if (status != kIterate) break;
        beta = v[1] / rho;
        rho = v[1];
        // p = beta p + z (cg.cc:241)
        const T bt = (T)beta;
#pragma unroll 4
        for (int k = 0; k < K; ++k) {
            const int r = 32 * (c0 + k * cs) + lane;
            if (r >= n) continue;
            const T rv = r_at(k, r);
            p[r] = fma(bt, p[r], invd ? rv * __ldg(invd + r) : rv);
        }
    }
    gg.close();
    if (gg.failed() && threadIdx.x == 0) a.out->pad0 = 1.0;   // by whichever CTA gave up
    if (scribe) {
        a.out->iter = it;
        a.out->status = status;
        a.out->res = res;
        a.out->res0 = res0;
        a.out->rr = res * res;
        a.out->rho = rho;
        a.out->beta = beta;
        a.out->alpha = alpha;
    }
}

template <typename T, int NB, bool HALF>
cudaError_t launch_stream(const CgFusedArgs &a, int grid, cudaStream_t st)
{
    const size_t sm = (size_t)a.per_warp * kStreamThreads * sizeof(T) * (a.r_shared ? 2 : 1);
    cudaError_t e = cudaFuncSetAttribute(cg_stream_kernel<T, NB, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kStreamSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = kStreamThreads;
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, cg_stream_kernel<T, NB, HALF>, a);
}

template <typename T, int NB, bool HALF, int E>
cudaError_t launch(const CgFusedArgs &a, int grid, cudaStream_t st)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = kCgThreads;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, cg_fused_kernel<T, NB, HALF, E>, a);
}

template <typename T, int NB, bool HALF>
cudaError_t launch_rows(const CgFusedArgs &a, int rows, int grid, cudaStream_t st)
{
    switch (rows) {
    case kCgStream: return launch_stream<T, NB, HALF>(a, grid, st);
    case 1: return launch<T, NB, HALF, 1>(a, grid, st);
    case 2: return launch<T, NB, HALF, 2>(a, grid, st);
    default: return launch<T, NB, HALF, 4>(a, grid, st);
    }
}

}  // namespace

// chunks per warp of the streaming form
static size_t stream_per_warp(const b200la_ctx *ctx, int n)
{
    const size_t warps = (size_t)gather_ctas(ctx->num_sms) * (kStreamThreads / 32);
    return ((size_t)(n + 31) / 32 + warps - 1) / warps;
}

// Rows per thread of the one-launch solve of A (or kCgStream), 0 where it does not run: an
// operator without the stencil layouts, or A p beyond shared memory (2.4 million
// rows in FP64, 4.8 in FP32).
// B200LA_CG_FUSED=0 turns it off, and so do the switches that ask for a form
// of the launch-per-step loop.
int cg_fused_rows(const b200la_ctx *ctx, const b200la_csr *A)
{
    const char *e = std::getenv("B200LA_CG_FUSED");
    if ((e && std::atoi(e) == 0) || std::getenv("B200LA_GRAPH_LOOP") || std::getenv("B200LA_NOGRAPH")) return 0;
    if (!ctx->cooperative || A->n < 1 || A->n != A->m || !A->st_use || (A->st_nb != 3 && A->st_nb != 9)) return 0;
    const bool half = A->sh_use && A->sh_val;
    if (half ? A->dtype != B200LA_F64 : !A->st_val) return 0;
    const size_t es = A->dtype == B200LA_F64 ? 8 : 4;
    const long long cap = (long long)gather_ctas(ctx->num_sms) * kCgThreads;
    for (int rows = 1; rows <= kCgMaxRows; rows *= 2)
        if (A->n <= cap * rows) return rows;
    return stream_per_warp(ctx, A->n) * kStreamThreads * es <= kStreamAp ? kCgStream : 0;
}

// The whole solve; the final state stands in ctx->st_host once the stream has
// passed it (and counts only if the error flag is clear then).  An error means that
// nothing was launched; cudaErrorCooperativeLaunchTooLarge where the CTAs would not
// all be resident, cudaErrorMemoryAllocation for want of the row words.  The row words are
// the context's own and nothing else is written there.
cudaError_t cg_fused_run(b200la_ctx *ctx, const b200la_csr *A, const void *invd, const void *b, void *x, void *r,
                         void *p, const b200la_control *ctl, double *hist, int hist_len, int rows)
{
    const bool half = A->sh_use && A->sh_val;
    if (rows > 0 && !ctx->rows) {
        const size_t bytes = 16 * (size_t)kGatherMaxCtas * kCgThreads * kCgMaxRows;
        cudaError_t e = cudaMalloc(&ctx->rows, bytes);
        if (e == cudaSuccess && (e = cudaMemsetAsync(ctx->rows, 0, bytes, ctx->stream)) != cudaSuccess) {
            cudaFree(ctx->rows);
            ctx->rows = nullptr;
        }
        if (e != cudaSuccess) return e;
        ctx->rows_bytes = bytes;
    }
    CgFusedArgs a;
    a.val = half ? A->sh_val : A->st_val;
    a.mask = A->sh_mask;
    for (int q = 0; q < kMaxBands; ++q) a.cen[q] = q < A->st_nb ? A->st_union[3 * q + 1] : 0;
    a.n = A->n;
    a.b = b;
    a.invd = invd;
    a.x = x;
    a.rows = static_cast<unsigned char *>(ctx->rows);
    a.maxits = ctl->maxits;
    a.abstol = ctl->abstol;
    a.reltol = ctl->reltol;
    a.divtol = ctl->divtol;
    a.hist = hist;
    a.hist_len = hist_len;
    a.out = ctx->st_host;
    a.out->pad0 = 0.0;
    a.gmem = ctx->gather;
    a.err = ctx->dev_err;
    a.first = gather_first();
    a.r = r;
    a.p = p;
    a.per_warp = (int)stream_per_warp(ctx, A->n);
    a.r_shared = 2 * (size_t)a.per_warp * kStreamThreads * (A->dtype == B200LA_F64 ? 8 : 4) <= kStreamSmem;
    a.l2hint = A->l2hint;
    const int grid = rows > 0 ? (A->n + kCgThreads * rows - 1) / (kCgThreads * rows)
                              : gather_ctas(ctx->num_sms);
    if (A->dtype == B200LA_F32)
        return A->st_nb == 3 ? launch_rows<float, 3, false>(a, rows, grid, ctx->stream)
                             : launch_rows<float, 9, false>(a, rows, grid, ctx->stream);
    if (half)
        return A->st_nb == 3 ? launch_rows<double, 3, true>(a, rows, grid, ctx->stream)
                             : launch_rows<double, 9, true>(a, rows, grid, ctx->stream);
    return A->st_nb == 3 ? launch_rows<double, 3, false>(a, rows, grid, ctx->stream)
                         : launch_rows<double, 9, false>(a, rows, grid, ctx->stream);
}
