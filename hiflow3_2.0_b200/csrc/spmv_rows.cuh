// spmv_rows.cuh -- one 32-row chunk of a structured operator times a vector, by
// one warp, one row per lane: the row sums of the stencil layout (kernels.cuh) for the
// SpMV kernels and the streaming CG, and of the half stencil layout: its values for
// the SpMV kernels, whose FP64 one keeps half_row's steps in line, and half_row for
// the streaming CG.  gx(j) is the vector's entry j.
#pragma once

#include "common.cuh"
#include "kernels.cuh"

namespace b200 {

template <typename T, int W>
struct StencilVec;
template <>
struct StencilVec<double, 1> {
    using type = double;
    static __device__ __forceinline__ void load(const double *p, uint64_t pol, double *o) { o[0] = ld_stream(p, pol); }
};
template <>
struct StencilVec<float, 4> {
    using type = float4;
    static __device__ __forceinline__ void load(const float4 *p, uint64_t pol, float *o)
    {
        float4 v;
        asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
            : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
            : "l"(p), "l"(pol));
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        o[3] = v.w;
    }
};

template <typename T, int NB>
struct HalfRow;

template <int NB>
struct HalfRow<float, NB> {
    static constexpr int U = (NB - 1) / 2, GH = half_groups(NB);
    static __device__ __forceinline__ float4 ld(const float4 *p, uint64_t pol)
    {
        float4 v;
        asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
            : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
            : "l"(p), "l"(pol));
        return v;
    }
    // av[b][m]: value of row 32 c + lane at column offset center[b] + m - 1
    static __device__ __forceinline__ void values(const void *sh, const int (&cen)[NB], int c, int lane, int rows,
                                                  uint64_t pol, float (&av)[NB][3])
    {
        const float4 *__restrict__ hv = static_cast<const float4 *>(sh);
        const int r0 = c << 5, r = r0 + lane;
        float4 u[GH];
#pragma unroll
        for (int g = 0; g < GH; ++g) StencilVec<float, 4>::load(hv + ((size_t)c * GH + g) * 32 + lane, pol, &u[g].x);
#pragma unroll
        for (int ub = 0; ub < U; ++ub) {
            av[U + 1 + ub][0] = u[ub].x;
            av[U + 1 + ub][1] = u[ub].y;
            av[U + 1 + ub][2] = u[ub].z;
        }
        av[U][1] = u[0].w;
        av[U][2] = u[1].w;
        // (r, r - 1) is row r - 1's +1 entry: lane - 1's, or the previous chunk's last row
        float lm = __shfl_up_sync(0xffffffffu, u[1].w, 1);
        if (lane == 0) lm = r0 > 0 ? ld(hv + ((size_t)(c - 1) * GH + 1) * 32 + 31, pol).w : 0.f;
        av[U][0] = lm;
        // lower band b mirrors upper band U - 1 - b: (r, r + d + m - 1) is
        // row (r + d + m - 1)'s entry at slot 2 - m of that band
#pragma unroll
        for (int b = 0; b < U; ++b) {
            const int d = cen[b], ub = U - 1 - b, q = r + d;
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 g = q >= 0 ? ld(hv + ((size_t)(q >> 5) * GH + ub) * 32 + (q & 31), pol) : z;
            const int hq = lane == 0 ? r0 + d - 1 : r0 + 32 + d;
            const float4 h = ((lane == 0 || lane == 31) && hq >= 0 && hq < rows)
                                 ? ld(hv + ((size_t)(hq >> 5) * GH + ub) * 32 + (hq & 31), pol)
                                 : z;
            float left = __shfl_up_sync(0xffffffffu, g.z, 1);
            float right = __shfl_down_sync(0xffffffffu, g.x, 1);
            if (lane == 0) left = h.z;
            if (lane == 31) right = h.x;
            av[b][0] = left;
            av[b][1] = g.y;
            av[b][2] = right;
        }
    }
};

template <int NB>
struct HalfRow<double, NB> {
    static constexpr int U = (NB - 1) / 2, H = half_positions(NB);
    static __device__ __forceinline__ double at(const double *hv, int q, int p, uint64_t pol)
    {
        return q >= 0 ? ld_keep(hv + ((size_t)(q >> 5) * H + p) * 32 + (q & 31), pol) : 0.0;
    }
    // the three values of band b of row 32 c + lane
    static __device__ __forceinline__ void band(const double *__restrict__ hv, int d, int c, int lane, int b,
                                                uint64_t pol, uint64_t pol_own, double (&a)[3])
    {
        const int r = (c << 5) + lane;
        const double *own = hv + (size_t)c * H * 32 + lane;
        if (b > U) {
#pragma unroll
            for (int m = 0; m < 3; ++m) a[m] = ld_stream(own + 32 * (2 + 3 * (b - U - 1) + m), pol_own);
        } else if (b == U) {
            a[0] = at(hv, r - 1, 1, pol);
            a[1] = ld_stream(own, pol_own);
            a[2] = ld_stream(own + 32, pol_own);
        } else {
            const int q = r + d, p = 2 + 3 * (U - 1 - b);
            a[0] = at(hv, q - 1, p + 2, pol);
            a[1] = at(hv, q, p + 1, pol);
            a[2] = at(hv, q + 1, p, pol);
        }
    }
};

// Full layout.  FP32 loads the whole row's values first, FP64 works in groups of
// three bands.  Columns outside [0, last] belong to zero entries and are clamped.
template <typename T, int NB, class GX>
__device__ __forceinline__ T stencil_row(const typename StencilVec<T, stencil_group<T>()>::type *__restrict__ sv,
                                         const int (&cen)[NB], int c, int lane, int last, uint64_t pol_v, GX gx)
{
    constexpr int W = stencil_group<T>();
    constexpr int L = 3 * NB, G = (L + W - 1) / W;
    const int r0 = c << 5, r = r0 + lane;
    const int he = lane == 0 ? r0 - 1 : r0 + 32;
    const bool edge = lane == 0 || lane == 31;
    const auto *v = sv + (size_t)c * (32 * G) + lane;
    T s = T(0);
    if constexpr (W > 1) {
        // FP32: the whole row's values first (G vector loads), then the bands
        T a[G * W];
#pragma unroll
        for (int g = 0; g < G; ++g) StencilVec<T, W>::load(v + 32 * g, pol_v, a + W * g);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const int d = cen[b];
            const T w = gx(min(max(r + d, 0), last));
            const T h = edge ? gx(min(max(he + d, 0), last)) : T(0);
            T left = __shfl_up_sync(0xffffffffu, w, 1);
            T right = __shfl_down_sync(0xffffffffu, w, 1);
            if (lane == 0) left = h;
            if (lane == 31) right = h;
            s += a[3 * b] * left;
            s += a[3 * b + 1] * w;
            s += a[3 * b + 2] * right;
        }
    } else {
        // FP64: groups of three bands, their value loads and gathers issued together
#pragma unroll
        for (int b0 = 0; b0 < NB; b0 += 3) {
            T a[9], w[3], h[3];
#pragma unroll
            for (int bb = 0; bb < 3; ++bb)
#pragma unroll
                for (int m = 0; m < 3; ++m) StencilVec<T, W>::load(v + 32 * (3 * (b0 + bb) + m), pol_v, a + 3 * bb + m);
#pragma unroll
            for (int bb = 0; bb < 3; ++bb) {
                const int d = cen[b0 + bb];
                w[bb] = gx(min(max(r + d, 0), last));
                h[bb] = edge ? gx(min(max(he + d, 0), last)) : T(0);
            }
#pragma unroll
            for (int bb = 0; bb < 3; ++bb) {
                T left = __shfl_up_sync(0xffffffffu, w[bb], 1);
                T right = __shfl_down_sync(0xffffffffu, w[bb], 1);
                if (lane == 0) left = h[bb];
                if (lane == 31) right = h[bb];
                s += a[3 * bb] * left;
                s += a[3 * bb + 1] * w[bb];
                s += a[3 * bb + 2] * right;
            }
        }
    }
    return s;
}

// Half layout, FP64: groups of three bands, their value loads and gathers issued
// together (register pressure of one group, not of the row); identity rows use
// their diagonal alone.  spmv_half_kernel (spmv.cu) holds the same steps in line and
// must change with them: a solve's residual is formed by either.
template <int NB, class GX>
__device__ __forceinline__ double half_row(const double *__restrict__ hv, const unsigned *__restrict__ mask,
                                           const int (&cen)[NB], int c, int lane, int last, uint64_t pol, uint64_t pol_own,
                                           bool prefetch, GX gx)
{
    constexpr int U = (NB - 1) / 2;
    const int r0 = c << 5, r = r0 + lane;
    const int he = lane == 0 ? r0 - 1 : r0 + 32;
    const bool edge = lane == 0 || lane == 31;
    // FP64: groups of three bands, their value loads and gathers
    // issued together (register pressure of one group, not of the row)
    if (prefetch) {   // the chunk's own value lines into L2 before the first group's loads
        constexpr int kLines = HalfRow<double, NB>::H * 32 * 8 / 128;
        if (lane < kLines) {
            const char *q = reinterpret_cast<const char *>(hv +
                                                           (size_t)c * HalfRow<double, NB>::H * 32) + 128 * lane;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
        }
    }
    const bool ident = (__ldg(mask + c) >> lane) & 1u;
    double s = 0.0;
#pragma unroll
    for (int b0 = 0; b0 < NB; b0 += 3) {
        double a[3][3], w[3], h[3];
#pragma unroll
        for (int bb = 0; bb < 3; ++bb) {
            const int b = b0 + bb, d = cen[b];
            HalfRow<double, NB>::band(hv, d, c, lane, b, pol, pol_own, a[bb]);
            if (ident) {
                // identity row: its upper slots serve the neighbours; off-diagonals are zero
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    if (b != U || m != 1) a[bb][m] = 0.0;
            }
        }
#pragma unroll
        for (int bb = 0; bb < 3; ++bb) {
            const int d = cen[b0 + bb];
            w[bb] = gx(min(max(r + d, 0), last));
            h[bb] = edge ? gx(min(max(he + d, 0), last)) : 0.0;
        }
#pragma unroll
        for (int bb = 0; bb < 3; ++bb) {
            double left = __shfl_up_sync(0xffffffffu, w[bb], 1);
            double right = __shfl_down_sync(0xffffffffu, w[bb], 1);
            if (lane == 0) left = h[bb];
            if (lane == 31) right = h[bb];
            s += a[bb][0] * left;
            s += a[bb][1] * w[bb];
            s += a[bb][2] * right;
        }
    }
    return s;
}

}  // namespace b200
