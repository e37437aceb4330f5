// Tiling and stencil pieces of the stencil kernels (sm_100a).
//
// Every thread owns TWO adjacent columns of RPT rows: a tile is 64 columns
// wide, the x-neighbourhood of a thread's two columns on one row is five
// aligned float2 shared loads (columns j-4 .. j+5), and the z-stencils come
// from a window of RPT + 2K rows.  Halo boxes arrive by TMA.
// The forward carries stresses (sxx = L2M ex + L ez, szz = L ex + L2M ez,
// sxz = 2 M es) instead of strains and the adjoint the buoyancy-scaled
// velocities P = B U_a, Q = B V_a: exact changes of variables that remove
// the halo transforms from the interior tiles.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace stfwi {

constexpr int TX4 = 64;               // tile width: 32 lanes x 2 columns
constexpr int XO4 = 4;                // x halo of the staged tile
constexpr int SW4 = TX4 + 2 * XO4;    // 72 floats = 288 B rows

// tiles of NW warps of RPT rows each
template <int FD, int RPT, int NW> struct G4 {
    static constexpr int K = FD / 2;
    static constexpr int TZH = RPT * NW;
    static constexpr int SH = TZH + 2 * K;
    static constexpr int SN = SH * SW4;
    static constexpr int W = RPT + 2 * K;
    static constexpr int S2 = al32_3(2 * SN), S3 = al32_3(3 * SN);
};

// rows per thread: every kernel is built for 1 and 2 (8- and 16-row tiles);
// a handle runs fwd_vel, fwd_str and adj_a on one tile height and adj_b on
// another, chosen by the autotuner (2 and 2 until it has run)
constexpr int RPT_MIN = 1, RPT_DEFAULT = 2;

// a[i] = f[j - 4 + i], i in [0, 10): the x-neighbourhood of columns j, j+1
__device__ __forceinline__ void xrow(float (&a)[10], const float *s, int q)
{
    const float2 *p = reinterpret_cast<const float2 *>(s + q - 4);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        const float2 t = p[m];
        a[2 * m] = t.x;
        a[2 * m + 1] = t.y;
    }
}

// x stencils at output column c of the pair from its neighbourhood a, with
// coefficients co(k) (both terms of a difference, or, transposed, A(k) of the
// + term and B(k) of the - term)
template <int FD, class C> __device__ __forceinline__ float a_dp(const float (&a)[10], int c, C co)
{
    float d = 0.f;
#pragma unroll
    for (int k = 1; k <= FD / 2; ++k) d += co(k) * (a[4 + c + k] - a[5 + c - k]);
    return d;
}
template <int FD, class C> __device__ __forceinline__ float a_dm(const float (&a)[10], int c, C co)
{
    float d = 0.f;
#pragma unroll
    for (int k = 1; k <= FD / 2; ++k) d += co(k) * (a[3 + c + k] - a[4 + c - k]);
    return d;
}
template <int FD, class CA, class CB> __device__ __forceinline__ float a_tdp(const float (&a)[10], int c, CA A, CB B)
{
    float d = 0.f;
#pragma unroll
    for (int k = 1; k <= FD / 2; ++k) {
        d += A(k) * a[4 + c - k];
        d -= B(k) * a[3 + c + k];
    }
    return d;
}
template <int FD, class CA, class CB> __device__ __forceinline__ float a_tdm(const float (&a)[10], int c, CA A, CB B)
{
    float d = 0.f;
#pragma unroll
    for (int k = 1; k <= FD / 2; ++k) {
        d += A(k) * a[5 + c - k];
        d -= B(k) * a[4 + c + k];
    }
    return d;
}

}  // namespace stfwi
