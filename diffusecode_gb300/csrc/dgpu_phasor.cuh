// Phasors of exact 64-bit phases on CUDA cores by table-driven angle
// addition (Tang's table-driven method for elementary functions): a phase
// ph (2^64 = one turn) plus PH_ROUND splits into
//   * its top 10 bits, the nearest of PH_TAB table angles 2 pi j / 1024,
//     whose exp(i angle) the table holds (FP64 sincospi rounded to FP32);
//   * the next 23 bits less 2^22, the remainder d in units of PH_KAPPA
//     (|d| <= pi / 1024 rad, resolution 2 pi 2^-33, rounded to nearest),
// and exp(i d) = 1 - d^2/2 + i d (1 - d^2/6) to within 4e-12.
#pragma once
#include <stdint.h>

#include "f32x2.cuh"

#define PH_TAB 1024                                      // table angles 2 pi j / PH_TAB
#define PH_ROUND ((1ull << 53) + (1ull << 30))           // table index and remainder rounded to nearest
#define PH_KAPPA (3.14159265358979f * 0x1p-32f)          // radians per unit of the remainder, 2 pi / 2^33
#define PH_S6 (-(PH_KAPPA * PH_KAPPA) / 6.0f)

// The weights of one atom: w, w PH_KAPPA and -w PH_KAPPA^2 / 2
struct PhWeight {
    float w, wk, wc;
};

__device__ __forceinline__ PhWeight ph_weight(float w)
{
    return {w, w * PH_KAPPA, w * (-0.5f * PH_KAPPA * PH_KAPPA)};
}

// w exp(2 pi i ph / 2^64) for a phase that already carries PH_ROUND; tab is
// the PH_TAB-entry table (shared memory).  w T is formed exactly inside the
// last FMA, so the weighted phasor is rounded once (plus the table's own
// rounding).
__device__ __forceinline__ float2 ph_phasor(uint64_t ph, const float2 *__restrict__ tab, PhWeight a)
{
    const float2 T = tab[(uint32_t)(ph >> 54)];
    const float d = __uint_as_float(((uint32_t)(ph >> 31) & 0x7FFFFFu) | 0x4B000000u) - 12582912.0f;
    const float d2 = d * d;
    const float v = (a.wk * d) * fmaf(d2, PH_S6, 1.0f);      // w sin(d)
    const float u = d2 * a.wc;                                // w (cos(d) - 1)
    return make_float2(fmaf(T.x, a.w, fmaf(T.x, u, -T.y * v)), fmaf(T.y, a.w, fmaf(T.y, u, T.x * v)));
}

// The same for two phases at once with packed FP32x2 arithmetic: every
// operation rounds as ph_phasor's, so the values are the same bit for bit.
// The table comes as separate arrays of x and y (tabs: x at tabs[j], y at
// tabs[PH_TAB + j]), whose entries load straight into the packed registers.
struct PhWeight2 {
    f32x2 w, wk, wc;
};

__device__ __forceinline__ PhWeight2 ph_weight2(float w)
{
    const PhWeight a = ph_weight(w);
    return {pack_f32(a.w, a.w), pack_f32(a.wk, a.wk), pack_f32(a.wc, a.wc)};
}

// j0, j1: table indices; r0, r1: the 23 remainder bits
__device__ __forceinline__ void ph_phasor2(uint32_t j0, uint32_t r0, uint32_t j1, uint32_t r1,
                                           const float *__restrict__ tabs, const PhWeight2 &a, f32x2 &ex, f32x2 &ey)
{
    const f32x2 tx = pack_f32(tabs[j0], tabs[j1]), ty = pack_f32(tabs[PH_TAB + j0], tabs[PH_TAB + j1]);
    const f32x2 d = add_f32x2(pack_f32(__uint_as_float(r0 | 0x4B000000u), __uint_as_float(r1 | 0x4B000000u)),
                              splat_f32x2(-12582912.0f));
    const f32x2 d2 = mul_f32x2(d, d);
    const f32x2 v = mul_f32x2(mul_f32x2(a.wk, d), fma_f32x2(d2, splat_f32x2(PH_S6), splat_f32x2(1.0f)));
    const f32x2 nv = mul_f32x2(v, splat_f32x2(-1.0f));
    const f32x2 u = mul_f32x2(d2, a.wc);
    ex = fma_f32x2(tx, a.w, fma_f32x2(tx, u, mul_f32x2(ty, nv)));
    ey = fma_f32x2(ty, a.w, fma_f32x2(ty, u, mul_f32x2(tx, v)));
}
