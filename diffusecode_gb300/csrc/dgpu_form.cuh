// Form factors at one grid point, shared by the combine and adjoint kernels:
// h of a box point, cfact of a type (table, four_formtab fourier_sup.f90:
// 2691-2743, or the same formula at the exact sin(theta)/lambda), the
// anisotropic Debye-Waller term (four_dbwtab, fourier_sup.f90:2809-2831) and
// the factor of a partial-sum group (tcsf_form_iso / tcsf_form_aniso,
// fourier_form.f90:106-177).
#pragma once
#include "dgpu_internal.h"

// h = eck + i vi_1 + j vi_2 + l vi_3, unfused (four_dbwtab :2810-2821)
__device__ __forceinline__ void form_hvec(const FormSpec *fs, int64_t i, int64_t j, int64_t l, double h[3])
{
    for (int k = 0; k < 3; k++)
        h[k] = __dadd_rn(__dadd_rn(__dadd_rn(fs->eck[k], __dmul_rn(fs->vi[k], (double)i)),
                                   __dmul_rn(fs->vi[3 + k], (double)j)),
                         __dmul_rn(fs->vi[6 + k], (double)l));
}

// cfact of type t (1-based) at a point: table or exact sin(theta)/lambda
__device__ __forceinline__ double2 form_cfact(const FormSpec *fs, const double2 *cfact, int32_t istl,
                                              int t, const double h[3])
{
    if (fs->mode == DGPU_FORM_TABLE) return cfact[(int64_t)(t - 1) * DGPU_NTAB + istl];
    const double *r = fs->rten;
    double t0 = __dadd_rn(__dadd_rn(__dmul_rn(r[0], h[0]), __dmul_rn(r[3], h[1])), __dmul_rn(r[6], h[2]));
    double t1 = __dadd_rn(__dadd_rn(__dmul_rn(r[1], h[0]), __dmul_rn(r[4], h[1])), __dmul_rn(r[7], h[2]));
    double t2 = __dadd_rn(__dadd_rn(__dmul_rn(r[2], h[0]), __dmul_rn(r[5], h[1])), __dmul_rn(r[8], h[2]));
    double q2 = __dadd_rn(__dadd_rn(__dmul_rn(h[0], t0), __dmul_rn(h[1], t1)), __dmul_rn(h[2], t2)) / 4.0;
    const double *sc = fs->scat + 11 * t;
    double f = sc[0];
    if (fs->lxray)
        for (int i = 1; i <= fs->power; i++) f = __dadd_rn(f, __dmul_rn(sc[2 * i - 1], exp(-__dmul_rn(sc[2 * i], q2))));
    double fp = fs->ano ? fs->delfr[t] : 0.0, fpp = fs->ano ? fs->delfi[t] : 0.0;
    double sb = fs->ldbw ? __dmul_rn(exp(-__dmul_rn(fs->dw[t], q2)), fs->occ[t]) : fs->occ[t];
    return make_double2(__dmul_rn(sb, __dadd_rn(f, fp)), __dmul_rn(sb, fpp));
}

// The part of the anisotropic exponent's terms that depends on h alone: h_i h_j
// a*_i a*_j in the reference's order of factors, the mixed ones doubled (exact)
struct AnisTerms {
    double t11, t22, t33, t23, t13, t12;
};

__device__ __forceinline__ AnisTerms form_anis_terms(const FormSpec *fs, const double h[3])
{
    const double *a = fs->ar;
    return {__dmul_rn(__dmul_rn(__dmul_rn(h[0], h[0]), a[0]), a[0]),
            __dmul_rn(__dmul_rn(__dmul_rn(h[1], h[1]), a[1]), a[1]),
            __dmul_rn(__dmul_rn(__dmul_rn(h[2], h[2]), a[2]), a[2]),
            2.0 * __dmul_rn(__dmul_rn(__dmul_rn(h[1], h[2]), a[1]), a[2]),
            2.0 * __dmul_rn(__dmul_rn(__dmul_rn(h[0], h[2]), a[0]), a[2]),
            2.0 * __dmul_rn(__dmul_rn(__dmul_rn(h[0], h[1]), a[0]), a[1])};
}

// exp(-2 pi^2 sum_ij h_i h_j a*_i a*_j U_ij) of group g, in the reference's
// order of terms: (U11 + U22 + U33 + 2 U23 + 2 U13 + 2 U12) * zpi * pi
__device__ __forceinline__ double form_anis_dbw(const FormSpec *fs, int g, const AnisTerms &p)
{
    const double pi = 3.1415926535897932384626433832795028841971693993751;
    const double *u = fs->gU + 6 * g;
    double arg = __dadd_rn(__dadd_rn(__dmul_rn(p.t11, u[0]), __dmul_rn(p.t22, u[1])), __dmul_rn(p.t33, u[2]));
    arg = __dadd_rn(__dadd_rn(__dadd_rn(arg, __dmul_rn(p.t23, u[3])), __dmul_rn(p.t13, u[4])), __dmul_rn(p.t12, u[5]));
    arg = __dmul_rn(__dmul_rn(arg, 2.0 * pi), pi);
    return exp(-arg);
}

// whether the factors need h (analytic form factor, anisotropic term, DISCAMB)
__host__ __device__ __forceinline__ bool form_needs_h(const FormSpec *fs)
{
    return fs->mode != DGPU_FORM_TABLE || fs->adbw || fs->disc;
}

// DISCAMB table of group g at nint(h) (tcsf_form_discamb, fourier_form.f90:
// 90-97; nint rounds half away from zero); NaN outside the table
__device__ __forceinline__ double2 form_discamb(const FormSpec *fs, int g, const double h[3])
{
    const int32_t m0 = fs->gtab[g];
    if (m0 < 0 || m0 >= fs->dntab) return make_double2(nan(""), nan(""));
    int64_t idx = 0, stride = 1;
    for (int k = 0; k < 3; k++) {
        const double r = round(h[k]);
        const int32_t m = fs->dmax[k];
        if (!(r >= -(double)m && r <= (double)m)) return make_double2(nan(""), nan(""));
        idx += ((int64_t)r + m) * stride;
        stride *= 2 * (int64_t)m + 1;
    }
    return fs->dtab[(int64_t)m0 * stride + idx];
}

// factor of partial-sum group g (1-based); an: the point's AnisTerms (read with adbw only)
__device__ __forceinline__ double2 form_group(const FormSpec *fs, const double2 *cfact, int32_t istl, int g,
                                              const double h[3], const AnisTerms &an)
{
    double2 c = fs->disc ? form_discamb(fs, g, h) : form_cfact(fs, cfact, istl, fs->gtype[g], h);
    if (fs->adbw) {
        const double d = form_anis_dbw(fs, g, an);
        c.x = __dmul_rn(c.x, d);
        c.y = __dmul_rn(c.y, d);
    }
    return c;
}

__device__ __forceinline__ double2 form_group(const FormSpec *fs, const double2 *cfact, int32_t istl, int g,
                                              const double h[3])
{
    AnisTerms an = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (fs->adbw) an = form_anis_terms(fs, h);
    return form_group(fs, cfact, istl, g, h, an);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// F += s c.  The factors are real except with anomalous dispersion or a
// DISCAMB table: two multiply-adds instead of four at this part's FP64 rate
// (the test is on the bits, in integer arithmetic; an infinite or NaN sum
// takes the general form, whose products with 0 are NaN).
__device__ __forceinline__ void cfma(double2 &F, double2 s, double2 c)
{
    const bool real = (__double_as_longlong(c.y) << 1) == 0 && (__double2hiint(s.x) & 0x7FF00000) != 0x7FF00000 &&
                      (__double2hiint(s.y) & 0x7FF00000) != 0x7FF00000;
    if (!real) {
        F.x = fma(-s.y, c.y, F.x);
        F.y = fma(s.x, c.y, F.y);
    }
    F.x = fma(s.x, c.x, F.x);
    F.y = fma(s.y, c.x, F.y);
}

// one-axis geometric series sum_{m<n} exp(2 pi i x m)
__device__ __forceinline__ double2 geom_series(double x, int32_t n)
{
    double xr = x - rint(x);
    if (xr == 0.0) return make_double2((double)n, 0.0);
    double num = sinpi((double)n * xr), den = sinpi(xr);
    double r = num / den, sp, cp;
    sincospi(xr * (double)(n - 1), &sp, &cp);
    return make_double2(r * cp, r * sp);
}

// exp(2 pi i h.d), the phase h.d reduced exactly
__device__ __forceinline__ double2 lattice_shift(const double h[3], double d0, double d1, double d2)
{
    double p0 = h[0] * d0, e0 = fma(h[0], d0, -p0);
    double p1 = h[1] * d1, e1 = fma(h[1], d1, -p1);
    double p2 = h[2] * d2, e2 = fma(h[2], d2, -p2);
    double ph = (p0 - rint(p0)) + (p1 - rint(p1)) + (p2 - rint(p2)) + (e0 + e1 + e2);
    double sp, cp;
    sincospi(2.0 * ph, &sp, &cp);
    return make_double2(cp, sp);
}

// Lattice sum of a box of c0 x c1 x c2 cells starting at d (four_strucf(0,..)
// over the lattice of four_getav, fourier_sup.f90:1315-1318) in closed form:
// a product of three geometric series times exp(2 pi i h.d).
__device__ __forceinline__ double2 lattice_closed(const double h[3], int32_t c0, int32_t c1, int32_t c2, double d0,
                                                  double d1, double d2)
{
    return cmul(cmul(cmul(geom_series(h[0], c0), geom_series(h[1], c1)), geom_series(h[2], c2)),
                lattice_shift(h, d0, d1, d2));
}

// box point of partial-sum layout slot r (PartLayout), false for a padding slot
__device__ __forceinline__ bool part_point(const PartLayout &L, const BoxSpec &box, int64_t r, int64_t &i,
                                           int64_t &j, int64_t &l)
{
    int64_t c0, c1, c2;
    if (L.nthr <= 0xFFFFFFFFll) {                 // 32-bit divisions, a quarter of the instructions
        const uint32_t q = (uint32_t)r, m1 = (uint32_t)L.m1, m2 = (uint32_t)L.m2;
        const uint32_t d2 = q / m2, rem = q - d2 * m2, d1 = m1 > 0 ? rem / m1 : 0;
        c2 = d2;
        c1 = d1;
        c0 = rem - d1 * m1;
    } else {
        c2 = r / L.m2;
        const int64_t rem = r - c2 * L.m2;
        c1 = L.m1 > 0 ? rem / L.m1 : 0;
        c0 = rem - c1 * L.m1;
    }
    if (c0 >= box.f[L.a0] || c1 >= box.f[L.a1] || c2 >= box.f[L.a2]) return false;
    i = L.a0 == 0 ? c0 : L.a1 == 0 ? c1 : c2;
    j = L.a0 == 1 ? c0 : L.a1 == 1 ? c1 : c2;
    l = L.a0 == 2 ? c0 : L.a1 == 2 ? c1 : c2;
    return true;
}

// (hi, lo) += x in float-float: Knuth's TwoSum, the error carried in lo
__device__ __forceinline__ void ff_add(float &hi, float &lo, float x)
{
    const float s = hi + x, bp = s - hi;
    lo += (hi - (s - bp)) + (x - bp);
    hi = s;
}

// The sum of a group's K-slice partials at one point, in slice order, eight
// slices loaded before any is added (loads in flight).  FP32 partials are
// added in float-float (TwoSum, 48-bit significands) rather than FP64, whose
// rate on this part bounded the combine; FP64 partials in FP64.  Whole rounds
// carry no tests and step one pointer: on a small box a warp's instructions,
// one after another, are the kernel's time.
template <class P, class Add>
__device__ __forceinline__ void slice_walk(const P *__restrict__ pt, int32_t nslice, int64_t slab, Add add)
{
    for (; nslice >= 8; nslice -= 8) {
        P v[8];
#pragma unroll
        for (int u = 0; u < 8; u++, pt += slab) v[u] = *pt;
#pragma unroll
        for (int u = 0; u < 8; u++) add(v[u]);
    }
    P v[7];
#pragma unroll
    for (int u = 0; u < 7; u++, pt += slab)
        if (u < nslice) v[u] = *pt;
#pragma unroll
    for (int u = 0; u < 7; u++)
        if (u < nslice) add(v[u]);
}

__device__ __forceinline__ double2 slice_sum(const float2 *__restrict__ pt, int32_t nslice, int64_t slab)
{
    float hx = 0.f, lx = 0.f, hy = 0.f, ly = 0.f;
    slice_walk(pt, nslice, slab, [&](float2 v) {
        ff_add(hx, lx, v.x);
        ff_add(hy, ly, v.y);
    });
    return make_double2((double)hx + (double)lx, (double)hy + (double)ly);
}

__device__ __forceinline__ double2 slice_sum(const double2 *__restrict__ pt, int32_t nslice, int64_t slab)
{
    double2 s = make_double2(0.0, 0.0);
    slice_walk(pt, nslice, slab, [&](double2 v) {
        s.x += v.x;
        s.y += v.y;
    });
    return s;
}

// An FP32 estimate of istl (below) that decides almost every point: h and the
// metric r rounded to FP32, each term of q = h.G*.h within 8 roundings of
// 2^-24, so q errs by less than 1e-6 of the terms' magnitudes and sqrt(q)/2
// 1000 by 500 / sqrt(q) of that, plus 4e-7 of itself.  -1: too near a half
// integer (or not finite), the exact form decides.
__device__ __forceinline__ int32_t stl_estimate(const double *r, float h0, float h1, float h2)
{
    const float p00 = (float)r[0] * h0 * h0, p11 = (float)r[4] * h1 * h1, p22 = (float)r[8] * h2 * h2;
    const float p01 = ((float)r[3] + (float)r[1]) * h0 * h1, p02 = ((float)r[6] + (float)r[2]) * h0 * h2,
                p12 = ((float)r[7] + (float)r[5]) * h1 * h2;
    const float q = p00 + p11 + p22 + p01 + p02 + p12;
    const float mag = fabsf(p00) + fabsf(p11) + fabsf(p22) + fabsf(p01) + fabsf(p02) + fabsf(p12);
    const float s = sqrtf(q), x = 500.0f * s, err = 2.0f * (500.0f * 1e-6f * mag / s + 1e-6f * x + 1e-6f);
    const float n = rintf(x);
    return fabsf(x - n) + err < 0.5f ? (int32_t)n : -1;
}

// istl = NINT(sqrt(h.G*.h/4)/CFINC) of a grid point with h rounded to REAL(4)
// (four_stltab, fourier_sup.f90:2637-2687); e = eck(:,1), r = rten column-major
__device__ __forceinline__ long long stl_index(const double *e, const double *vi, const double *r, int64_t i,
                                               int64_t j, int64_t l)
{
    double h[3];
    for (int k = 0; k < 3; k++) {
        double s = __dadd_rn(__dadd_rn(__dadd_rn(e[k], __dmul_rn(vi[k], (double)i)),
                                       __dmul_rn(vi[3 + k], (double)j)),
                             __dmul_rn(vi[6 + k], (double)l));
        h[k] = (double)__double2float_rn(s);
    }
    const int32_t n = stl_estimate(r, (float)h[0], (float)h[1], (float)h[2]);
    if (n >= 0) return n;
    double t0 = __dadd_rn(__dadd_rn(__dmul_rn(r[0], h[0]), __dmul_rn(r[3], h[1])), __dmul_rn(r[6], h[2]));
    double t1 = __dadd_rn(__dadd_rn(__dmul_rn(r[1], h[0]), __dmul_rn(r[4], h[1])), __dmul_rn(r[7], h[2]));
    double t2 = __dadd_rn(__dadd_rn(__dmul_rn(r[2], h[0]), __dmul_rn(r[5], h[1])), __dmul_rn(r[8], h[2]));
    double q = __dadd_rn(__dadd_rn(__dmul_rn(h[0], t0), __dmul_rn(h[1], t1)), __dmul_rn(h[2], t2));
    double q2 = q / 4.0;
    return llround(__dmul_rn(__dsqrt_rn(q2), 1000.0));
}
