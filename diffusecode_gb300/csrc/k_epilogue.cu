// Epilogue kernels of four_run (discus/prog/fourier_sup.f90:136-294):
//   * combine: csf = sum_g factor_g(point) * S_g - acsf ; dsi = |csf|^2
//     (tcsf_form_iso / tcsf_form_aniso, fourier_form.f90:106-177;
//     fourier_sup.f90:205,232,250-254), with diff_scale applied
//     (fourier_sup.f90:281-282);
//   * lots: the same per lot of a chunk, dsi accumulated over the lots and
//     normalised by icc1*icc2*icc3 / (ncell*nlots) (fourier_sup.f90:136-277);
//   * <F>: acsf = (sum_t cfact_t * Savg_t) * lattice / ncell
//     (four_aver, fourier_sup.f90:1194-1357); the lattice sum is either the
//     direct sum over all cells or its closed form (a product of three
//     geometric series);
//   * Friedel mirror (four_apply_friedel, fourier_sup.f90:3726-3757), with the
//     net effect of its sequential in-place loop on the middle slab;
//   * four_qinfo statistics (fourier_sup.f90:2859-2942).
// A run without <F>, lots or filter does all of it in one pass
// (k_combine_finish); the others combine first and mirror last (k_mirror_stats).
#include <algorithm>

#include "dgpu_form.cuh"
#include "dgpu_lots.h"

__device__ __forceinline__ double2 ld_part(const double2 *p) { return *p; }
__device__ __forceinline__ double2 ld_part(const float2 *p)
{
    float2 v = *p;
    return make_double2((double)v.x, (double)v.y);
}

// element offsets of a partial-sum array (see PartRef)
// Strides of the partial sums along the box axes, and the order in which the
// combine kernels walk them: thread r takes slot r of the partials' own layout
// (axis a0 innermost), so that the reads of the partials -- the bulk of the
// traffic -- are coalesced; padding slots of the tensor-core layout idle.
// (PartLayout: dgpu_internal.h)
PartLayout dgpu_part_layout(const PartRef &r, const BoxSpec &box)
{
    PartLayout L;
    int64_t s[3];
    if (r.s[0] == 0) {
        s[0] = 1;
        s[1] = box.f[0];
        s[2] = (int64_t)box.f[0] * box.f[1];
        L.slab = s[2] * box.f[2];
    } else {
        for (int k = 0; k < 3; k++) s[k] = r.s[k];
        L.slab = r.slab;
    }
    L.s0 = s[0];
    L.s1 = s[1];
    L.s2 = s[2];
    // axes by stride; of two equal strides the axis of extent 1 goes first
    int a[3] = {0, 1, 2};
    auto before = [&](int x, int y) { return s[x] < s[y] || (s[x] == s[y] && box.f[x] == 1 && box.f[y] != 1); };
    for (int p = 0; p < 3; p++)
        for (int q = p + 1; q < 3; q++)
            if (before(a[q], a[p])) {
                const int t = a[p];
                a[p] = a[q];
                a[q] = t;
            }
    L.a0 = a[0];
    L.a1 = a[1];
    L.a2 = a[2];
    L.m1 = s[a[1]];
    L.m2 = s[a[2]];
    L.nthr = L.m2 * box.f[a[2]];
    return L;
}


// F - <F> of box point (i, j, l), unscaled; idx: its place on the full grid.
// HEAVY: the factors need h (form_needs_h), whose code takes twice the
// registers of the table's.
template <bool HEAVY, class P>
__device__ __forceinline__ double2 combine_value(const FormSpec *fs, const P *__restrict__ part, int32_t nslice,
                                                 const PartLayout &lay, const int32_t *__restrict__ istl,
                                                 const double2 *__restrict__ cfact,
                                                 const double2 *__restrict__ acsf, int64_t i, int64_t j, int64_t l,
                                                 int64_t idx)
{
    double h[3];
    AnisTerms an = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (HEAVY) {
        form_hvec(fs, i, j, l, h);
        if (fs->adbw) an = form_anis_terms(fs, h);
    }
    int32_t q = istl ? istl[idx] : 0;
    double2 F = make_double2(0.0, 0.0);
    const P *pt = part + i * lay.s0 + j * lay.s1 + l * lay.s2;
    for (int t = 1; t <= fs->ngroup; t++, pt += nslice * lay.slab) {
        const double2 s = slice_sum(pt, nslice, lay.slab);
        cfma(F, s, HEAVY ? form_group(fs, cfact, q, t, h, an) : cfact[(int64_t)(fs->gtype[t] - 1) * DGPU_NTAB + q]);
    }
    if (acsf) {
        double2 a = acsf[idx];
        F.x -= a.x;
        F.y -= a.y;
    }
    return F;
}

template <bool HEAVY, class P>
__device__ __forceinline__ void combine_slot(const FormSpec *fs, const BoxSpec &box, const P *__restrict__ part,
                                             int32_t nslice, const PartLayout &lay, const int32_t *__restrict__ istl,
                                             const double2 *__restrict__ cfact, const double2 *__restrict__ acsf,
                                             double2 *__restrict__ csf, double *__restrict__ dsi, double ds,
                                             double sqds, int64_t r)
{
    int64_t i, j, l;
    if (r >= lay.nthr || !part_point(lay, box, r, i, j, l)) return;
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    const double2 F = combine_value<HEAVY>(fs, part, nslice, lay, istl, cfact, acsf, i, j, l, idx);
    csf[idx] = make_double2(F.x * sqds, F.y * sqds);
    dsi[idx] = (F.x * F.x + F.y * F.y) * ds;
}

template <bool HEAVY, class P>
__global__ void k_combine(const FormSpec *fs, BoxSpec box, const P *__restrict__ part,
                          int32_t nslice, PartLayout lay, const int32_t *__restrict__ istl,
                          const double2 *__restrict__ cfact, const double2 *__restrict__ acsf,
                          double2 *__restrict__ csf, double *__restrict__ dsi, double ds, double sqds)
{
    combine_slot<HEAVY>(fs, box, part, nslice, lay, istl, cfact, acsf, csf, dsi, ds, sqds,
                 (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// The closed-form lattice sum's geometric series per component of h, where
// that component changes along one grid axis only (any grid whose axes follow
// the reciprocal axes): g[off[a] + n] for component a at index n of its axis.
// The series are FP64 sines and a quotient, which for every point of an 881 x
// 441 box took most of 285 us; the values are the same.
struct LatTab {
    const double2 *g;          // null: evaluated per point
    int32_t axis[3];           // grid axis of component a (0 where it is constant)
    int64_t off[3];
    int32_t shifted;           // the lattice's origin is not 0
};

__global__ void k_lattice_tab(const FormSpec *fs, LatTab t, double2 *__restrict__ g, int32_t c0, int32_t c1,
                              int32_t c2, int32_t n0, int32_t n1, int32_t n2)
{
    const int a = blockIdx.y;
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t len = t.axis[a] == 0 ? n0 : t.axis[a] == 1 ? n1 : n2;
    if (k >= len) return;
    double h[3];
    form_hvec(fs, t.axis[a] == 0 ? k : 0, t.axis[a] == 1 ? k : 0, t.axis[a] == 2 ? k : 0, h);
    g[t.off[a] + k] = geom_series(h[a], a == 0 ? c0 : a == 1 ? c1 : c2);
}

template <class P>
__global__ void k_aver_combine(const FormSpec *fs, BoxSpec box, const P *__restrict__ apart,
                               int32_t anslice, PartLayout lay, const int32_t *__restrict__ istl,
                               const double2 *__restrict__ cfact, const double2 *__restrict__ lat,
                               int32_t lat_nslice, int32_t lat_closed, LatTab tab, int32_t c0, int32_t c1,
                               int32_t c2, double d0, double d1, double d2, double norm,
                               double2 *__restrict__ acsf)
{
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t i, j, l;
    if (r >= lay.nthr || !part_point(lay, box, r, i, j, l)) return;
    int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    int64_t nfull = (int64_t)box.num[0] * box.num[1] * box.num[2];
    double h[3];
    form_hvec(fs, i, j, l, h);
    int32_t q = istl ? istl[idx] : 0;
    double2 A = make_double2(0.0, 0.0);
    for (int t = 1; t <= fs->nscat; t++) {
        double2 s = make_double2(0.0, 0.0);
        const P *pt = apart + (int64_t)(t - 1) * anslice * lay.slab + i * lay.s0 + j * lay.s1 + l * lay.s2;
        for (int k = 0; k < anslice; k++) {
            double2 v = ld_part(pt + (int64_t)k * lay.slab);
            s.x += v.x;
            s.y += v.y;
        }
        double2 m = cmul(s, form_cfact(fs, cfact, q, t, h));
        A.x += m.x;
        A.y += m.y;
    }
    double2 L;
    if (tab.g) {
        const int64_t n[3] = {i, j, l};
        L = cmul(cmul(tab.g[tab.off[0] + n[tab.axis[0]]], tab.g[tab.off[1] + n[tab.axis[1]]]),
                 tab.g[tab.off[2] + n[tab.axis[2]]]);
        if (tab.shifted) L = cmul(L, lattice_shift(h, d0, d1, d2));
    } else if (lat_closed) {
        L = lattice_closed(h, c0, c1, c2, d0, d1, d2);
    } else {
        L = make_double2(0.0, 0.0);
        for (int k = 0; k < lat_nslice; k++) {
            double2 v = lat[(int64_t)k * nfull + idx];
            L.x += v.x;
            L.y += v.y;
        }
    }
    const double2 av = cmul(A, L);
    acsf[idx] = make_double2(av.x * norm, av.y * norm);
}

// indices of point p of a grid of np = n0 n1 n2 points (32-bit divisions where they do)
__device__ __forceinline__ void grid_point(const int32_t *n, int64_t np, int64_t p, int32_t c[3])
{
    if (np <= 0xFFFFFFFFll) {
        const uint32_t q = (uint32_t)p, r = q / (uint32_t)n[0];
        c[0] = (int32_t)(q - r * (uint32_t)n[0]);
        c[2] = (int32_t)(r / (uint32_t)n[1]);
        c[1] = (int32_t)(r - (uint32_t)c[2] * (uint32_t)n[1]);
    } else {
        c[0] = (int32_t)(p % n[0]);
        c[1] = (int32_t)((p / n[0]) % n[1]);
        c[2] = (int32_t)(p / ((int64_t)n[0] * n[1]));
    }
}

// four_apply_friedel: points past the halved axis' middle take the conjugate
// of their mirror; on the middle slab the sequential loop leaves the first
// half, conjugates the centre and mirrors the second half.
__device__ __forceinline__ void mirror_point(const BoxSpec &box, int32_t a, double2 *csf, double2 *acsf,
                                             double *dsi, int64_t p)
{
    const int32_t *n = box.num;
    int64_t np = (int64_t)n[0] * n[1] * n[2];
    if (p >= np) return;
    int32_t c[3];
    grid_point(n, np, p, c);
    int32_t mid = box.f[a] - 1;
    if (c[a] < mid) return;
    int64_t m = (n[0] - 1 - c[0]) + (int64_t)n[0] * ((n[1] - 1 - c[1]) + (int64_t)n[1] * (n[2] - 1 - c[2]));
    if (c[a] == mid) {
        // linear index over the later axes, last axis fastest
        int64_t L = 0, N = 1;
        for (int k = a + 1; k < 3; k++) {
            L = L * n[k] + c[k];
            N *= n[k];
        }
        if (2 * L < N - 1) return;
        if (2 * L == N - 1) {
            csf[p].y = -csf[p].y;
            if (acsf) acsf[p].y = -acsf[p].y;
            return;
        }
    }
    double2 v = csf[m];
    csf[p] = make_double2(v.x, -v.y);
    if (acsf) {
        double2 u = acsf[m];
        acsf[p] = make_double2(u.x, -u.y);
    }
    dsi[p] = dsi[m];
}

// member-indexed combine and mirror of a batch (member blockIdx.y)
template <bool HEAVY>
__global__ void k_combine_m(const EpiMember *__restrict__ M)
{
    const EpiMember &m = M[blockIdx.y];
    combine_slot<HEAVY, float2>(m.fs, m.box, m.part, m.nslice, m.lay, m.istl, m.cfact, nullptr, m.csf, m.dsi, m.ds,
                         m.sqds, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void k_mirror_m(const EpiMember *__restrict__ M)
{
    const EpiMember &m = M[blockIdx.y];
    if (m.idim < 1 || m.idim > 3) return;
    mirror_point(m.box, m.idim - 1, m.csf, nullptr, m.dsi, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

int dgpu_epilogue_members(dgpu_ctx *ctx, const EpiMember *d_m, int32_t nc, bool heavy, int64_t max_thr,
                          int64_t max_np)
{
    if (nc < 1) return DGPU_OK;
    const dim3 grid((unsigned)dgpu_cdiv(max_thr, 256), (unsigned)nc);
    if (heavy)
        k_combine_m<true><<<grid, 256, 0, ctx->stream>>>(d_m);
    else
        k_combine_m<false><<<grid, 256, 0, ctx->stream>>>(d_m);
    k_mirror_m<<<dim3((unsigned)dgpu_cdiv(max_np, 256), (unsigned)nc), 256, 0, ctx->stream>>>(d_m);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

// Whether h = e + v0 i + v1 j + v2 l can be an integer: the FP32 estimate
// errs by at most 7 roundings of 2^-24 times mag = |e| + |v0| i + |v1| j +
// |v2| l (four inputs, three FMAs), well inside 1e-6 mag + 1e-5, so an
// estimate farther than that from every integer rules the point out and the
// FP64 test in the reference's order is needed only near integers.
__device__ __forceinline__ bool maybe_integral(float e, float v0, float v1, float v2, float fi, float fj, float fl)
{
    const float h = fmaf(v2, fl, fmaf(v1, fj, fmaf(v0, fi, e)));
    const float mag = fabsf(e) + fabsf(v0) * fi + fabsf(v1) * fj + fabsf(v2) * fl;
    return fabsf(h - rintf(h)) <= fmaf(1e-6f, mag, 1e-5f);
}

// the grid's corner and increments, by value (four_qinfo's h), and in FP32
struct GridVec {
    double e[3], vi[9];
    float fe[3], fvi[9];
};

// whether grid point (i, j, l) is a Bragg position: mod(h, 1) == 0 for the
// three components, h as the reference computes it
__device__ __forceinline__ bool is_bragg(const GridVec &g, uint32_t i, uint32_t j, uint32_t l)
{
    const float fi = (float)i, fj = (float)j, fl = (float)l;
    bool bragg = true;
#pragma unroll
    for (int k = 0; k < 3; k++)
        bragg = bragg && maybe_integral(g.fe[k], g.fvi[k], g.fvi[3 + k], g.fvi[6 + k], fi, fj, fl);
    if (bragg)
        for (int k = 0; k < 3; k++) {
            const double h = __dadd_rn(__dadd_rn(__dadd_rn(g.e[k], __dmul_rn(g.vi[k], (double)i)),
                                                 __dmul_rn(g.vi[3 + k], (double)j)),
                                       __dmul_rn(g.vi[6 + k], (double)l));
            bragg = bragg && (h == trunc(h));
        }
    return bragg;
}

// One thread's statistics.  FP64 instructions are what the kernels below run
// out of, so minima and maxima are taken on order-preserving integer keys (NaN
// taken for none, as fmin and fmax do) and a value that stands for itself and
// its Friedel mate is added once, into p1 and p2.
struct QAcc {
    long long bmax, bmin, dmax, dmin;
    double s1, s2, p1, p2;
    uint32_t n1, np;
};

// The statistics of several threads' points (extrema as keys).
struct QStat {
    long long bmax, bmin, dmax, dmin;
    double dsum, dsum2;
    long long nd;
};

// the key of a finite or infinite value; its own inverse
__device__ __forceinline__ long long qkey(long long b) { return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFll); }
#define QKEY_INF 0x7FF0000000000000ll          // +infinity; -infinity: ~QKEY_INF

__device__ __forceinline__ QAcc qinit()
{
    const long long lo = qkey(__double_as_longlong(-9999.0)), hi = qkey(__double_as_longlong((double)1e19f));
    return {lo, hi, lo, hi, 0.0, 0.0, 0.0, 0.0, 0u, 0u};
}

__device__ __forceinline__ void qminmax(long long &mx, long long &mn, long long k)
{
    if (k > mx && k <= QKEY_INF) mx = k;
    if (k < mn && k >= ~QKEY_INF) mn = k;
}

// v at one point
__device__ __forceinline__ void qadd(QAcc &s, double v, bool bragg)
{
    const long long k = qkey(__double_as_longlong(v));
    if (bragg) {
        qminmax(s.bmax, s.bmin, k);
    } else {
        qminmax(s.dmax, s.dmin, k);
        s.s1 += v;
        s.s2 = fma(v, v, s.s2);
        s.n1++;
    }
}

// v at a point and at its Friedel mate
__device__ __forceinline__ void qadd_pair(QAcc &s, double v, bool bragg, bool mate)
{
    if (bragg || mate) {
        qadd(s, v, bragg);
        qadd(s, v, mate);
    } else {
        qminmax(s.dmax, s.dmin, qkey(__double_as_longlong(v)));
        s.p1 += v;
        s.p2 = fma(v, v, s.p2);
        s.np++;
    }
}

__device__ __forceinline__ QStat qstat(const QAcc &s)
{
    return {s.bmax, s.bmin, s.dmax, s.dmin, fma(2.0, s.p1, s.s1), fma(2.0, s.p2, s.s2), (long long)s.n1 + 2ll * s.np};
}

__device__ __forceinline__ void qmerge(QStat &a, const QStat &b)
{
    a.bmax = max(a.bmax, b.bmax);
    a.bmin = min(a.bmin, b.bmin);
    a.dmax = max(a.dmax, b.dmax);
    a.dmin = min(a.dmin, b.dmin);
    a.dsum += b.dsum;
    a.dsum2 += b.dsum2;
    a.nd += b.nd;
}

__device__ __forceinline__ double qvalue(long long key) { return __longlong_as_double(qkey(key)); }

// What a run's last kernel leaves in pinned host memory: res(0:6) of
// four_qinfo and the tensor-core engine's error flag.
struct FinishOut {
    QStat *parts;                 // one per block
    unsigned int *tick;           // zero before and after the launch
    const int32_t *err;           // null: no tensor-core launch
    double *res;
    int32_t *h_err;
};

#define QNT 128
#define QBLOCKS_PER_SM 4
// The statistics of the blocks' points: added up in the block, and the block
// that finishes last merges all blocks' and writes the results.
__device__ __forceinline__ void finish_stats(const QStat &mine, const FinishOut &o)
{
    __shared__ QStat sh[QNT / 32];
    __shared__ bool last;
    // the block's, on thread 0: a warp's by shuffles, then the warps in order
    auto block = [&](QStat s) {
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            QStat b;
            b.bmax = __shfl_down_sync(0xffffffffu, s.bmax, m);
            b.bmin = __shfl_down_sync(0xffffffffu, s.bmin, m);
            b.dmax = __shfl_down_sync(0xffffffffu, s.dmax, m);
            b.dmin = __shfl_down_sync(0xffffffffu, s.dmin, m);
            b.dsum = __shfl_down_sync(0xffffffffu, s.dsum, m);
            b.dsum2 = __shfl_down_sync(0xffffffffu, s.dsum2, m);
            b.nd = __shfl_down_sync(0xffffffffu, s.nd, m);
            qmerge(s, b);
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < QNT / 32; w++) qmerge(s, sh[w]);
        return s;
    };
    __syncwarp();
    QStat s = block(mine);
    if (threadIdx.x == 0) {
        o.parts[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(o.tick, 1u) == gridDim.x - 1;
        if (last) *o.tick = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = qstat(qinit());
#pragma unroll 4
    for (int k = threadIdx.x; k < (int)gridDim.x; k += QNT) qmerge(s, o.parts[k]);
    s = block(s);
    if (threadIdx.x != 0) return;
    double ave = 0.0, sig = 0.0;
    if (s.nd) {
        ave = s.dsum / (double)s.nd;
        // not contracted: with equal values the two terms round alike, where a
        // fused difference is the rounding error of the square, of either
        // sign; a negative rest in other sums is rounding as well
        const double var = __dsub_rn(s.dsum2 / (double)s.nd, __dmul_rn(ave, ave));
        sig = sqrt(var < 0.0 && isfinite(var) ? 0.0 : var);
    }
    o.res[0] = 6.0;
    o.res[1] = qvalue(s.dmin);
    o.res[2] = qvalue(s.dmax);
    o.res[3] = ave;
    o.res[4] = sig;
    o.res[5] = qvalue(s.bmin);
    o.res[6] = qvalue(s.bmax);
    *o.h_err = o.err ? *(volatile const int32_t *)o.err : 0;
}

// Friedel mirror (axis a, -1: none) of every grid point and its statistics
__global__ void __launch_bounds__(QNT, QBLOCKS_PER_SM) k_mirror_stats(BoxSpec box, int32_t a, double2 *csf, double2 *acsf,
                                                      double *dsi, const __grid_constant__ GridVec g, FinishOut o)
{
    QAcc s = qinit();
    const int64_t np = (int64_t)box.num[0] * box.num[1] * box.num[2];
    for (int64_t p = (int64_t)blockIdx.x * QNT + threadIdx.x; p < np; p += (int64_t)gridDim.x * QNT) {
        if (a >= 0) mirror_point(box, a, csf, acsf, dsi, p);
        int32_t c[3];
        grid_point(box.num, np, p, c);
        qadd(s, dsi[p], is_bragg(g, (uint32_t)c[0], (uint32_t)c[1], (uint32_t)c[2]));
    }
    finish_stats(qstat(s), o);
}

// The whole epilogue of a run without <F>, lots or filter in one pass: each
// computed point's F, its Friedel mirror (four_apply_friedel's net effect, as
// mirror_point), and the statistics of both, read back by nothing.  Separate
// kernels re-read csf and dsi: 45 + 15 + 31 + 8 us on 101^3 points, and three
// more launches for a small grid.  Bound by this part's FP64 rate on large
// boxes (form-factor products and the sums of the statistics: what can be is
// done in integers or once for a point and its mate) and by one warp's string
// of instructions on small ones.  101^3 points of two types, eight slices: 100
// -> 55 us; 61 x 45 x 31 with anisotropic factors, 21 slices: 56 -> 45; a plane
// of 201^2, 33 slices: 40 -> 30 (four or eight threads to a point were no
// faster).  Four blocks per SM: with 16 the merge of the blocks' statistics,
// one block's work, took 20 us more, with 3 or 6 either grid was slower.  At
// the 128 registers that four blocks leave, the HEAVY form spills (196 bytes
// of stores, 272 with FP32 partials) and the table's does not.
template <bool HEAVY, class P>
__global__ void __launch_bounds__(QNT, QBLOCKS_PER_SM)
k_combine_finish(const FormSpec *fs, BoxSpec box, const P *__restrict__ part, int32_t nslice, PartLayout lay,
                 const int32_t *__restrict__ istl, const double2 *__restrict__ cfact, double2 *__restrict__ csf,
                 double *__restrict__ dsi, double ds, double sqds, int32_t a, const __grid_constant__ GridVec g,
                 FinishOut o)
{
    QAcc s = qinit();
    const int32_t *n = box.num;
    const bool scaled = ds != 1.0;
    for (int64_t r = (int64_t)blockIdx.x * QNT + threadIdx.x; r < lay.nthr; r += (int64_t)gridDim.x * QNT) {
        int64_t i, j, l;
        if (!part_point(lay, box, r, i, j, l)) continue;
        // 0: own value only, 1: own value and the mirror's, 2: the conjugate of
        // the own value (centre), 3: the mirror's thread writes this point
        int role = 0;
        if (a >= 0) {
            const int64_t ca = a == 0 ? i : a == 1 ? j : l;
            role = 1;
            if (ca == box.f[a] - 1) {
                // linear index over the later axes, last axis fastest
                const int64_t L = a == 0 ? j * n[2] + l : a == 1 ? l : 0;
                const int64_t N = a == 0 ? (int64_t)n[1] * n[2] : a == 1 ? n[2] : 1;
                role = 2 * L < N - 1 ? 1 : 2 * L == N - 1 ? 2 : 3;
            }
        }
        if (role == 3) continue;
        const int64_t idx = i + (int64_t)n[0] * (j + (int64_t)n[1] * l);
        const double2 F = combine_value<HEAVY>(fs, part, nslice, lay, istl, cfact, (const double2 *)nullptr, i, j, l, idx);
        double2 v = F;
        double w = fma(F.x, F.x, F.y * F.y);
        if (scaled) {
            v = make_double2(F.x * sqds, F.y * sqds);
            w *= ds;
        }
        csf[idx] = make_double2(v.x, role == 2 ? -v.y : v.y);
        dsi[idx] = w;
        const bool bragg = is_bragg(g, (uint32_t)i, (uint32_t)j, (uint32_t)l);
        if (role == 1) {
            const int64_t mi = n[0] - 1 - i, mj = n[1] - 1 - j, ml = n[2] - 1 - l;
            const int64_t m = mi + (int64_t)n[0] * (mj + (int64_t)n[1] * ml);
            csf[m] = make_double2(v.x, -v.y);
            dsi[m] = w;
            qadd_pair(s, w, bragg, is_bragg(g, (uint32_t)mi, (uint32_t)mj, (uint32_t)ml));
        } else {
            qadd(s, w, bragg);
        }
    }
    finish_stats(qstat(s), o);
}

// ---------------------------------------------------------------------------
// The device copy of a FormSpec (slot 0: the combine's groups, 1: the plain
// types), uploaded only when it differs from what the slot holds.
int dgpu_spec_device(dgpu_ctx *ctx, int slot, const FormSpec &fs, const FormSpec **d)
{
    dgpu_ctx::SpecSlot &s = ctx->spec[slot];
    if (s.host.size() != sizeof(FormSpec) || memcmp(s.host.data(), &fs, sizeof(FormSpec)) != 0) {
        s.host.clear();
        DGPU_CUDA(ctx, s.dev.ensure(sizeof(FormSpec)));
        // copied from the slot's bytes, which outlive the copy: fs may be gone
        // before the stream reaches it (a run holds one value per slot)
        s.host.assign(reinterpret_cast<const char *>(&fs), reinterpret_cast<const char *>(&fs) + sizeof(FormSpec));
        const cudaError_t e =
            cudaMemcpyAsync(s.dev.p, s.host.data(), sizeof(FormSpec), cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) s.host.clear();
        DGPU_CUDA(ctx, e);
    }
    *d = s.dev.as<FormSpec>();
    return DGPU_OK;
}

int dgpu_combine(dgpu_ctx *ctx, const FormSpec &fs, const BoxSpec &box, const PartRef &part,
                 const int32_t *istl, const double2 *cfact,
                 const double2 *acsf_in, double2 *csf, double *dsi, double diff_scale)
{
    const FormSpec *d;
    int rc = dgpu_spec_device(ctx, 0, fs, &d);
    if (rc) return rc;
    const PartLayout lay = dgpu_part_layout(part, box);
    const unsigned nblk = (unsigned)dgpu_cdiv(lay.nthr, 128);
    const bool heavy = form_needs_h(&fs);
    auto launch = [&](auto kernel, auto *p) {
        kernel<<<nblk, 128, 0, ctx->stream>>>(d, box, p, part.nslice, lay, istl, cfact, acsf_in, csf, dsi, diff_scale,
                                              sqrt(diff_scale));
    };
    if (part.f32)
        launch(heavy ? k_combine<true, float2> : k_combine<false, float2>, (const float2 *)part.p);
    else
        launch(heavy ? k_combine<true, double2> : k_combine<false, double2>, (const double2 *)part.p);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

// blocks over n points, and where the launch leaves its results
static int finish_setup(dgpu_ctx *ctx, int64_t n, bool tc, unsigned &nblk, FinishOut &o)
{
    const int64_t most = (int64_t)QBLOCKS_PER_SM * ctx->nsm, want = dgpu_cdiv(n > 0 ? n : 1, QNT);
    nblk = (unsigned)(want < most ? want : most);
    DGPU_CUDA(ctx, ctx->stats.ensure((size_t)most * sizeof(QStat)));
    o.parts = ctx->stats.as<QStat>();
    o.tick = ctx->tick.as<unsigned int>() + 8;
    o.err = tc ? ctx->flag.as<int32_t>() + 8 : nullptr;
    o.res = ctx->h_fin->res;
    o.h_err = &ctx->h_fin->err;
    return DGPU_OK;
}

static GridVec grid_vec(const dgpu_grid *grid)
{
    GridVec g;
    for (int k = 0; k < 3; k++) g.e[k] = grid->eck[k];
    memcpy(g.vi, grid->vi, sizeof(g.vi));
    for (int k = 0; k < 3; k++) g.fe[k] = (float)g.e[k];
    for (int k = 0; k < 9; k++) g.fvi[k] = (float)g.vi[k];
    return g;
}

int dgpu_combine_finish(dgpu_ctx *ctx, const FormSpec &fs, const BoxSpec &box, int32_t idim, const PartRef &part,
                        const int32_t *istl, const double2 *cfact, const dgpu_grid *grid, double2 *csf, double *dsi,
                        double diff_scale, bool tc)
{
    const FormSpec *d;
    int rc = dgpu_spec_device(ctx, 0, fs, &d);
    if (rc) return rc;
    const PartLayout lay = dgpu_part_layout(part, box);
    unsigned nblk;
    FinishOut o;
    rc = finish_setup(ctx, lay.nthr, tc, nblk, o);
    if (rc) return rc;
    const GridVec g = grid_vec(grid);
    const int32_t a = idim >= 1 && idim <= 3 ? idim - 1 : -1;
    const bool heavy = form_needs_h(&fs);
    auto launch = [&](auto kernel, auto *p) {
        kernel<<<nblk, QNT, 0, ctx->stream>>>(d, box, p, part.nslice, lay, istl, cfact, csf, dsi, diff_scale,
                                              sqrt(diff_scale), a, g, o);
    };
    if (part.f32)
        launch(heavy ? k_combine_finish<true, float2> : k_combine_finish<false, float2>, (const float2 *)part.p);
    else
        launch(heavy ? k_combine_finish<true, double2> : k_combine_finish<false, double2>, (const double2 *)part.p);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

int dgpu_aver_combine(dgpu_ctx *ctx, const FormSpec &fs, const BoxSpec &box, const PartRef &apart,
                      const int32_t *istl, const double2 *cfact, const double2 *lat,
                      int32_t lat_nslice, int32_t lat_closed, const int32_t icc[3],
                      const double dim0[3], double norm, double2 *acsf)
{
    const FormSpec *d;
    int rc = dgpu_spec_device(ctx, 1, fs, &d);
    if (rc) return rc;
    const PartLayout lay = dgpu_part_layout(apart, box);
    const unsigned nblk = (unsigned)dgpu_cdiv(lay.nthr, 128);
    LatTab tab;
    memset(&tab, 0, sizeof(tab));
    bool separable = lat_closed != 0;
    for (int a = 0; a < 3 && separable; a++) {
        int moved = 0;
        for (int k = 0; k < 3; k++)
            if (fs.vi[3 * k + a] != 0.0 && box.f[k] > 1) {
                tab.axis[a] = k;
                moved++;
            }
        separable = moved <= 1;
    }
    if (separable) {
        const int64_t len = std::max(box.f[0], std::max(box.f[1], box.f[2]));
        for (int a = 0; a < 3; a++) tab.off[a] = a * len;
        tab.shifted = dim0[0] != 0.0 || dim0[1] != 0.0 || dim0[2] != 0.0;
        DGPU_CUDA(ctx, ctx->lat_tab.ensure((size_t)(3 * len) * sizeof(double2)));
        k_lattice_tab<<<dim3((unsigned)dgpu_cdiv(len, 128), 3), 128, 0, ctx->stream>>>(
            d, tab, ctx->lat_tab.as<double2>(), icc[0], icc[1], icc[2], box.f[0], box.f[1], box.f[2]);
        DGPU_CUDA(ctx, cudaGetLastError());
        tab.g = ctx->lat_tab.as<double2>();
    }
    if (apart.f32)
        k_aver_combine<float2><<<nblk, 128, 0, ctx->stream>>>(
            d, box, (const float2 *)apart.p, apart.nslice, lay, istl, cfact, lat, lat_nslice, lat_closed, tab, icc[0],
            icc[1], icc[2], dim0[0], dim0[1], dim0[2], norm, acsf);
    else
        k_aver_combine<double2><<<nblk, 128, 0, ctx->stream>>>(
            d, box, (const double2 *)apart.p, apart.nslice, lay, istl, cfact, lat, lat_nslice, lat_closed, tab,
            icc[0], icc[1], icc[2], dim0[0], dim0[1], dim0[2], norm, acsf);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

int dgpu_mirror_stats(dgpu_ctx *ctx, const BoxSpec &box, int32_t idim, const dgpu_grid *grid, double2 *csf,
                      double2 *acsf, double *dsi, bool tc)
{
    unsigned nblk;
    FinishOut o;
    int rc = finish_setup(ctx, (int64_t)box.num[0] * box.num[1] * box.num[2], tc, nblk, o);
    if (rc) return rc;
    k_mirror_stats<<<nblk, QNT, 0, ctx->stream>>>(box, idim >= 1 && idim <= 3 ? idim - 1 : -1, csf, acsf, dsi,
                                                  grid_vec(grid), o);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

// ---------------------------------------------------------------------------
// Lots (fourier_sup.f90:136-277).  The group factors do not depend on the
// lot: they are tabulated once per run on the box, fac[(g-1)*nb + box point].
__global__ void k_group_factors(const FormSpec *fs, BoxSpec box, const int32_t *__restrict__ istl,
                                const double2 *__restrict__ cfact, double2 *__restrict__ fac)
{
    const int64_t pb = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    if (pb >= nb) return;
    const int64_t i = pb % box.f[0], j = (pb / box.f[0]) % box.f[1], l = pb / ((int64_t)box.f[0] * box.f[1]);
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    double h[3];
    if (form_needs_h(fs)) form_hvec(fs, i, j, l, h);
    const int32_t q = istl ? istl[idx] : 0;
    for (int g = 1; g <= fs->ngroup; g++) fac[(int64_t)(g - 1) * nb + pb] = form_group(fs, cfact, q, g, h);
}

// One chunk of nlot lots whose partial sums come as nlot*ngroup types (lot-
// major): dsi += sum_L |sum_g fac_g S_{L,g} - acsf|^2 (unscaled) and, for the
// chunk's lot `last` (-1: none), csf = its F - acsf (unscaled).  part == null:
// the chunk has no atoms.
template <class P>
__global__ void k_lot_combine(int32_t ngroup, int32_t nlot, BoxSpec box, const P *__restrict__ part,
                              int32_t nslice, PartLayout lay, const double2 *__restrict__ fac,
                              const double2 *__restrict__ acsf, double2 *__restrict__ csf,
                              double *__restrict__ dsi, int32_t last)
{
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t i, j, l;
    if (r >= lay.nthr || !part_point(lay, box, r, i, j, l)) return;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    const int64_t pb = i + (int64_t)box.f[0] * (j + (int64_t)box.f[1] * l);
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    const double2 a = acsf ? acsf[idx] : make_double2(0.0, 0.0);
    const int64_t off = i * lay.s0 + j * lay.s1 + l * lay.s2;
    double acc = 0.0;
    if constexpr (sizeof(P) == sizeof(float2)) {
        // FP32 partials (tensor-core engine): the group products in FP32 --
        // the partials carry FP32 rounding already -- with the group factors
        // of the point loaded once; F - <F> and |.|^2 in FP64
        constexpr int GMAX = 8;
        float2 fg[GMAX];
#pragma unroll
        for (int g = 0; g < GMAX; g++) {
            const double2 f = g < ngroup ? fac[(int64_t)g * nb + pb] : make_double2(0.0, 0.0);
            fg[g] = make_float2((float)f.x, (float)f.y);
        }
        for (int L = 0; L < nlot; L++) {
            float fr = 0.f, fi = 0.f;
            if (part)
                for (int g = 0; g < ngroup; g++) {
                    const P *pt = part + (int64_t)(L * ngroup + g) * nslice * lay.slab + off;
                    float sr = 0.f, si = 0.f;
                    for (int k = 0; k < nslice; k++) {
                        const float2 v = *reinterpret_cast<const float2 *>(pt + (int64_t)k * lay.slab);
                        sr += v.x;
                        si += v.y;
                    }
                    float2 f;
                    if (g < GMAX) f = fg[g];
                    else {
                        const double2 fd = fac[(int64_t)g * nb + pb];
                        f = make_float2((float)fd.x, (float)fd.y);
                    }
                    fr = fmaf(sr, f.x, fmaf(-si, f.y, fr));
                    fi = fmaf(sr, f.y, fmaf(si, f.x, fi));
                }
            const double2 F = make_double2((double)fr - a.x, (double)fi - a.y);
            acc += F.x * F.x + F.y * F.y;
            if (L == last) csf[idx] = F;
        }
    } else {
        for (int L = 0; L < nlot; L++) {
            double2 F = make_double2(0.0, 0.0);
            if (part)
                for (int g = 0; g < ngroup; g++) {
                    const P *pt = part + (int64_t)(L * ngroup + g) * nslice * lay.slab + off;
                    double2 s = make_double2(0.0, 0.0);
                    for (int k = 0; k < nslice; k++) {
                        const double2 v = ld_part(pt + (int64_t)k * lay.slab);
                        s.x += v.x;
                        s.y += v.y;
                    }
                    const double2 m = cmul(s, fac[(int64_t)g * nb + pb]);
                    F.x += m.x;
                    F.y += m.y;
                }
            F.x -= a.x;
            F.y -= a.y;
            acc += F.x * F.x + F.y * F.y;
            if (L == last) csf[idx] = F;
        }
    }
    dsi[idx] += acc;
}

// k_lot_combine for FP32 partials with nq = ngroup * nslice partials per lot
// known at compile time: partial q = g * nslice + k of lot L sits at
// (L * NQ + q) * slab, and LB lots' partials are loaded before any is used,
// so that each thread keeps about eight loads in flight (the kernel reads
// nlot * nq partials per point and is bound by those reads).  The arithmetic
// is the generic kernel's, operation for operation: a group's slices are
// added first, then multiplied by its factor.  Without <F> (AV false) F of a
// lot is an FP32 pair and |F|^2 is summed over the lots in float-float (exact
// FMA products, TwoSum, 48-bit significands) rather than FP64, whose rate on
// this part made that sum the kernel's bound; F - <F> keeps FP64.
// 31 lots of two groups on 121 x 91 x 43 points: 80 -> 59 us with the sum of
// lot `last` kept in registers and stored after the loop (its conversions and
// store stood in every lot's path), dsi loaded before it, one stepped pointer
// and blocks of 128 (sixteen loads in flight, blocks of 64 and whole batches
// without tests made no difference).
template <int NQ, bool AV>
__global__ void k_lot_combine_f32(int32_t nslice, int32_t nlot, BoxSpec box, const float2 *__restrict__ part,
                                  PartLayout lay, const double2 *__restrict__ fac, const double2 *__restrict__ acsf,
                                  double2 *__restrict__ csf, double *__restrict__ dsi, int32_t last)
{
    constexpr int LB = NQ >= 8 ? 1 : 8 / NQ;
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t i, j, l;
    if (r >= lay.nthr || !part_point(lay, box, r, i, j, l)) return;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    const int64_t pb = i + (int64_t)box.f[0] * (j + (int64_t)box.f[1] * l);
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    const double2 a = AV ? acsf[idx] : make_double2(0.0, 0.0);
    const float2 *p0 = part + i * lay.s0 + j * lay.s1 + l * lay.s2;
    const int64_t slab = lay.slab;
    const double before = dsi[idx];        // loaded now, added to at the end
    float2 fq[NQ];                         // the group factor of each partial of a lot
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        const double2 f = fac[(int64_t)(q / nslice) * nb + pb];
        fq[q] = make_float2((float)f.x, (float)f.y);
    }
    double acc = 0.0;
    float ah = 0.f, al = 0.f;              // float-float sum of |F|^2 (AV false)
    float lr = 0.f, li = 0.f;              // the group sum of lot `last`
    for (int L0 = 0; L0 < nlot; L0 += LB, p0 += LB * NQ * slab) {
        float2 v[LB][NQ];
#pragma unroll
        for (int b = 0; b < LB; b++)
#pragma unroll
            for (int q = 0; q < NQ; q++)
                v[b][q] = L0 + b < nlot ? __ldg(p0 + (b * NQ + q) * slab) : make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < LB; b++) {
            if (L0 + b < nlot) {
                // the slices of a group added first (in slice order), then the
                // group product: the generic kernel's arithmetic
                float fr = 0.f, fi = 0.f, sr = 0.f, si = 0.f;
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    sr += v[b][q].x;
                    si += v[b][q].y;
                    if ((q + 1) % nslice == 0) {
                        fr = fmaf(sr, fq[q].x, fmaf(-si, fq[q].y, fr));
                        fi = fmaf(sr, fq[q].y, fmaf(si, fq[q].x, fi));
                        sr = 0.f;
                        si = 0.f;
                    }
                }
                if (L0 + b == last) {
                    lr = fr;
                    li = fi;
                }
                if (AV) {
                    const double2 F = make_double2((double)fr - a.x, (double)fi - a.y);
                    acc += F.x * F.x + F.y * F.y;
                } else {
                    const float pr = fr * fr, pi = fi * fi;
                    const float er = fmaf(fr, fr, -pr), ei = fmaf(fi, fi, -pi);   // exact product errors
                    ff_add(ah, al, pr);
                    ff_add(ah, al, pi);
                    al += er + ei;
                }
            }
        }
    }
    if (last >= 0) csf[idx] = make_double2((double)lr - a.x, (double)li - a.y);
    dsi[idx] = before + (AV ? acc : (double)ah + (double)al);
}

// dsi *= dscale, csf *= cscale on the box (lot normalisation and diff_scale)
__global__ void k_lot_scale(BoxSpec box, double2 *__restrict__ csf, double *__restrict__ dsi, double dscale,
                            double cscale)
{
    const int64_t pb = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    if (pb >= nb) return;
    const int64_t i = pb % box.f[0], j = (pb / box.f[0]) % box.f[1], l = pb / ((int64_t)box.f[0] * box.f[1]);
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    dsi[idx] *= dscale;
    const double2 c = csf[idx];
    csf[idx] = make_double2(c.x * cscale, c.y * cscale);
}

int dgpu_group_factors(dgpu_ctx *ctx, const FormSpec &fs, const BoxSpec &box, const int32_t *istl,
                       const double2 *cfact, double2 *fac)
{
    const FormSpec *d;
    int rc = dgpu_spec_device(ctx, 0, fs, &d);
    if (rc) return rc;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    k_group_factors<<<(unsigned)dgpu_cdiv(nb, 256), 256, 0, ctx->stream>>>(d, box, istl, cfact, fac);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

int dgpu_lot_combine(dgpu_ctx *ctx, int32_t ngroup, int32_t nlot, const BoxSpec &box, const PartRef *part,
                     const double2 *fac, const double2 *acsf, double2 *csf, double *dsi, int32_t last)
{
    PartRef none;
    memset(&none, 0, sizeof(none));
    const PartRef &r = part ? *part : none;
    const PartLayout lay = dgpu_part_layout(r, box);
    const unsigned nblk = (unsigned)dgpu_cdiv(lay.nthr, 128);
    const int32_t nslice = r.nslice > 0 ? r.nslice : 1;
    const int32_t nq = ngroup * nslice;
    if (r.f32 && r.p && nq >= 1 && nq <= 8) {
        const float2 *p = (const float2 *)r.p;
        switch (nq) {
#define LOT_F32(Q)                                                                                              \
    case Q:                                                                                                     \
        if (acsf)                                                                                               \
            k_lot_combine_f32<Q, true><<<nblk, 128, 0, ctx->stream>>>(nslice, nlot, box, p, lay, fac, acsf, csf,  \
                                                                      dsi, last);                               \
        else                                                                                                    \
            k_lot_combine_f32<Q, false><<<nblk, 128, 0, ctx->stream>>>(nslice, nlot, box, p, lay, fac, acsf, csf, \
                                                                       dsi, last);                              \
        break;
            LOT_F32(1) LOT_F32(2) LOT_F32(3) LOT_F32(4) LOT_F32(5) LOT_F32(6) LOT_F32(7) LOT_F32(8)
#undef LOT_F32
        }
    } else if (r.f32)
        k_lot_combine<float2><<<nblk, 128, 0, ctx->stream>>>(ngroup, nlot, box, (const float2 *)r.p, nslice, lay,
                                                              fac, acsf, csf, dsi, last);
    else
        k_lot_combine<double2><<<nblk, 128, 0, ctx->stream>>>(ngroup, nlot, box, (const double2 *)r.p, nslice,
                                                               lay, fac, acsf, csf, dsi, last);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

int dgpu_lot_scale(dgpu_ctx *ctx, const BoxSpec &box, double2 *csf, double *dsi, double dscale, double cscale)
{
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    k_lot_scale<<<(unsigned)dgpu_cdiv(nb, 256), 256, 0, ctx->stream>>>(box, csf, dsi, dscale, cscale);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}
