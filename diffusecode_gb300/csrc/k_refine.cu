// Exact recomputation of the points where <F> cancels most of F.
//
// With the average structure factor subtracted (four_aver, fourier_sup.f90:
// 1194-1357, then csf = F - acsf at :250-254), a point near a Bragg position
// of the average lattice has |F| and |<F>| many times larger than the
// incoherent level while F - <F> stays small.  The tensor-core engine's type
// sums carry a relative error of a few 1e-7 (FP32 accumulation in TMEM), so
// there the error of |F - <F>|^2 grows with |<F>| / sqrt(N <|f|^2>): about
// 3.4e-7 times that ratio, measured against FP64.  Those points are found
// after the combine (|acsf|^2 > REFINE_TAU * N <|f|^2>) and their type sums
// -- of the crystal and of the atoms folded into one cell -- are evaluated
// again on CUDA cores: FP32 phasors of the exact 64-bit phase by table-driven
// angle addition (1024-entry table of exp(2 pi i j / 1024) in shared memory
// times a two-term series for the remainder, the method of Tang's
// table-driven elementary functions), FP32 sums of short chunks, FP64 across
// chunks and threads.  csf, acsf and dsi of those
// points are then formed with the same form-factor and lattice code as the
// combine kernels.
//
//  * k_refine_select: one thread per point of the Friedel-reduced box, a flag
//    byte per point;
//  * k_refine_adjacent: along which box axis flagged points most often have a
//    flagged neighbour;
//  * k_refine_list: the flagged points, line by line along that axis, so that
//    a point is usually the previous one plus one step along it and its phase
//    the previous phase plus one 64-bit add (the order decides nothing else:
//    each point's sums are its own);
//  * k_refine_sums: work item = (8 listed points, type, atom slice) of either
//    atom set; FP64 partial per (point, type, slice);
//  * k_refine_combine: one thread per listed point.
// The list used to be appended in no order and sorted on the host, with the
// neighbours counted there by binary search: 6 ms for 7800 points of an
// 881 x 881 plane, as long as the sums.
#include <algorithm>

#include "dgpu_form.cuh"
#include "dgpu_phasor.cuh"
#include "tc_ptx.cuh"

#define RF_PTS 8            // points per work item (each atom's data is read once for all of them)
#define RF_NT 256
#define RF_CHUNK 16         // atoms per FP32 partial before it is added in FP64 (at the most coherent
                            // points FP32 chunks of 32 atoms round alike chunk after chunk: 1.8e-5)
#define RF_SLICE 65536      // atoms per work item
struct RefineTypes {
    int64_t ts[65];         // type ranges of a prepared atom set (0-based types)
    double n[64];           // atoms per type
    int32_t ntype;
};

// flag points with |<F>|^2 > tau * sum_t n_t |cfact_t|^2
__global__ void k_refine_select(const FormSpec *fs, BoxSpec box, const int32_t *__restrict__ istl,
                                const double2 *__restrict__ cfact, const double2 *__restrict__ acsf,
                                const RefineTypes rt, double tau, uint8_t *__restrict__ flag)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    if (p >= nb) return;
    const int64_t i = p % box.f[0], j = (p / box.f[0]) % box.f[1], l = p / ((int64_t)box.f[0] * box.f[1]);
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    const double2 a = acsf[idx];
    double h[3];
    form_hvec(fs, i, j, l, h);
    const int32_t q = istl ? istl[idx] : 0;
    double floor = 0.0;
    for (int t = 1; t <= fs->nscat; t++) {
        const double2 c = form_cfact(fs, cfact, q, t, h);
        floor += rt.n[t - 1] * (c.x * c.x + c.y * c.y);
    }
    flag[p] = a.x * a.x + a.y * a.y > tau * floor;
}

// what the selection leaves: flagged neighbours per axis, listed points
struct RefineCount {
    int32_t adj[3], npts;
};

// the step axis: the one with most flagged neighbours, the first of equals,
// of the axes longer than one point
__device__ __forceinline__ int refine_axis(const BoxSpec &box, const RefineCount *c)
{
    int sa = 0, best = -1;
    for (int a = 0; a < 3; a++)
        if (box.f[a] >= 2 && c->adj[a] > best) {
            best = c->adj[a];
            sa = a;
        }
    return sa;
}

__global__ void k_refine_adjacent(BoxSpec box, const uint8_t *__restrict__ flag, RefineCount *__restrict__ count)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    const bool on = p < nb && flag[p];
    const int64_t st[3] = {1, box.f[0], (int64_t)box.f[0] * box.f[1]};
    for (int a = 0; a < 3; a++) {
        const bool adj = on && (p / st[a]) % box.f[a] + 1 < box.f[a] && flag[p + st[a]];
        const unsigned b = __ballot_sync(0xffffffffu, adj);
        if ((threadIdx.x & 31) == 0 && b) atomicAdd(&count->adj[a], __popc(b));
    }
}

// a warp per line along the step axis: 32 points at a time, the flagged ones
// appended in order
__global__ void k_refine_list(BoxSpec box, const uint8_t *__restrict__ flag, RefineCount *__restrict__ count,
                              int32_t *__restrict__ list)
{
    const int sa = refine_axis(box, count), o1 = sa == 0 ? 1 : 0, o2 = 3 - sa - o1;
    const int64_t st[3] = {1, box.f[0], (int64_t)box.f[0] * box.f[1]};
    const int lane = threadIdx.x & 31;
    const int64_t line = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (line >= (int64_t)box.f[o1] * box.f[o2]) return;
    const int64_t p0 = (line % box.f[o1]) * st[o1] + line / box.f[o1] * st[o2];
    int n = 0;                                   // flagged points of the line, then their place in the list
    for (int c = lane; c < box.f[sa]; c += 32) n += flag[p0 + c * st[sa]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (n == 0) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(&count->npts, n);
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int c0 = 0; c0 < box.f[sa]; c0 += 32) {
        const int64_t p = p0 + (int64_t)(c0 + lane) * st[sa];
        const bool on = c0 + lane < box.f[sa] && flag[p];
        const unsigned b = __ballot_sync(0xffffffffu, on);
        if (on) list[at + __popc(b & ((1u << lane) - 1u))] = (int32_t)p;
        at += __popc(b);
    }
}

__global__ void k_refine_report(BoxSpec box, const RefineCount *__restrict__ count, int32_t *__restrict__ h_out)
{
    h_out[0] = count->npts;
    h_out[1] = refine_axis(box, count);
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The atoms of one work item, n of them: FP32 sums of RF_CHUNK atoms per point
// and thread, added to FP64.  A point is the previous one plus one step along
// axis A, its phase one 64-bit add from the last, or (its bit of brk, never
// with RUN) starts again from its indices along A, B and, if the box has a
// third axis, C.  Pairs of points are evaluated and summed with packed FP32x2
// arithmetic (the roundings of ph_phasor).
//
// Bound by instruction issue, so the loop spends as few as it can beside the
// ~16 of a phasor: every trip count is the same for the whole warp (a thread
// past the end takes the last atom with weight zero) and brk is a ballot, so
// the tests are on uniform registers and need no reconvergence (31 -> 27
// instructions per phasor on short runs of points).  4 blocks of 64 registers
// cover the rest of the waiting better than 3 of 80 registers with or without
// the next atom's loads in flight (a plane of 881 x 881 points, 400 000 atoms,
// 11.96 ms, 12.17 and 12.45).  Its 7800 listed points: 3.61 -> 3.15 ms per
// atom set, 990 phasors per ns.
template <bool RUN, bool THIRD>
__device__ __forceinline__ void refine_loop(int32_t n, const uint64_t *__restrict__ ph0,
                                            const uint64_t *__restrict__ dA, const uint64_t *__restrict__ dB,
                                            const uint64_t *__restrict__ dC, const float *__restrict__ w,
                                            const float *__restrict__ tabs, const uint4 *sn, double (*acc)[RF_NT],
                                            uint32_t brk, bool fA, bool fB)
{
    const uint4 m0 = sn[0];
    for (int32_t a0 = 0; a0 < n;) {
        f32x2 chk[RF_PTS / 2][2];
#pragma unroll
        for (int k = 0; k < RF_PTS / 2; k++) chk[k][0] = chk[k][1] = 0ull;
        const int32_t end = min(n, a0 + RF_CHUNK * RF_NT);
#pragma unroll 1
        for (; a0 < end; a0 += RF_NT) {
            const int32_t i = a0 + (int32_t)threadIdx.x, a = min(i, n - 1);
            // an axis of extent 1 has index 0 at every point: its step is not read
            const uint64_t b = ph0[a] + PH_ROUND, da = fA ? dA[a] : 0, db = fB ? dB[a] : 0, dc = THIRD ? dC[a] : 0;
            const PhWeight2 wa = ph_weight2(i < n ? w[a] : 0.0f);
            auto at = [&](const uint4 &m) {
                uint64_t p = b + (uint64_t)m.x * da + (uint64_t)m.y * db;
                if (THIRD) p += (uint64_t)m.z * dc;
                return p;
            };
            uint64_t ph = at(m0);
            auto step = [&](int k) { ph = !RUN && (brk >> k & 1u) ? at(sn[k]) : ph + da; };
#pragma unroll
            for (int k = 0; k < RF_PTS; k += 2) {
                if (k > 0) step(k);
                const uint64_t qa = ph;
                step(k + 1);
                f32x2 ex, ey;
                ph_phasor2((uint32_t)(qa >> 54), (uint32_t)(qa >> 31) & 0x7FFFFFu, (uint32_t)(ph >> 54),
                           (uint32_t)(ph >> 31) & 0x7FFFFFu, tabs, wa, ex, ey);
                chk[k / 2][0] = add_f32x2(chk[k / 2][0], ex);
                chk[k / 2][1] = add_f32x2(chk[k / 2][1], ey);
                asm volatile("" ::: "memory");   // one pair's table loads at a time: more would spill
            }
        }
#pragma unroll
        for (int k = 0; k < RF_PTS / 2; k++)
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const float2 v = unpack_f32(chk[k][x]);
                acc[4 * k + x][threadIdx.x] += (double)v.x;
                acc[4 * k + 2 + x][threadIdx.x] += (double)v.y;
            }
    }
}

// One of the two atom sets of a refinement (the crystal's groups, the folded
// atoms' types)
struct RefineSet {
    const uint64_t *ph0, *du, *dv, *dw;
    const float *w;
    RefineTypes rt;
    int32_t nsl;           // atom slices
    double2 *out;          // out[(k * ntype + t) * nsl + s]
};

// The type-t sum over atom slice s at listed point k.  The FP64 sums of the
// chunks live in shared memory (one column per thread): 4 blocks of 256
// threads per SM.
__global__ void __launch_bounds__(RF_NT, 4)
k_refine_sums(const int32_t *__restrict__ list, int32_t npts, BoxSpec box, const __grid_constant__ RefineSet S,
              const float2 *__restrict__ gtab, int32_t sa)
{
    __shared__ double red[RF_NT / 32][RF_PTS][2];
    __shared__ float tab[2 * PH_TAB];
    __shared__ double acc[2 * RF_PTS][RF_NT];
    for (int j = threadIdx.x; j < PH_TAB; j += RF_NT) {
        const float2 v = gtab[j];
        tab[j] = v.x;
        tab[PH_TAB + j] = v.y;
    }
#pragma unroll
    for (int k = 0; k < 2 * RF_PTS; k++) acc[k][threadIdx.x] = 0.0;
    const RefineTypes &rt = S.rt;
    const int32_t nsl = S.nsl;
    const int64_t item = blockIdx.x;
    const int s = (int)(item % nsl);
    const int t = (int)((item / nsl) % rt.ntype);
    const int pg = (int)(item / ((int64_t)nsl * rt.ntype));
    const int64_t lo = rt.ts[t] + (int64_t)s * RF_SLICE;
    const int64_t hi = min(rt.ts[t + 1], lo + RF_SLICE);
    // axis A is the step axis, B the other one of a plane
    const auto axis = [](int a, auto x, auto y, auto z) { return a == 0 ? x : a == 1 ? y : z; };
    const int o1 = sa == 0 ? 1 : 0, o2 = 3 - sa - o1;
    const bool flat1 = axis(o1, box.f[0], box.f[1], box.f[2]) <= 1;
    const int sb = flat1 ? o2 : o1, sc = flat1 ? o1 : o2;
    // the points' indices along A, B and C; bit k of brk: point k is not point
    // k-1 plus one step along A
    __shared__ uint4 s_n[RF_PTS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int pk = pg * RF_PTS + lane;
    bool jump = false;
    if (lane < RF_PTS) {
        const int64_t p = pk < npts ? list[pk] : 0, q = pk > 0 && pk - 1 < npts ? list[pk - 1] : 0;
        const uint32_t c0 = (uint32_t)(p % box.f[0]), c1 = (uint32_t)((p / box.f[0]) % box.f[1]),
                       c2 = (uint32_t)(p / ((int64_t)box.f[0] * box.f[1]));
        const uint32_t e0 = (uint32_t)(q % box.f[0]), e1 = (uint32_t)((q / box.f[0]) % box.f[1]),
                       e2 = (uint32_t)(q / ((int64_t)box.f[0] * box.f[1]));
        if (wid == 0) s_n[lane] = make_uint4(axis(sa, c0, c1, c2), axis(sb, c0, c1, c2), axis(sc, c0, c1, c2), 0u);
        jump = pk >= npts || c0 != e0 + (sa == 0 ? 1u : 0u) || c1 != e1 + (sa == 1 ? 1u : 0u) ||
               c2 != e2 + (sa == 2 ? 1u : 0u);
        jump = jump && lane > 0;
    }
    const uint32_t brk = __ballot_sync(0xffffffffu, jump);
    __syncthreads();
    const int32_t n = (int32_t)max(hi - lo, (int64_t)0);
    const uint64_t *dA = axis(sa, S.du, S.dv, S.dw) + lo, *dB = axis(sb, S.du, S.dv, S.dw) + lo,
                   *dC = axis(sc, S.du, S.dv, S.dw) + lo;
    const bool fA = axis(sa, box.f[0], box.f[1], box.f[2]) > 1, fB = axis(sb, box.f[0], box.f[1], box.f[2]) > 1,
               third = axis(sc, box.f[0], box.f[1], box.f[2]) > 1;
    if (third)
        if (brk)
            refine_loop<false, true>(n, S.ph0 + lo, dA, dB, dC, S.w + lo, tab, s_n, acc, brk, fA, fB);
        else
            refine_loop<true, true>(n, S.ph0 + lo, dA, dB, dC, S.w + lo, tab, s_n, acc, 0, fA, fB);
    else if (brk)
        refine_loop<false, false>(n, S.ph0 + lo, dA, dB, dC, S.w + lo, tab, s_n, acc, brk, fA, fB);
    else
        refine_loop<true, false>(n, S.ph0 + lo, dA, dB, dC, S.w + lo, tab, s_n, acc, 0, fA, fB);
#pragma unroll
    for (int k = 0; k < RF_PTS; k++) {
        const double x = warp_sum(acc[2 * k][threadIdx.x]);
        const double y = warp_sum(acc[2 * k + 1][threadIdx.x]);
        if (lane == 0) {
            red[wid][k][0] = x;
            red[wid][k][1] = y;
        }
    }
    __syncthreads();
    if (threadIdx.x < RF_PTS) {
        const int k = threadIdx.x, pk = pg * RF_PTS + k;
        double x = 0.0, y = 0.0;
        for (int v = 0; v < RF_NT / 32; v++) {
            x += red[v][k][0];
            y += red[v][k][1];
        }
        if (pk < npts) S.out[((int64_t)pk * rt.ntype + t) * nsl + s] = make_double2(x, y);
    }
}

// csf, acsf and dsi of the listed points from the exact sums: the group sums
// sf (main atom set) and the type sums sa (folded atoms), as k_combine and
// k_aver_combine form them (closed-form lattice)
__global__ void k_refine_combine(const int32_t *__restrict__ list, int32_t npts, const FormSpec *fsm,
                                 const FormSpec *fst, BoxSpec box, const int32_t *__restrict__ istl,
                                 const double2 *__restrict__ cfact, const double2 *__restrict__ sf, int32_t nslf,
                                 const double2 *__restrict__ sa, int32_t nsla, int32_t c0, int32_t c1, int32_t c2,
                                 double d0, double d1, double d2, double norm, double ds, double sqds,
                                 double2 *__restrict__ csf, double2 *__restrict__ acsf, double *__restrict__ dsi)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= npts) return;
    const int64_t p = list[k];
    const int64_t i = p % box.f[0], j = (p / box.f[0]) % box.f[1], l = p / ((int64_t)box.f[0] * box.f[1]);
    const int64_t idx = i + (int64_t)box.num[0] * (j + (int64_t)box.num[1] * l);
    double h[3];
    form_hvec(fst, i, j, l, h);
    const int32_t q = istl ? istl[idx] : 0;
    double2 A = make_double2(0.0, 0.0);
    for (int t = 1; t <= fst->nscat; t++) {
        double2 s = make_double2(0.0, 0.0);
        for (int u = 0; u < nsla; u++) {
            const double2 v = sa[((int64_t)k * fst->nscat + (t - 1)) * nsla + u];
            s.x += v.x;
            s.y += v.y;
        }
        const double2 m = cmul(s, form_cfact(fst, cfact, q, t, h));
        A.x += m.x;
        A.y += m.y;
    }
    const double2 L = lattice_closed(h, c0, c1, c2, d0, d1, d2);
    const double2 av = cmul(A, L);
    const double2 a = make_double2(av.x * norm, av.y * norm);
    double2 F = make_double2(0.0, 0.0);
    for (int g = 1; g <= fsm->ngroup; g++) {
        double2 s = make_double2(0.0, 0.0);
        for (int u = 0; u < nslf; u++) {
            const double2 v = sf[((int64_t)k * fsm->ngroup + (g - 1)) * nslf + u];
            s.x += v.x;
            s.y += v.y;
        }
        const double2 m = cmul(s, form_group(fsm, cfact, q, g, h));
        F.x += m.x;
        F.y += m.y;
    }
    F.x -= a.x;
    F.y -= a.y;
    acsf[idx] = a;
    csf[idx] = make_double2(F.x * sqds, F.y * sqds);
    dsi[idx] = (F.x * F.x + F.y * F.y) * ds;
}

static void fill_types(RefineTypes &rt, const int64_t *ts, int32_t ntype)
{
    memset(&rt, 0, sizeof(rt));
    rt.ntype = ntype;
    for (int t = 0; t <= ntype; t++) rt.ts[t] = ts[t];
    for (int t = 0; t < ntype; t++) rt.n[t] = (double)ts[ntype + 1 + t];
}

static int32_t slices_of(const RefineTypes &rt)
{
    int64_t most = 1;
    for (int t = 0; t < rt.ntype; t++) most = std::max(most, rt.ts[t + 1] - rt.ts[t]);
    return (int32_t)dgpu_cdiv(most, RF_SLICE);
}

int dgpu_refine_aver(dgpu_ctx *ctx, const RefineSpec &r, double2 *csf, double2 *acsf, double *dsi, int64_t *nref)
{
    *nref = 0;
    const BoxSpec &box = r.box;
    const int64_t nb = (int64_t)box.f[0] * box.f[1] * box.f[2];
    if (nb < 1) return DGPU_OK;
    if (nb > 0x7fffffffLL) return dgpu_set_error(ctx, DGPU_ERR_ARG, "box too large for the refinement list");
    RefineTypes rm, ra;
    fill_types(rm, r.ts_main, r.ngroup);
    fill_types(ra, r.ts_fold, r.nscat);
    const FormSpec *d_fsm, *d_fst;
    int rc = dgpu_spec_device(ctx, 0, *r.fsm, &d_fsm);
    if (!rc) rc = dgpu_spec_device(ctx, 1, *r.fst, &d_fst);
    if (rc) return rc;
    // counters, the point list, the flags
    const size_t lbytes = ((size_t)nb * sizeof(int32_t) + 255) & ~(size_t)255;
    DGPU_CUDA(ctx, ctx->rlist.ensure(256 + lbytes + (size_t)nb));
    RefineCount *d_count = ctx->rlist.as<RefineCount>();
    int32_t *d_list = (int32_t *)((char *)ctx->rlist.p + 256);
    uint8_t *d_flag = (uint8_t *)ctx->rlist.p + 256 + lbytes;
    int32_t *h_out = static_cast<int32_t *>(ctx->stage.take(2 * sizeof(int32_t)));
    if (!h_out) return dgpu_set_error(ctx, DGPU_ERR_NOMEM, "pinned staging memory");
    const unsigned nblk = (unsigned)dgpu_cdiv(nb, 256);
    int32_t shortest = 0x7fffffff;                         // axis that the lines may run along
    for (int a = 0; a < 3; a++)
        if (box.f[a] >= 2) shortest = std::min(shortest, box.f[a]);
    const int64_t lines = dgpu_cdiv(nb, shortest);         // at most
    DGPU_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(RefineCount), ctx->stream));
    k_refine_select<<<nblk, 256, 0, ctx->stream>>>(d_fst, box, r.istl, r.cfact, acsf, ra, REFINE_TAU, d_flag);
    k_refine_adjacent<<<nblk, 256, 0, ctx->stream>>>(box, d_flag, d_count);
    k_refine_list<<<(unsigned)dgpu_cdiv(lines, 8), 256, 0, ctx->stream>>>(box, d_flag, d_count, d_list);
    k_refine_report<<<1, 1, 0, ctx->stream>>>(box, d_count, h_out);
    DGPU_CUDA(ctx, cudaGetLastError());
    DGPU_CUDA(ctx, cudaStreamSynchronize(ctx->stream));      // the number of points sizes what follows
    const int32_t npts = h_out[0], sa = h_out[1];
    if (npts == 0) return DGPU_OK;
    const int64_t ngrp = dgpu_cdiv(npts, RF_PTS);
    RefineSet sf = {r.ph0, r.du, r.dv, r.dw, r.w, rm, slices_of(rm), nullptr};
    RefineSet sg = {r.aph0, r.adu, r.adv, r.adw, r.aw, ra, slices_of(ra), nullptr};
    const int32_t nslf = sf.nsl, nsla = sg.nsl;
    DGPU_CUDA(ctx, ctx->rsum.ensure((size_t)npts * ((size_t)r.ngroup * nslf + (size_t)r.nscat * nsla) *
                                    sizeof(double2)));
    sf.out = ctx->rsum.as<double2>();
    sg.out = sf.out + (size_t)npts * r.ngroup * nslf;
    const int64_t itf = ngrp * r.ngroup * nslf, ita = ngrp * r.nscat * nsla;
    if (itf > 0x7fffffffLL || ita > 0x7fffffffLL) return dgpu_set_error(ctx, DGPU_ERR_ARG, "refinement too large");
    const float2 *d_tab = ctx->ph_tab.as<float2>();
    k_refine_sums<<<(unsigned)itf, RF_NT, 0, ctx->stream>>>(d_list, npts, box, sf, d_tab, sa);
    k_refine_sums<<<(unsigned)ita, RF_NT, 0, ctx->stream>>>(d_list, npts, box, sg, d_tab, sa);
    DGPU_CUDA(ctx, cudaGetLastError());
    k_refine_combine<<<(unsigned)dgpu_cdiv(npts, 128), 128, 0, ctx->stream>>>(
        d_list, npts, d_fsm, d_fst, box, r.istl, r.cfact, sf.out, nslf, sg.out, nsla, r.lat_n[0], r.lat_n[1], r.lat_n[2],
        r.lat_d[0], r.lat_d[1], r.lat_d[2], r.norm, r.diff_scale, sqrt(r.diff_scale), csf, acsf, dsi);
    DGPU_CUDA(ctx, cudaGetLastError());
    *nref = npts;
    return DGPU_OK;
}
