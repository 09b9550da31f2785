// Plain FP32 direct sum on CUDA cores.
//
// Replaces the hot loop of four_strucf_omp (discus/prog/four_strucf_OMP_mod.f90:155-182):
// for every grid point of the computed box and every atom of a type,
// phase = ph0 + n0*d0 + n1*d1 + n2*d2 (64-bit fixed point, exact mod 1),
// then w exp(2 pi i phase) in FP32 by table-driven angle addition
// (dgpu_phasor.cuh, the table in shared memory) accumulated in FP32 over one
// chunk of 128 atoms and in FP64 across chunks.  Each thread owns Q
// consecutive points along one grid axis, so consecutive points differ by one
// add.  In REF22 mode the phase keeps only its top 16 bits, the reference's
// (iarg >> 6) & 0xFFFF table index.
//
// Work split: blockIdx.x = point tile, blockIdx.y = group of chunks, blockIdx.z =
// atom type.  Each (type, group) writes its own partial sum part[t][s][p];
// the combine kernel adds the groups in a fixed order (deterministic).  The
// chunks are cut from slices whose length depends on the box and the types
// alone; a group is as many of them as leave a few waves of blocks, and a
// small box gives each thread fewer points: 1500 atoms on 51 x 101 points
// took 66 us on 36 blocks and take 18 us on 252, 1000 atoms on 7 x 13 x 13
// points 87 and 13 us.
//
// What bounds it: the FP32 pipe and instruction issue, each about two thirds
// busy, in dependent chains.  Pairs of points are evaluated and summed with
// packed FP32x2 instructions (the same roundings), REF22 phases in 32 bits,
// and several atoms are in flight per thread.  16 000 atoms in three groups
// on 31 x 45 x 31 points: 952 -> 666 us (shared-memory bank conflicts of the
// table and more resident blocks made no difference).
#include "dgpu_internal.h"
#include "dgpu_phasor.cuh"

#define DIR_NT 128
#define DIR_WAVE 5          // resident blocks per SM

struct DirectGeom {
    int32_t f[3];          // box
    int32_t a0, a1, a2;    // axis permutation, a0 = per-thread run axis
    int32_t nq;            // ceil(f[a0]/Q)
    int64_t nslots;        // nq * f[a1] * f[a2]
    int64_t pbox;          // f0*f1*f2
    int64_t slice_len;     // atoms per slice
    int32_t cps;           // chunks of DIR_NT atoms per slice
    int32_t nchunk;        // chunks per type: slices x cps
    int32_t group;         // chunks per work item
    int32_t ngroup;        // work items per type and point tile
    int64_t ts[65];        // type_start (0-based types)
};

// One atom's phase data in shared memory.  REF22 phases are multiples of
// 2^-22 turn, so that their top 32 bits hold them exactly.
template <bool REF>
struct PhaseWord {
    using T = uint64_t;
};
template <>
struct PhaseWord<true> {
    using T = uint32_t;
};

// Q consecutive points per thread along axis a0.  The FP32 sums and their
// Fast2Sum compensation are packed FP32x2 over pairs of points.
template <bool REF, int Q>
__global__ void __launch_bounds__(DIR_NT, DIR_WAVE)
k_direct(const uint64_t *__restrict__ ph0, const uint64_t *__restrict__ du,
         const uint64_t *__restrict__ dv, const uint64_t *__restrict__ dw,
         const float *__restrict__ w, const float2 *__restrict__ gtab, const __grid_constant__ DirectGeom g,
         double2 *__restrict__ part)
{
    using T = typename PhaseWord<REF>::T;
    __shared__ T s_b[DIR_NT], s_d0[DIR_NT], s_d1[DIR_NT], s_d2[DIR_NT];
    __shared__ float s_w[DIR_NT];
    __shared__ float tabs[2 * PH_TAB];
    // FP64 sums of the chunks, a column per thread: touched once per chunk,
    // and not worth the registers that more resident blocks can use
    __shared__ double accd[2 * Q][DIR_NT];
    for (int j = threadIdx.x; j < PH_TAB; j += DIR_NT) {
        const float2 v = gtab[j];
        tabs[j] = v.x;
        tabs[PH_TAB + j] = v.y;
    }

    const int t = blockIdx.z;
    const int c_lo = (int)blockIdx.y * g.group, c_hi = min(g.nchunk, c_lo + g.group);

    const int64_t slot = (int64_t)blockIdx.x * DIR_NT + threadIdx.x;
    const bool valid = slot < g.nslots;
    int32_t n[3] = {0, 0, 0};
    {
        int64_t sl = valid ? slot : 0;
        int32_t iq = (int32_t)(sl % g.nq);
        int64_t rest = sl / g.nq;
        n[g.a0] = iq * Q;
        n[g.a1] = (int32_t)(rest % g.f[g.a1]);
        n[g.a2] = (int32_t)(rest / g.f[g.a1]);
    }
    const uint32_t m0 = (uint32_t)n[g.a0], m1 = (uint32_t)n[g.a1], m2 = (uint32_t)n[g.a2];

#pragma unroll
    for (int k = 0; k < 2 * Q; k++) accd[k][threadIdx.x] = 0.0;

    for (int c = c_lo; c < c_hi; c++) {
        const int s = c / g.cps;
        const int64_t a_lo = g.ts[t] + (int64_t)s * g.slice_len;
        const int64_t a_hi = min(g.ts[t + 1], a_lo + g.slice_len);
        const int64_t base = a_lo + (int64_t)(c - s * g.cps) * DIR_NT;
        const int cnt = (int)min((int64_t)DIR_NT, a_hi - base);
        if (cnt <= 0) continue;                     // the same for every thread of the block
        __syncthreads();
        if (threadIdx.x < cnt) {
            const int64_t a = base + threadIdx.x;
            const uint64_t d[3] = {du[a], dv[a], dw[a]};
            constexpr int sh = REF ? 32 : 0;
            // REF22: the phase keeps its top 16 bits, the reference's table
            // index; adding half a table step does not reach the bits below
            // them, so the cut is made when the remainder is taken
            s_b[threadIdx.x] = REF ? (T)(ph0[a] >> 32) + (T)(PH_ROUND >> 32) : (T)(ph0[a] + PH_ROUND);
            s_d0[threadIdx.x] = (T)(d[g.a0] >> sh);
            s_d1[threadIdx.x] = (T)(d[g.a1] >> sh);
            s_d2[threadIdx.x] = (T)(d[g.a2] >> sh);
            s_w[threadIdx.x] = w[a];
        }
        __syncthreads();
        // FP32 sums over the chunk with Fast2Sum compensation: a coherent sum
        // of nearly equal terms would otherwise round with a bias that grows
        // with the chunk length (~ n 2^-24 of the sum)
        f32x2 acc[Q / 2][2], cmp[Q / 2][2];
#pragma unroll
        for (int k = 0; k < Q / 2; k++) acc[k][0] = acc[k][1] = cmp[k][0] = cmp[k][1] = 0ull;
        // several atoms in flight: the loads and the origin phase of the next
        // ones overlap the sums of this one
#pragma unroll 4
        for (int j = 0; j < cnt; j++) {
            const T d0 = s_d0[j];
            T ph = s_b[j] + m0 * d0 + m1 * s_d1[j] + m2 * s_d2[j];
            const PhWeight2 wj = ph_weight2(s_w[j]);
#pragma unroll
            for (int k = 0; k < Q / 2; k++) {
                const T qh = ph + d0;
                f32x2 e[2];
                if (REF)
                    ph_phasor2((uint32_t)ph >> 22, ((uint32_t)ph << 1) & 0x7E0000u, (uint32_t)qh >> 22,
                               ((uint32_t)qh << 1) & 0x7E0000u, tabs, wj, e[0], e[1]);
                else
                    ph_phasor2((uint32_t)((uint64_t)ph >> 54), (uint32_t)((uint64_t)ph >> 31) & 0x7FFFFFu,
                               (uint32_t)((uint64_t)qh >> 54), (uint32_t)((uint64_t)qh >> 31) & 0x7FFFFFu, tabs, wj,
                               e[0], e[1]);
#pragma unroll
                for (int x = 0; x < 2; x++) {
                    const f32x2 sum = add_f32x2(acc[k][x], e[x]);
                    cmp[k][x] = add_f32x2(cmp[k][x], sub_f32x2(e[x], sub_f32x2(sum, acc[k][x])));
                    acc[k][x] = sum;
                }
                ph = qh + d0;
            }
        }
#pragma unroll
        for (int k = 0; k < Q / 2; k++)
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const float2 a = unpack_f32(acc[k][x]), b = unpack_f32(cmp[k][x]);
                accd[4 * k + x][threadIdx.x] += (double)a.x + (double)b.x;
                accd[4 * k + 2 + x][threadIdx.x] += (double)a.y + (double)b.y;
            }
    }
    if (!valid) return;
    double2 *out = part + ((int64_t)t * g.ngroup + blockIdx.y) * g.pbox;
#pragma unroll
    for (int k = 0; k < Q; k++) {
        int32_t nn[3] = {n[0], n[1], n[2]};
        nn[g.a0] += k;
        if (nn[g.a0] >= g.f[g.a0]) break;
        int64_t p = nn[0] + (int64_t)g.f[0] * (nn[1] + (int64_t)g.f[1] * nn[2]);
        out[p] = make_double2(accd[2 * k][threadIdx.x], accd[2 * k + 1][threadIdx.x]);
    }
}

// Work items of the launch: point tiles x groups of chunks x types.  The
// chunks, the unit of the FP32 sums, follow from the slices (about eight
// blocks of 8 points per thread for every SM); how many of them one item adds
// in FP64, and how many points a thread owns, only decide how many blocks
// there are.
#define DIR_WAVES 4         // waves of blocks aimed at (2 cost 11% more time on the case below, 6 no less)

template <int Q>
static void launch_direct(dgpu_ctx *ctx, const uint64_t *ph0, const uint64_t *du, const uint64_t *dv,
                          const uint64_t *dw, const float *w, int32_t ref_mask, const DirectGeom &g, dim3 grid,
                          double2 *part)
{
    if (ref_mask)
        k_direct<true, Q><<<grid, DIR_NT, 0, ctx->stream>>>(ph0, du, dv, dw, w, ctx->ph_tab.as<float2>(), g, part);
    else
        k_direct<false, Q><<<grid, DIR_NT, 0, ctx->stream>>>(ph0, du, dv, dw, w, ctx->ph_tab.as<float2>(), g, part);
}

int dgpu_direct_sums(dgpu_ctx *ctx, const uint64_t *ph0, const uint64_t *du, const uint64_t *dv,
                     const uint64_t *dw, const float *w, const int64_t *h_type_start, int32_t ntype,
                     int32_t ref_mask, const BoxSpec &box, DevBuf &part, int32_t *nslice_out)
{
    if (ntype < 1 || ntype > 64) return dgpu_set_error(ctx, DGPU_ERR_ARG, "ntype=%d", ntype);
    DirectGeom g;
    memset(&g, 0, sizeof(g));
    for (int k = 0; k < 3; k++) g.f[k] = box.f[k];
    // run axis: the longest axis of the box
    int a0 = 0;
    for (int k = 1; k < 3; k++)
        if (box.f[k] > box.f[a0]) a0 = k;
    g.a0 = a0;
    g.a1 = (a0 + 1) % 3;
    g.a2 = (a0 + 2) % 3;
    g.pbox = (int64_t)box.f[0] * box.f[1] * box.f[2];
    int64_t maxn = 0;
    for (int t = 0; t < ntype; t++) {
        g.ts[t] = h_type_start[t];
        maxn = maxn > (h_type_start[t + 1] - h_type_start[t]) ? maxn : (h_type_start[t + 1] - h_type_start[t]);
    }
    g.ts[ntype] = h_type_start[ntype];
    const int64_t lines = (int64_t)box.f[g.a1] * box.f[g.a2];
    // slices and their chunks
    const int64_t tiles8 = dgpu_cdiv(dgpu_cdiv(box.f[a0], 8) * lines, DIR_NT);
    int64_t want = dgpu_cdiv(8LL * ctx->nsm, tiles8 * ntype);
    int64_t maxs = maxn / 256 > 1 ? maxn / 256 : 1;
    int64_t nslice = want < 1 ? 1 : (want > maxs ? maxs : want);
    if (nslice > 65535) nslice = 65535;
    g.slice_len = dgpu_cdiv(maxn > 0 ? maxn : 1, nslice);
    g.cps = (int32_t)dgpu_cdiv(g.slice_len, DIR_NT);
    const int64_t nchunk = nslice * g.cps;
    if (nchunk > 0x7fffffff) return dgpu_set_error(ctx, DGPU_ERR_ARG, "too many atoms");
    g.nchunk = (int32_t)nchunk;
    // fewer points per thread where eight leave the chip short of blocks
    // (8 points amortise an atom's loads and its origin phase best)
    const int64_t wave = (int64_t)DIR_WAVE * ctx->nsm;
    int q = 8;
    int64_t tiles = tiles8;
    while (q > 2 && tiles * ntype * nchunk < 2 * wave) {
        q /= 2;
        tiles = dgpu_cdiv(dgpu_cdiv(box.f[a0], q) * lines, DIR_NT);
    }
    g.nq = (int32_t)dgpu_cdiv(box.f[a0], q);
    g.nslots = g.nq * lines;
    int64_t groups = dgpu_cdiv(DIR_WAVES * wave, tiles * ntype);
    if (groups > nchunk) groups = nchunk;
    if (groups > 65535) groups = 65535;
    g.group = (int32_t)dgpu_cdiv(nchunk, groups);
    g.ngroup = (int32_t)dgpu_cdiv(nchunk, g.group);
    DGPU_CUDA(ctx, part.ensure((size_t)ntype * g.ngroup * g.pbox * sizeof(double2)));
    if (tiles > 0x7fffffff) return dgpu_set_error(ctx, DGPU_ERR_ARG, "grid too large");
    dim3 grid((unsigned)tiles, (unsigned)g.ngroup, (unsigned)ntype);
    double2 *out = part.as<double2>();
    if (q == 8) launch_direct<8>(ctx, ph0, du, dv, dw, w, ref_mask, g, grid, out);
    else if (q == 4) launch_direct<4>(ctx, ph0, du, dv, dw, w, ref_mask, g, grid, out);
    else launch_direct<2>(ctx, ph0, du, dv, dw, w, ref_mask, g, grid, out);
    DGPU_CUDA(ctx, cudaGetLastError());
    *nslice_out = g.ngroup;
    return DGPU_OK;
}
