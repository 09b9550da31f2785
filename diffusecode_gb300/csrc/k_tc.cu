// Tensor-core engine: the type sums as a split-precision complex GEMM on
// tcgen05 (sm_100 family), accumulators in TMEM.
//
// For the computed box, one grid axis ac is the GEMM's N dimension
// ("columns"); the other two, ra (the longer) and rb, flattened with ra padded
// to a multiple of 8 (fra_p), form its M dimension ("rows": rg = nb*fra_p+na).
// The phase of point (row, column c) and atom j splits exactly:
//     phase = [ph0_j + na d_ra,j + nb d_rb,j] + [n_c d_ac,j]
// so  S(row,c) = sum_j U[row,j] V[j,c]  with  U = w_j exp(2 pi i A-phase),
// V = exp(2 pi i B-phase); K = the atoms of one type (a slice of them per
// work item).
//
// Operand generation.  Each CTA generates its U tile (128 rows) in shared
// memory from the 64-bit fixed-point phases, and V either the same way (V
// generated in the kernel: planes, where an image would be read by fewer than
// four row tiles) or not at all: with V images (k_tc_vgen, written once per
// launch) a copy warp streams them into a ring.  Every producer warp owns a
// chunk of eight atoms of each stage and runs on its own.  A producer thread
// evaluates exp(2 pi i phase) at the start of a run of rows (or columns) (from
// the exact 64-bit phase) and then steps by the per-atom factors
// exp(2 pi i 8 d) and exp(2 pi i 16 d) (computed once per atom, rounded
// stochastically); a row run restarts from the exact phase wherever nb
// changes.  With V in the kernel the producers used to meet at a barrier per
// 32-atom stage; on their own, with 64-atom stages for N <= 64, the type sums
// of a population of 16 planes take 273 us instead of 364.  U is evaluated at
// phase + rot_j and V at phase - rot_j, a pseudo-random offset per atom
// (tc_rot): the product is the same, but the evaluation errors of atoms at
// equivalent positions no longer coincide (they would add up coherently).
// Every FP32 value is split into hi (the value with its mantissa cut to the
// fp16 / bf16 width, exact in that format) and lo (the exact remainder,
// rounded).  V is scaled by 2^12 so that its lo parts stay normal fp16
// numbers; all accumulators therefore carry 2^12, removed when they are
// drained.
//
// MMA form.  B holds the rows [Vr; Vi; -Vr] (3N rows), so per 16 atoms
//     D[:, 0:2N] += Ur [Vr;Vi]^T   and   D += (-Ui) [Vi;-Vr]^T
// give Re (accumulator columns 0..N-1) and Im (N..2N-1) with two MMAs of
// width 2N.  The (hi,hi) products go to the main accumulator, the (hi,lo) and
// (lo,hi) products to the correction accumulator.
//
// Accumulation.  Every MMA truncates its FP32 accumulator by about one ulp, so
// the error of one TMEM accumulator grows with the number of MMAs chained into
// it.  The main accumulator is therefore drained every `flush` stages
// (128 atoms) and added with round-to-nearest FP32 adds to a running sum
// (kept in TMEM when N <= 64, otherwise in the work item's partial in global
// memory); the small corrections accumulate over the whole work item.  With
// nbuf = 2 the main accumulator is double-buffered so that a drain overlaps the
// next chunk.  The combine kernels add the K slices of all work items in
// float-float (slice_sum, dgpu_form.cuh) or FP64.
//
// Partials: part[(t*nslice + ks)*slab + c*nrows_p + rg], a column-major image
// of the tile space (rows with na >= fra are never written).
//
// Warp roles (768 threads, six warpgroups): warps 0-15 produce operand stages
// in two sets of eight that take the stages in turn, warps 16-19 drain TMEM,
// warp 20 owns TMEM and issues the MMAs (one elected lane), warp 21 streams the
// V operand images into their ring (one lane).  The last two groups hand
// registers to the producers (96, 56 and 40 per thread instead of 80).  All
// waits are bounded (globaltimer); a wait that gives up sets an error flag,
// the CTA stops issuing, waits for its own MMAs, frees TMEM and returns.
//
// What bounds it, on the 500 000-atom, 101^3 volume: 4.38 ms on a cool chip,
// 4.65 in a long run, of which the MMAs alone need 3.73 and the producers alone
// about 4.2.  The MMAs are bound by the operand bytes they read from shared
// memory (128 B per cycle) more than by their 56 cycles; the main and the
// correction MMA of one A operand follow each other so that the second takes A
// from the collector buffer (3.92 -> 3.73).  The producers run out of issue
// slots and of latency to hide: with one set of eight warps they needed 5.05,
// with two of 80 registers 4.43; with 96 registers the next stage's atoms are
// loaded ahead, and the drain, which shares their schedulers, got by with half
// its instructions (packed adds, sixteen columns at a time): 4.83 -> 4.45; the
// atoms' phase offset stepped from stage to stage: 4.38.
// (Without the seeds of the chains it would be 0.6 ms less; computing the next
// chain's seeds early, eight groups per pass of the chain loop, or 104
// registers were all slower.)
//
// Shared-memory operands use the canonical K-major layouts: a row holds the
// 64 atoms of a stage (128 B) with the 128-byte swizzle (8-row groups 1024 B
// apart, the 16-byte chunk c of row r at chunk c ^ (r & 7)); where two such
// stages with V do not fit (V in the kernel, N > 64), 32 atoms (64 B) with the
// 64-byte swizzle (8-row groups 512 B apart, chunk c of row r at
// c ^ ((r & 7) >> 1)).
#include "dgpu_internal.h"

#define TC_KA 32                               // atoms per stage of 64-byte rows (V generated in the kernel, N > 64)
#define TC_KB 64                               // atoms per stage of 128-byte rows
#define TC_M 128
#define TC_SET_WARPS 8                         // producer warps of one stage
#define TC_PROD_WARPS (2 * TC_SET_WARPS)       // two sets, which take the stages in turn
#define TC_EPI_WARP0 TC_PROD_WARPS
#define TC_MMA_WARP (TC_EPI_WARP0 + 4)
#define TC_COPY_WARP (TC_MMA_WARP + 1)
#define TC_THREADS (TC_PROD_WARPS * 32 + 256)  // whole warpgroups: two warps of the last are idle
// Registers per thread of the producers, of the drain warps and of the last
// warpgroup.  Their sum over the six warpgroups is what the block is launched
// with (6 x 80, tested before the first launch): the producers' increase
// waits for the others' decrease and never for more than that.
#define TC_REG_PROD 96
#define TC_REG_EPI 56
#define TC_REG_MMA 40
#define TC_B_BYTES (TC_M * TC_KB * 2)          // one A operand (e.g. Ur_hi) of a 64-atom stage: 16 KB
#define TC_VSLOTS 2                            // V ring: 64-atom images, one stage ahead
#define TC_BAR_BYTES 256
#define TC_SMEM_MAX (227 * 1024)                // the opt-in maximum of one CTA
#define TC_SLICE_MAX ((int64_t)1 << 28)        // atoms of a work item
#define TC_FLUSH_ATOMS 128                     // atoms per drain of the main accumulator
#define TC_V_SCALE 4096.0f
#define TC_UNSCALE (1.0f / 4096.0f)

#include "dgpu_phasor.cuh"
#include "tc_ptx.cuh"

__device__ __forceinline__ void decode_item(const TcProblem &g, int64_t item, int &t, int &ks, int &nt, int &mt)
{
    mt = (int)(item % g.m_tiles);
    int64_t r = item / g.m_tiles;
    nt = (int)(r % g.n_tiles);
    r /= g.n_tiles;
    ks = (int)(r % g.nslice);
    t = (int)(r / g.nslice);
}

// Source arrays of one problem from an item's first atom on.  The pointers are
// the same on every lane (uniform registers) and an atom is a 32-bit byte
// offset from them, so that a load needs no 64-bit address arithmetic.
struct TcSrc {
    const uint64_t *ph0, *dra, *drb, *dac;
    const float *w;
    const float2 *ma, *mc, *ma2, *mc2;
};

template <class T>
__device__ __forceinline__ const T *uniform_ptr(const T *p)
{
    const uint64_t v = reinterpret_cast<uint64_t>(p);
    const uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)v, 0), hi = __shfl_sync(0xffffffffu, (uint32_t)(v >> 32), 0);
    return reinterpret_cast<const T *>((uint64_t)hi << 32 | lo);
}

template <class V, class T>
__device__ __forceinline__ V load_at(const T *base, uint32_t bytes)
{
    return __ldg(reinterpret_cast<const V *>(reinterpret_cast<const char *>(base) + bytes));
}

// Phase data of the thread's two atoms for one stage, loaded from global
// memory one stage ahead (16-byte loads: the atoms are consecutive and even).
struct AtomPair {
    ulonglong2 ph0, dra, drb;
    float2 w;
    float4 m;               // step factors exp(2 pi i 8 d_ra) of the two atoms
    float4 m2;              // and exp(2 pi i 16 d_ra)
};

__device__ __forceinline__ void load_pair(AtomPair &r, const TcSrc &P, uint32_t k)
{
    r.ph0 = load_at<ulonglong2>(P.ph0, 8 * k);
    r.dra = load_at<ulonglong2>(P.dra, 8 * k);
    r.drb = load_at<ulonglong2>(P.drb, 8 * k);
    r.w = load_at<float2>(P.w, 4 * k);
    r.m = load_at<float4>(P.ma, 8 * k);
    r.m2 = load_at<float4>(P.ma2, 8 * k);
}

// The same for the column axis (V generated in the kernel): loaded before the
// stage's U rows are generated, used after them.
struct ColPair {
    ulonglong2 dac;
    float4 m, m2;
};

__device__ __forceinline__ void load_cols(ColPair &r, const TcSrc &P, uint32_t k)
{
    r.dac = load_at<ulonglong2>(P.dac, 8 * k);
    r.m = load_at<float4>(P.mc, 8 * k);
    r.m2 = load_at<float4>(P.mc2, 8 * k);
}

// The groups of eight rows [q0, q1) of U and of eight columns [c0, c1) of V
// that a producer warp generates, and where their chains start from the exact
// phase: at every row group that begins a new nb and, with V generated in the
// kernel, at every `per`-th group of the list of row and column groups (the
// list is cut into four ranges of `per`, the unit that a warp takes).  gi, nb:
// place of group q0; rmask / cmask: bit q, a chain starts at group q.
struct WarpWork {
    int q0, q1, c0, c1, gi, nb, gpn;
    uint32_t rmask, cmask;
};

__device__ __forceinline__ WarpWork warp_work(int mt, int gpn, int N, bool vgen, bool halves, int half)
{
    const int ngr = TC_M / 8, ntot = ngr + (vgen ? N >> 3 : 0), per = (ntot + 3) >> 2;
    const int r0 = halves ? half * 2 * per : 0, r1 = halves && !half ? 2 * per : ntot;
    WarpWork k;
    k.q0 = min(r0, ngr);
    k.q1 = min(r1, ngr);
    k.c0 = max(r0, ngr) - ngr;
    k.c1 = max(r1, ngr) - ngr;
    const int G0 = mt * ngr + k.q0;
    k.gi = G0 % gpn;
    k.nb = G0 / gpn;
    k.gpn = gpn;
    k.rmask = k.cmask = 0;
    int gi = k.gi;
    for (int q = k.q0; q < k.q1; q++) {
        if (q > k.q0 && (gi == 0 || (vgen && q % per == 0))) k.rmask |= 1u << q;
        if (++gi == gpn) gi = 0;
    }
    for (int c = k.c0; c < k.c1; c++)
        if (c > k.c0 && (ngr + c) % per == 0) k.cmask |= 1u << c;
    return k;
}

// One chain of groups [q, qe): values x at group q, stepping from group to
// group by m on two chains (x and x m, each by m^2).
template <class Emit>
__device__ __forceinline__ void run_chain(int q, int qe, C2 x0, const M2 &m, const M2 &m2, Emit emit)
{
    C2 x1 = cmul2(x0, m);
#pragma unroll 1
    for (; q + 3 < qe; q += 4) {
        const C2 y0 = cmul2(x0, m2), y1 = cmul2(x1, m2);
        emit(q, x0);
        emit(q + 1, x1);
        x0 = cmul2(y0, m2);
        x1 = cmul2(y1, m2);
        emit(q + 2, y0);
        emit(q + 3, y1);
    }
    if (q + 1 < qe) {
        emit(q, x0);
        emit(q + 1, x1);
        if (q + 2 < qe) emit(q + 2, cmul2(x0, m2));
    } else if (q < qe) {
        emit(q, x0);
    }
}

// byte offset of (row r, 16-byte chunk c) in the operand layout of a KS-atom stage, and its 8-row group stride
template <int KS>
__device__ __forceinline__ uint32_t op_off(int r, int c)
{
    return KS == TC_KB ? sw128_off(r, c) : sw_off(r, c);
}
template <int KS>
__host__ __device__ constexpr uint32_t op_sbo()
{
    return KS == TC_KB ? TC_SBO128 : TC_SBO;
}

// U rows of one stage, stored with stmatrix: a warp generates its row groups
// for one chunk of eight atoms; lane l owns row l >> 2 of each group and atoms
// 2 (l & 3) + {0, 1} of the chunk, the fragment layout of an 8x8 b16 matrix,
// so that one stmatrix.x4 stores the four operand arrays (Ur hi, Ur lo, Ui hi,
// Ui lo) of one row group; adr is the lane's address in group 0 (array l >> 3,
// row l & 7).  Chains start from the exact phase and step from group to group
// by exp(2 pi i 8 d_ra).
//
// Four warps per scheduler run this, so its latency counts as much as its
// instructions.  The two atoms are stepped and split with packed FP32x2
// arithmetic (the same roundings), a group is stored as soon as it is split,
// and the chains are loops, with no test per group: on the 500 000-atom,
// 101^3 volume the producers alone (no MMA issued) took 6.58 ms before, with
// four groups collected per store and the segment tests between them, and
// 4.94 ms so.
template <bool BF, int KS>
__device__ __forceinline__ void gen_rows(const WarpWork &k, const AtomPair &ap, uint64_t rot0, uint32_t adr, int lane)
{
    const uint32_t s = (uint32_t)(lane >> 2);
    const uint64_t ph0[2] = {ap.ph0.x, ap.ph0.y}, dra[2] = {ap.dra.x, ap.dra.y}, drb[2] = {ap.drb.x, ap.drb.y};
    const float w[2] = {ap.w.x, ap.w.y};
    const uint64_t rot[2] = {rot0, rot0 + tc_rot(1)};
    const M2 m = factors2(make_float2(ap.m.x, ap.m.y), make_float2(ap.m.z, ap.m.w));
    const M2 m2 = factors2(make_float2(ap.m2.x, ap.m2.y), make_float2(ap.m2.z, ap.m2.w));
    auto emit = [&](int q, const C2 &x) {
        uint32_t rh, rl, ih, il;
        split2<BF>(x.re, rh, rl);
        split2<BF>(x.im, ih, il);
        stmatrix_x4(adr + (uint32_t)q * op_sbo<KS>(), rh, rl, ih, il);
    };
    uint32_t gi = (uint32_t)k.gi, nb = (uint32_t)k.nb, rest = k.rmask;
    for (int q = k.q0; q < k.q1;) {                // chains (warp-uniform)
        const int qe = rest ? __ffs(rest) - 1 : k.q1;
        rest &= rest - 1;
        const uint32_t na = gi * 8 + s;
        float2 p[2];
#pragma unroll
        for (int a = 0; a < 2; a++) {
            p[a] = phasor_fast(rot[a] + ph0[a] + (uint64_t)na * dra[a] + (uint64_t)nb * drb[a]);
            p[a] = make_float2(p[a].x * w[a], p[a].y * w[a]);
        }
        run_chain(q, qe, values2(p[0], p[1]), m, m2, emit);
        gi += (uint32_t)(qe - q);
        if (gi == (uint32_t)k.gpn) {
            gi = 0;
            nb++;
        }
        q = qe;
    }
}

// V columns of one stage (column n0 + 8 q + row of the lane), scaled by 2^12,
// as B rows Vr, Vi and -Vr of the hi and the lo operand: the first four by one
// stmatrix.x4 per column group (adr4: the lane's address in array l >> 3 of
// Vr hi, Vr lo, Vi hi, Vi lo), -Vr hi and lo by a stmatrix.x2 (adr2).  Chains
// step by exp(2 pi i 8 d_ac).
template <bool BF, int KS>
__device__ __forceinline__ void gen_cols(const WarpWork &k, const ColPair &cp, uint64_t rot0, uint32_t n0,
                                         uint32_t adr4, uint32_t adr2, int lane)
{
    const uint32_t s = (uint32_t)(lane >> 2);
    const M2 m = factors2(make_float2(cp.m.x, cp.m.y), make_float2(cp.m.z, cp.m.w));
    const M2 m2 = factors2(make_float2(cp.m2.x, cp.m2.y), make_float2(cp.m2.z, cp.m2.w));
    auto emit = [&](int q, const C2 &x) {
        uint32_t rh, rl, ih, il;
        split2<BF>(x.re, rh, rl);
        split2<BF>(x.im, ih, il);
        const uint32_t o = (uint32_t)q * op_sbo<KS>();
        stmatrix_x4(adr4 + o, rh, rl, ih, il);
        stmatrix_x2(adr2 + o, rh ^ 0x80008000u, rl ^ 0x80008000u);
    };
    uint32_t rest = k.cmask;
    for (int q = k.c0; q < k.c1;) {
        const int qe = rest ? __ffs(rest) - 1 : k.c1;
        rest &= rest - 1;
        const uint64_t nc = n0 + (uint32_t)q * 8 + s;
        const float2 p0 = phasor_fast(nc * cp.dac.x - rot0), p1 = phasor_fast(nc * cp.dac.y - (rot0 + tc_rot(1)));
        run_chain(q, qe,
                  values2(make_float2(p0.x * TC_V_SCALE, p0.y * TC_V_SCALE),
                          make_float2(p1.x * TC_V_SCALE, p1.y * TC_V_SCALE)),
                  m, m2, emit);
        q = qe;
    }
}

// A producer warp: generates its chunk of eight atoms of every second stage
// of the CTA's work items (KS = 64: eight chunks, one per warp of a set; KS =
// 32: four chunks of two warps, which share the groups).  The two sets take
// the stages in turn, so that four warps per scheduler hide each other's
// latency.  The warps run on their own: a warp loads its atoms' phase data,
// waits for its half of the stage buffer (a vote keeps the warp together if a
// wait gives up), writes, and lane 0 arrives on the half's full barrier.  A
// half is the atoms of the first or the second half of the stage's MMAs
// (barrier 2 s + h), which are refilled as soon as those have read them.
// Stage index and round are counted, not divided out of the stage count (S is
// a run-time value, and these loops are latency-bound).
template <bool BF, int KS, bool VGEN>
__device__ __forceinline__ void produce(const TcLaunch &L, uint32_t smem, uint32_t stage_bytes, uint64_t *full,
                                        uint64_t *empty, int warp, int lane, volatile int32_t *err)
{
    const uint32_t S = (uint32_t)L.stages, set = (uint32_t)warp / TC_SET_WARPS;
    const int wid = warp % TC_SET_WARPS;
    const int chunk = KS == TC_KB ? wid : wid & 3, part = KS == TC_KB ? 0 : wid >> 2;
    const uint32_t half = chunk >= KS / 16 ? 1u : 0u;
    const int kq = 8 * chunk + 2 * (lane & 3);          // the thread's first atom in a stage
    const uint32_t o0 = op_off<KS>(lane & 7, chunk), arr = (uint32_t)(lane >> 3);
    const uint32_t adr = smem + arr * (TC_M * KS * 2) + o0;
    uint32_t it = set, it0 = 0;                         // the set's next stage, the item's first (over all items)
    uint32_t sb = set, round = 0;                       // it = round * S + sb
    for (int64_t item = blockIdx.x; item < L.nitems; item += gridDim.x) {
        const TcProblem &g = L.probs[L.item_prob[item]];
        int t, ks, nt, mt;
        decode_item(g, item - g.item0, t, ks, nt, mt);
        const int64_t a0 = g.ts[t] + (int64_t)ks * g.slice_len;
        const int64_t a1 = min(g.ts[t + 1], a0 + g.slice_len);
        const int nst = warp_uniform(a1 > a0 ? (int)((a1 - a0) / KS) : 0);
        if (nst == 0) continue;
        const TcSrc src = {uniform_ptr(g.ph0 + a0), uniform_ptr(g.dra + a0), uniform_ptr(g.drb + a0),
                           VGEN ? uniform_ptr(g.dac + a0) : nullptr, uniform_ptr(g.w + a0), uniform_ptr(g.ma + a0),
                           VGEN ? uniform_ptr(g.mc + a0) : nullptr, uniform_ptr(g.ma2 + a0),
                           VGEN ? uniform_ptr(g.mc2 + a0) : nullptr};
        const int N = g.N;
        const WarpWork k = warp_work(mt, g.fra_p >> 3, N, VGEN, KS != TC_KB, part);
        const uint32_t b_bytes = (uint32_t)3 * L.Nmax * KS * 2, blk = (uint32_t)(N >> 3) * op_sbo<KS>();
        const uint32_t v0 = smem + 4u * TC_M * KS * 2 + o0 + (arr & 1) * b_bytes;
        AtomPair nx;
        if (it < it0 + (uint32_t)nst) load_pair(nx, src, (it - it0) * KS + (uint32_t)kq);
        uint64_t rot = tc_rot((uint64_t)(a0 + (int64_t)(it - it0) * KS + kq));
        for (; it < it0 + (uint32_t)nst; it += 2, rot += tc_rot(2 * KS)) {
            const uint32_t a = (it - it0) * KS + (uint32_t)kq;           // from a0
            const AtomPair ap = nx;
            load_pair(nx, src, it + 2 < it0 + (uint32_t)nst ? a + 2 * KS : a);
            ColPair cp;
            if (VGEN) load_cols(cp, src, a);
            const bool got =
                round == 0 || mbar_wait(&empty[2 * sb + half], (round - 1) & 1, err, 1, L.timeout_ns);
            if (!__all_sync(0xffffffffu, got)) return;
            gen_rows<BF, KS>(k, ap, rot, adr + sb * stage_bytes, lane);
            if (VGEN)
                gen_cols<BF, KS>(k, cp, rot, (uint32_t)(nt * N), v0 + (arr >> 1) * blk + sb * stage_bytes,
                                 v0 + 2 * blk + sb * stage_bytes, lane);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[2 * sb + half]);      // one arrival per producer warp
            for (sb += 2; sb >= S; sb -= S) round++;
        }
        it0 += (uint32_t)nst;
    }
}

// a += b of two FP32 values in 32-bit words
__device__ __forceinline__ void add_words(uint32_t &a0, uint32_t &a1, uint32_t b0, uint32_t b1)
{
    const float2 v = unpack_f32(add_f32x2(pack_f32(__uint_as_float(a0), __uint_as_float(a1)),
                                          pack_f32(__uint_as_float(b0), __uint_as_float(b1))));
    a0 = __float_as_uint(v.x);
    a1 = __float_as_uint(v.y);
}

// KS: atoms per stage; VRING: the V operand streamed from images (KS = 64)
template <bool BF, int KS, bool VRING>
__global__ void __launch_bounds__(TC_THREADS, 1) k_tc(const TcLaunch L)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int S = L.stages;
    const int NM = L.Nmax;
    const uint32_t b_bytes = (uint32_t)3 * NM * KS * 2;         // one B operand: 3N rows
    // stages hold U (and V when it is generated in-kernel); with V images,
    // V lives in a ring of TC_VSLOTS slots of 2 * b_bytes after the stages
    const uint32_t stage_bytes = 4u * TC_M * KS * 2 + (VRING ? 0u : 2 * b_bytes);
    const uint32_t vbytes = 2 * b_bytes;
    uint8_t *vring = smem + (size_t)S * stage_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(vring + (VRING ? (size_t)TC_VSLOTS * vbytes : 0));
    uint64_t *empty = full + 2 * S;   // [2 S] both per half of a stage
    uint64_t *mfull = empty + 2 * S;  // [2] main accumulator b ready
    uint64_t *mempty = mfull + 2;     // [2] main accumulator b drained
    uint64_t *cfull = mempty + 2;     // correction accumulator ready (end of item)
    uint64_t *cempty = cfull + 1;     // correction accumulator drained
    uint64_t *drain = cempty + 1;
    uint64_t *vfull = drain + 1;      // [TC_VSLOTS] V image of the slot landed
    uint64_t *vempty = vfull + TC_VSLOTS;   // [TC_VSLOTS] MMAs reading the slot done
    uint32_t *tbase = reinterpret_cast<uint32_t *>(vempty + TC_VSLOTS);
    volatile int32_t *err = L.err;

    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2 * S; s++) {
            mbar_init(&full[s], TC_SET_WARPS / 2);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&mfull[b], 1);
            mbar_init(&mempty[b], 4 * 32);
        }
        mbar_init(cfull, 1);
        mbar_init(cempty, 4 * 32);
        mbar_init(drain, 1);
        for (int v = 0; v < TC_VSLOTS; v++) {
            mbar_init(&vfull[v], 1);
            mbar_init(&vempty[v], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TC_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tbase)),
                     "r"(L.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tbase;

    if (warp < TC_PROD_WARPS) {
        setmaxnreg_inc<TC_REG_PROD>();
        // ------------------------------------------------------------ producers
        produce<BF, KS, !VRING>(L, smem_u32(smem), stage_bytes, full, empty, warp, lane, err);
    } else if (warp >= TC_MMA_WARP) {
        setmaxnreg_dec<TC_REG_MMA>();
        if (warp == TC_MMA_WARP) {
            // -------------------------------------------------------- MMA issuer
            // The whole warp runs the loop and one elected lane issues and
            // commits (a predicate on the instruction): in warp-uniform control
            // flow the operand descriptors stay in uniform registers, where a
            // branch taken by one lane had them moved there for every MMA (95
            // cycles per MMA; 77 so, with nothing else running).
            const uint32_t lead = elect_lane();
            bool issued = false;
            {
                const uint32_t fmt = BF ? 1u : 0u;
                const uint32_t c_acc = tmem;                                  // correction accumulator
                uint32_t it = 0, nitem = 0, nchunk = 0, s = 0, round = 0;   // it = round * S + s
                bool ok = true;
                for (int64_t item = blockIdx.x; item < L.nitems && ok; item += gridDim.x) {
                    const TcProblem &g = L.probs[L.item_prob[item]];
                    const int N = warp_uniform(g.N);
                    int t, ks, nt, mt;
                    decode_item(g, item - g.item0, t, ks, nt, mt);
                    const int64_t a0 = g.ts[t] + (int64_t)ks * g.slice_len;
                    const int64_t a1 = min(g.ts[t + 1], a0 + g.slice_len);
                    const int nst = warp_uniform(a1 > a0 ? (int)((a1 - a0) / KS) : 0);
                    if (nst == 0) continue;
                    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)((2 * N) >> 3) << 17) |
                                           ((uint32_t)(TC_M >> 4) << 24);
                    const uint32_t idesc_neg = idesc | (1u << 13);     // negate A: the -Ui products
                    const uint32_t b2off = (uint32_t)(N >> 3) * (KS == TC_KB ? TC_SBO128 : TC_SBO);
                    if (nitem > 0 && !__all_sync(0xffffffffu, mbar_wait(cempty, (nitem - 1) & 1, err, 2, L.timeout_ns))) {
                        ok = false;
                        break;
                    }
                    for (int st0 = 0; st0 < nst && ok; st0 += L.flush, nchunk++) {
                        const uint32_t b = L.nbuf == 2 ? nchunk & 1u : 0u;
                        const uint32_t use = L.nbuf == 2 ? nchunk >> 1 : nchunk;
                        if (use > 0 && !__all_sync(0xffffffffu, mbar_wait(&mempty[b], (use - 1) & 1, err, 6, L.timeout_ns))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t m_acc = tmem + 2u * NM * (1u + b);
                        const int st1 = min(nst, st0 + L.flush);
                        for (int st = st0; st < st1; st++, it++) {
                            const uint32_t A = smem_u32(smem) + s * stage_bytes;
                            const uint32_t Bh =
                                VRING ? smem_u32(vring) + (it % TC_VSLOTS) * vbytes : A + 4u * TC_M * (uint32_t)KS * 2u;
                            const uint64_t dA = KS == TC_KB ? sdesc128(A) : sdesc(A);
                            const uint64_t dB = KS == TC_KB ? sdesc128(Bh) : sdesc(Bh);
                            const uint64_t bl_off = b_bytes >> 4, b2_off = b2off >> 4;
                            constexpr uint32_t a_bytes = TC_M * KS * 2;
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                bool got = mbar_wait(&full[2 * s + h], round & 1, err, 3, L.timeout_ns);
                                if (VRING && h == 0)
                                    got = got &&
                                          mbar_wait(&vfull[it % TC_VSLOTS], (it / TC_VSLOTS) & 1, err, 8, L.timeout_ns);
                                ok = __all_sync(0xffffffffu, got);
                                if (!ok) break;
                                tc_fence_after();
                                // descriptors: the start-address field (addr >> 4, 14 bits) is the
                                // low field, and every operand lies below 256 KB, so an offset is a
                                // plain add to the base descriptor; a K step of 16 atoms is 32 bytes
#pragma unroll
                                for (int kk = h * KS / 32; kk < (h + 1) * KS / 32; kk++) {
                                    const uint64_t ko = (uint64_t)kk * 2;
                                    const uint64_t arh = dA + ko, arl = dA + (a_bytes >> 4) + ko;
                                    const uint64_t aih = dA + (2 * a_bytes >> 4) + ko, ail = dA + (3 * a_bytes >> 4) + ko;
                                    const uint64_t b1h = dB + ko, b2h = dB + b2_off + ko;
                                    const uint64_t b1l = dB + bl_off + ko, b2l = dB + bl_off + b2_off + ko;
                                    const uint32_t am = (st > st0 || kk > 0) ? 1u : 0u;   // main restarts per chunk
                                    const uint32_t ac = (st > 0 || kk > 0) ? 1u : 0u;     // correction per item
                                    // main (hi,hi) and correction (hi,lo) of one A, then the corrections (lo,hi)
                                    mma_f16_lead_pair(m_acc, b1h, am, c_acc, b1l, ac, arh, idesc, lead);
                                    mma_f16_lead_pair(m_acc, b2h, 1u, c_acc, b2l, 1u, aih, idesc_neg, lead);
                                    mma_f16_lead(c_acc, arl, b1h, idesc, 1u, lead);
                                    mma_f16_lead(c_acc, ail, b2h, idesc_neg, 1u, lead);
                                }
                                mma_commit_lead(&empty[2 * s + h], lead);
                                issued = true;
                            }
                            if (!ok) break;
                            if (VRING) mma_commit_lead(&vempty[it % TC_VSLOTS], lead);
                            if (++s == (uint32_t)S) {
                                s = 0;
                                round++;
                            }
                        }
                        if (!ok) break;
                        mma_commit_lead(&mfull[b], lead);
                    }
                    if (!ok) break;
                    mma_commit_lead(cfull, lead);
                    nitem++;
                }
                // make sure no MMA of this CTA is still running before TMEM is freed
                if (issued) {
                    mma_commit_lead(drain, lead);
                    mbar_wait_quiet(drain, 0);
                }
            }
            __syncwarp();
            tc_fence_before();
        } else if (warp == TC_COPY_WARP) {
            // ------------------------------------------------------------ V copies
            // Lane 0 streams the V operand images of every stage into the ring, up
            // to TC_VSLOTS stages ahead of the MMAs: a slot is refilled once the
            // MMAs that read it have completed.  Off the producers' path, so that
            // their stage barrier never waits for a slot.
            if (VRING && lane == 0) {
                uint32_t x = 0, landed = 0;       // copies issued / first copy not known to have landed
                bool ok = true;
                for (int64_t item = blockIdx.x; item < L.nitems && ok; item += gridDim.x) {
                    const TcProblem &g = L.probs[L.item_prob[item]];
                    int t, ks, nt, mt;
                    decode_item(g, item - g.item0, t, ks, nt, mt);
                    const int64_t a0 = g.ts[t] + (int64_t)ks * g.slice_len;
                    const int64_t a1 = min(g.ts[t + 1], a0 + g.slice_len);
                    const int nst = a1 > a0 ? (int)((a1 - a0) / TC_KB) : 0;
                    const int64_t g0 = a0 / TC_KB;
                    for (int y = 0; y < nst; y++, x++) {
                        const int v = (int)(x % TC_VSLOTS);
                        if (x >= TC_VSLOTS) {
                            if (!mbar_wait(&vempty[v], ((x / TC_VSLOTS) - 1) & 1, err, 9, L.timeout_ns)) {
                                ok = false;
                                break;
                            }
                            landed = x - TC_VSLOTS + 1;       // the MMAs consumed that copy: it landed
                        }
                        mbar_arrive_tx(&vfull[v], vbytes);
                        bulk_g2s(vring + (size_t)v * vbytes, g.vimg + ((g0 + y) * g.vstride + nt) * (int64_t)vbytes,
                                 vbytes, &vfull[v]);
                    }
                }
                // copies still in flight land before the CTA can exit (after an
                // error the MMA side may not have waited for them)
                for (uint32_t y = landed; y < x; y++) mbar_wait_quiet(&vfull[y % TC_VSLOTS], (y / TC_VSLOTS) & 1);
            }
            __syncwarp();
        }
    } else {
        setmaxnreg_dec<TC_REG_EPI>();
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3;                       // TMEM lane quadrant of this warp
        const int r = q * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const uint32_t t_corr = tmem + lane_off;
        const uint32_t t_sum = tmem + lane_off + 2u * NM * (1u + (uint32_t)L.nbuf);
        uint32_t nitem = 0, nchunk = 0;
        bool ok = true;
        for (int64_t item = blockIdx.x; item < L.nitems && ok; item += gridDim.x) {
            const TcProblem &g = L.probs[L.item_prob[item]];
            const int N = g.N;
            int t, ks, nt, mt;
            decode_item(g, item - g.item0, t, ks, nt, mt);
            const int64_t a0 = g.ts[t] + (int64_t)ks * g.slice_len;
            const int64_t a1 = min(g.ts[t + 1], a0 + g.slice_len);
            const int nst = a1 > a0 ? (int)((a1 - a0) / KS) : 0;
            const int64_t rg = (int64_t)mt * TC_M + r;
            const bool rv = rg < g.nrows_p && (int)(rg % g.fra_p) < g.fra;
            const int64_t nrp = g.nrows_p;
            const int ncv = min(N, g.ncols - nt * N);             // valid columns of this tile
            float2 *oc = g.part + ((int64_t)t * g.nslice + ks) * g.slab + (int64_t)nt * N * nrp + rg;
            if (nst == 0) {
                if (rv)
                    for (int c = 0; c < ncv; c++) oc[(int64_t)c * nrp] = make_float2(0.f, 0.f);
                continue;
            }
            for (int st0 = 0; st0 < nst; st0 += L.flush, nchunk++) {
                const int b = (int)(nchunk % L.nbuf);
                const bool got = lane == 0 ? mbar_wait(&mfull[b], (nchunk / L.nbuf) & 1, err, 5, L.timeout_ns) : true;
                if (!__shfl_sync(0xffffffffu, got, 0)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const bool first = st0 == 0, last = st0 + L.flush >= nst;
                if (last) {                                        // the item's corrections
                    const bool gc = lane == 0 ? mbar_wait(cfull, nitem & 1, err, 7, L.timeout_ns) : true;
                    if (!__shfl_sync(0xffffffffu, gc, 0)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                }
                const uint32_t t_main = tmem + lane_off + 2u * NM * (1u + (uint32_t)b);
                const bool keep = L.tsum && !last;                 // running sum stays in TMEM
                if (keep) {
                    // sixteen columns at a time, real and imaginary parts alike: few registers
                    for (int c = 0; c < 2 * N; c += 16) {
                        uint32_t v[16];
                        tmem_ld(t_main + (uint32_t)c, v);
                        if (!first) {
                            uint32_t a[16];
                            tmem_ld(t_sum + (uint32_t)c, a);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 16; k += 2) add_words(v[k], v[k + 1], a[k], a[k + 1]);
                        } else {
                            tmem_wait_ld();
                        }
                        tmem_st(t_sum + (uint32_t)c, v);
                    }
                    tmem_wait_st();
                } else {
                    for (int c0 = 0; c0 < N; c0 += 8) {
                        uint32_t vr[8], vi[8];
                        tmem_ld(t_main + (uint32_t)c0, vr);
                        tmem_ld(t_main + (uint32_t)(N + c0), vi);
                        auto add = [&](uint32_t t) {
                            uint32_t ar[8], ai[8];
                            tmem_ld(t + (uint32_t)c0, ar);
                            tmem_ld(t + (uint32_t)(N + c0), ai);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 8; k += 2) {
                                add_words(vr[k], vr[k + 1], ar[k], ar[k + 1]);
                                add_words(vi[k], vi[k + 1], ai[k], ai[k + 1]);
                            }
                        };
                        if (L.tsum && !first)
                            add(t_sum);
                        else
                            tmem_wait_ld();
                        if (last) add(t_corr);
                        if (rv) {
#pragma unroll
                            for (int k = 0; k < 8; k++) {
                                if (c0 + k < ncv) {
                                    float2 *o = oc + (int64_t)(c0 + k) * nrp;
                                    float2 v = make_float2(__uint_as_float(vr[k]) * TC_UNSCALE,
                                                           __uint_as_float(vi[k]) * TC_UNSCALE);
                                    if (!L.tsum && !first) {
                                        const float2 old = *o;
                                        v.x += old.x;
                                        v.y += old.y;
                                    }
                                    *o = v;
                                }
                            }
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive(&mempty[b]);
                if (last) mbar_arrive(cempty);
            }
            if (!ok) break;
            nitem++;
        }
    }
    __syncthreads();
    if (warp == TC_MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L.tmem_cols)
                     : "memory");
    }
}

// FP64 -> FP32 with stochastic rounding, in integer arithmetic on the bits:
// the 29 significand bits that FP32 drops get a uniform 29-bit draw added
// (u >> 3) and are cut off, so the magnitude rounds up (a carry, which may
// run into the exponent) with probability equal to its distance from the
// lower neighbour in units of the spacing, and the rounding error has mean
// zero over draws.  The FP32 word is then assembled from sign, rebased
// exponent and the top 23 significand bits (no FP64 instruction: this part's
// FP64 rate is low).  For |y| in the normal FP32 range; zero stays zero.
__device__ __forceinline__ float round_stochastic(double y, uint32_t u)
{
    uint64_t b = (uint64_t)__double_as_longlong(y);
    const int e0 = (int)((b >> 52) & 0x7FF);
    if (e0 < 1023 - 125) return __uint_as_float((uint32_t)(b >> 32) & 0x80000000u);   // |y| < 2^-125: zero
    b += (uint64_t)(u >> 3);
    const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
    const uint32_t e = (uint32_t)((b >> 52) & 0x7FF) - 1023u + 127u;
    const uint32_t man = (uint32_t)(b >> 29) & 0x7FFFFFu;
    return __uint_as_float(sign | (e << 23) | man);
}

// exp(2 pi i t) for a 64-bit fixed-point turn t, in FP64 to about 1e-16:
// the table entry of its top 12 bits (tab[k] = exp(2 pi i k / 4096)) times
// exp(i e) of the remaining angle e < 2 pi 2^-12, by its Taylor series
// (the first omitted terms are below 1e-16).
__device__ __forceinline__ double2 phasor_f64(uint64_t t, const double2 *__restrict__ tab)
{
    const double2 a = tab[t >> 52];
    const double e = (double)(t & 0xFFFFFFFFFFFFFull) * (6.283185307179586 * 0x1p-64);
    const double e2 = e * e;
    const double c = 1.0 - e2 * (0.5 - e2 * (1.0 / 24.0));
    const double s = e * (1.0 - e2 * (1.0 / 6.0));
    return make_double2(a.x * c - a.y * s, a.x * s + a.y * c);
}

__global__ void k_tc_tab(double2 *tab)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 4096) return;
    double s, c;
    sincospi((double)k / 2048.0, &s, &c);
    tab[k] = make_double2(c, s);
}

// the CUDA-core engines' phasor table (dgpu_phasor.cuh): exp(2 pi i j / 1024)
// rounded to FP32, entry 4j of the table above
__global__ void k_ph_tab(const double2 *__restrict__ tc_tab, float2 *__restrict__ tab)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < PH_TAB) tab[j] = make_float2((float)tc_tab[4 * j].x, (float)tc_tab[4 * j].y);
}

__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Per-atom step factors exp(2 pi i 8 d) and exp(2 pi i 16 d) along the three
// grid axes: FP64 values (table and Taylor series; the square of the first
// for the second), rounded stochastically to FP32 (a draw per atom and
// component).  The producers step a row by these
// factors up to 16 times, so a factor's rounding error recurs in every value
// of the chain; atoms at equivalent positions have identical increments, and
// with round-to-nearest their chains would share one error and add it up
// coherently.  Stochastic rounding gives each atom its own, zero-mean error.
// mask: bit a set for each axis a whose factors are written.
__global__ void k_tc_mult(const uint64_t *__restrict__ du, const uint64_t *__restrict__ dv,
                          const uint64_t *__restrict__ dw, int64_t n, int64_t stride,
                          const double2 *__restrict__ tab, float2 *__restrict__ out, int mask)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t *d[3] = {du, dv, dw};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (!((mask >> a) & 1)) continue;
        const double2 m = phasor_f64(d[a][i] << 3, tab);
        const double2 m2 = make_double2(m.x * m.x - m.y * m.y, 2.0 * m.x * m.y);
        const uint64_t r = mix64((uint64_t)i * 4u + (uint64_t)a + 0x9E3779B97F4A7C15ull);
        const uint64_t q = mix64(r);
        out[a * stride + i] = make_float2(round_stochastic(m.x, (uint32_t)r), round_stochastic(m.y, (uint32_t)(r >> 32)));
        out[(3 + a) * stride + i] =
            make_float2(round_stochastic(m2.x, (uint32_t)q), round_stochastic(m2.y, (uint32_t)(q >> 32)));
    }
}

// V operand images: for every (64-atom group gi, column tile nt) the B rows
// [Vr; Vi; -Vr] (hi operand, then lo) of the tile's N columns, in the
// 128-byte-swizzled K-major layout the MMAs read (768 N bytes).  Each value is
// evaluated from its exact 64-bit phase; grid: one block per (gi, nt).  A
// half-warp takes the 16 atom quads of one column, i.e. one 128-byte row of
// each of the six row blocks, so every 8-byte store instruction of a warp
// fills two whole rows and goes straight to global memory (no staging in
// shared memory, no block barrier: the warps' evaluation and stores overlap).
template <bool BF>
__global__ void __launch_bounds__(256) k_tc_vgen(const uint64_t *__restrict__ dac, int N, int n_tiles,
                                                  uint8_t *__restrict__ vimg)
{
    constexpr int NQ = TC_KB / 4;      // atom quads per row
    const int64_t gi = blockIdx.x / n_tiles;
    const int nt = (int)(blockIdx.x % n_tiles);
    const uint32_t vbytes = (uint32_t)N * 768u;
    uint8_t *img = vimg + (int64_t)blockIdx.x * vbytes;
    const uint32_t half = vbytes / 2, blk = (uint32_t)(N >> 3) * TC_SBO128;
    for (int u = threadIdx.x; u < N * NQ; u += blockDim.x) {
        const int c = u / NQ, jq = u % NQ;                     // column, atom quad
        const uint32_t nc = (uint32_t)(nt * N + c);
        float2 x[4];
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const int64_t j = gi * TC_KB + 4 * jq + a;
            const float2 p = phasor_acc((uint64_t)nc * dac[j] - tc_rot((uint64_t)j));
            x[a] = make_float2(p.x * TC_V_SCALE, p.y * TC_V_SCALE);
        }
        uint2 rh, rl, ih, il;
        split4<BF>(x[0].x, x[1].x, x[2].x, x[3].x, rh, rl);
        split4<BF>(x[0].y, x[1].y, x[2].y, x[3].y, ih, il);
        uint8_t *d = img + sw128_off(c, jq >> 1) + (jq & 1) * 8;
        *reinterpret_cast<uint2 *>(d) = rh;
        *reinterpret_cast<uint2 *>(d + half) = rl;
        *reinterpret_cast<uint2 *>(d + blk) = ih;
        *reinterpret_cast<uint2 *>(d + blk + half) = il;
        *reinterpret_cast<uint2 *>(d + 2 * blk) = make_uint2(rh.x ^ 0x80008000u, rh.y ^ 0x80008000u);
        *reinterpret_cast<uint2 *>(d + 2 * blk + half) = make_uint2(rl.x ^ 0x80008000u, rl.y ^ 0x80008000u);
    }
}

// ---------------------------------------------------------------------------
int dgpu_tc_init(dgpu_ctx *ctx)
{
    DGPU_CUDA(ctx, ctx->tc_tab.ensure(4096 * sizeof(double2)));
    k_tc_tab<<<16, 256, 0, ctx->stream>>>(ctx->tc_tab.as<double2>());
    DGPU_CUDA(ctx, cudaGetLastError());
    DGPU_CUDA(ctx, ctx->ph_tab.ensure(PH_TAB * sizeof(float2)));
    k_ph_tab<<<PH_TAB / 256, 256, 0, ctx->stream>>>(ctx->tc_tab.as<double2>(), ctx->ph_tab.as<float2>());
    DGPU_CUDA(ctx, cudaGetLastError());
    DGPU_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DGPU_OK;
}

bool dgpu_tc_available(dgpu_ctx *ctx)
{
    if (ctx->tc_avail < 0) {
        cudaDeviceProp p;
        ctx->tc_avail = (cudaGetDeviceProperties(&p, ctx->device) == cudaSuccess && p.major == 10) ? 1 : 0;
    }
    return ctx->tc_avail == 1;
}

static uint32_t pow2_cols(int n)
{
    uint32_t c = 32;
    while (c < (uint32_t)n) c <<= 1;
    return c;
}

// row axes for a column axis: ra is the longer of the other two
static void tc_row_axes(const BoxSpec &box, int ac, int &ra, int &rb)
{
    const int a = ac == 0 ? 1 : 0, b = 3 - ac - a;
    if (box.f[b] > box.f[a]) { ra = b; rb = a; }
    else { ra = a; rb = b; }
}

// padded MMA area of a column axis / tile width
static double tc_area(const BoxSpec &box, int ac, int N)
{
    const int64_t npts = (int64_t)box.f[0] * box.f[1] * box.f[2];
    const int nc = box.f[ac];
    if (nc < 2 && npts != nc) return -1.0;
    int ra, rb;
    tc_row_axes(box, ac, ra, rb);
    const int64_t rows = (int64_t)dgpu_cdiv(box.f[ra], 8) * 8 * box.f[rb];
    return (double)dgpu_cdiv(nc, N) * N * dgpu_cdiv(rows, TC_M) * TC_M;
}

// Geometry of one problem for a column axis, tile width and slicing.
// slice_atoms > 0: K slices of about that many atoms (a multi-problem launch,
// where the items of all problems share the SMs), else about slice_mult
// work items per SM for this problem alone
static void tc_problem(dgpu_ctx *ctx, const TcInput &in, const dgpu_opts *op, int axis, int N, int slice_mult,
                       int64_t slice_atoms, TcProblem &g)
{
    memset(&g, 0, sizeof(g));
    const BoxSpec &box = in.box;
    for (int k = 0; k < 3; k++) g.f[k] = box.f[k];
    g.ac = axis;
    tc_row_axes(box, axis, g.ra, g.rb);
    g.ncols = box.f[axis];
    g.fra = box.f[g.ra];
    g.fra_p = (int32_t)dgpu_cdiv(g.fra, 8) * 8;
    g.frb = box.f[g.rb];
    g.nrows_p = (int64_t)g.fra_p * g.frb;
    g.N = N;
    g.n_tiles = (int32_t)dgpu_cdiv(g.ncols, N);
    g.vstride = g.n_tiles;
    g.m_tiles = (int32_t)dgpu_cdiv(g.nrows_p, TC_M);
    g.slab = g.nrows_p * g.ncols;
    g.ntype = in.ntype;
    int64_t maxn = 0;
    for (int t = 0; t < in.ntype; t++) {
        g.ts[t] = in.ts[t];
        const int64_t n = in.ts[t + 1] - in.ts[t];
        maxn = n > maxn ? n : maxn;
    }
    g.ts[in.ntype] = in.ts[in.ntype];
    // K slices: about slice_mult work items per SM, or tc_kslice atoms each when given
    const int64_t tiles = (int64_t)g.m_tiles * g.n_tiles * in.ntype;
    int64_t nsl;
    if (op->tc_kslice > 0) {
        nsl = dgpu_cdiv(maxn, op->tc_kslice);
    } else if (slice_atoms > 0) {
        nsl = dgpu_cdiv(maxn, slice_atoms);
    } else {
        nsl = dgpu_cdiv((int64_t)slice_mult * ctx->nsm, tiles);
        if (nsl > 1 && dgpu_cdiv(maxn, nsl) < 2048) nsl = dgpu_cdiv(maxn, 2048);
    }
    // the kernel's producers address a slice's atoms by 32-bit byte offsets
    if (nsl < dgpu_cdiv(maxn, TC_SLICE_MAX)) nsl = dgpu_cdiv(maxn, TC_SLICE_MAX);
    if (nsl < 1) nsl = 1;
    g.slice_len = dgpu_cdiv(dgpu_cdiv(maxn > 0 ? maxn : 1, nsl), TC_KB) * TC_KB;   // whole stages of either path
    g.nslice = (int32_t)dgpu_cdiv(maxn > 0 ? maxn : 1, g.slice_len);
    g.nitems = tiles * g.nslice;
    const uint64_t *dd[3] = {in.du, in.dv, in.dw};
    g.ph0 = in.ph0;
    g.dra = dd[g.ra];
    g.drb = dd[g.rb];
    g.dac = dd[axis];
    g.w = in.w;
    g.ma = in.mult + (int64_t)g.ra * in.mult_stride;
    g.mc = in.mult + (int64_t)axis * in.mult_stride;
    g.ma2 = in.mult + (int64_t)(3 + g.ra) * in.mult_stride;
    g.mc2 = in.mult + (int64_t)(3 + axis) * in.mult_stride;
}

void dgpu_tc_partref(const TcProblem &g, const float2 *p, PartRef &ref)
{
    ref.p = p;
    ref.nslice = g.nslice;
    ref.f32 = 1;
    ref.s[g.ra] = 1;
    ref.s[g.rb] = g.fra_p;
    ref.s[g.ac] = g.nrows_p;
    ref.slab = g.slab;
}

// the kernel of an operand type, stage size and V operand path
static void (*tc_kernel(bool bf, int ks, bool vring))(const TcLaunch)
{
    if (vring) return bf ? k_tc<true, TC_KB, true> : k_tc<false, TC_KB, true>;
    if (ks == TC_KB) return bf ? k_tc<true, TC_KB, false> : k_tc<false, TC_KB, false>;
    return bf ? k_tc<true, TC_KA, false> : k_tc<false, TC_KA, false>;
}

#define TC_VIMG_BUDGET ((int64_t)16 << 30)    // bytes of V images per launch

int dgpu_tc_plan(dgpu_ctx *ctx, int nprob, const TcInput *in, const dgpu_opts *op, int N, int slice_mult,
                 TcPlan &plan, DevBuf &part, DevBuf &desc, DevBuf *vimg)
{
    plan.probs.assign(nprob, TcProblem());
    plan.part_off.assign(nprob, 0);
    plan.nslice.assign(nprob, 0);
    int64_t items = 0, elems = 0;
    std::vector<int> axes(nprob);
    for (int p = 0; p < nprob; p++) {
        int axis = in[p].axis;
        if (axis < 0) {
            double best = 1e300;
            for (int a = 0; a < 3; a++) {
                const double ar = tc_area(in[p].box, a, N);
                if (ar >= 0 && ar < best * (1 - 1e-9)) { best = ar; axis = a; }
            }
        }
        if (axis < 0) return dgpu_set_error(ctx, DGPU_ERR_ARG, "no tensor-core tile fits the box");
        axes[p] = axis;
    }
    // several problems share the SMs: one slice length for all, from their
    // total work (tiles x atoms), so that the whole launch has about
    // slice_mult items per SM of about equal size (at least 2048 atoms)
    int64_t slice_atoms = 0;
    if (nprob > 1 && op->tc_kslice <= 0) {
        double work = 0.0;
        for (int p = 0; p < nprob; p++) {
            TcProblem g;
            tc_problem(ctx, in[p], op, axes[p], N, slice_mult, 0, g);
            work += (double)(g.nitems / g.nslice) * (double)(g.nslice * g.slice_len);
        }
        slice_atoms = (int64_t)ceil(work / ((double)slice_mult * ctx->nsm));
        if (slice_atoms < 2048) slice_atoms = 2048;
    }
    for (int p = 0; p < nprob; p++) {
        TcProblem &g = plan.probs[p];
        tc_problem(ctx, in[p], op, axes[p], N, slice_mult, slice_atoms, g);
        g.item0 = items;
        items += g.nitems;
        plan.part_off[p] = elems;
        plan.nslice[p] = g.nslice;
        elems += (int64_t)g.ntype * g.nslice * g.slab;
    }
    plan.item_prob.resize(items);
    for (int p = 0; p < nprob; p++)
        for (int64_t i = 0; i < plan.probs[p].nitems; i++) plan.item_prob[plan.probs[p].item0 + i] = p;
    DGPU_CUDA(ctx, part.ensure((size_t)(elems > 0 ? elems : 1) * sizeof(float2)));
    for (int p = 0; p < nprob; p++) plan.probs[p].part = part.as<float2>() + plan.part_off[p];
    // V images: one per (64-atom group, column tile) of every problem.  The
    // images depend only on the atoms' column steps and the column index, so
    // problems over the same atoms with the same column axis (boxes of one
    // grid at different origins) share one set, as wide as the widest.
    bool share = nprob > 1;
    int32_t wide = 0;
    for (int p = 0; p < nprob; p++) {
        const TcProblem &g = plan.probs[p];
        share = share && g.dac == plan.probs[0].dac && in[p].ts == in[0].ts && in[p].ntype == in[0].ntype;
        wide = g.n_tiles > wide ? g.n_tiles : wide;
    }
    std::vector<int64_t> voff(nprob, 0);                // in images
    int64_t vtot = 0;
    int need = 0;
    for (int p = 0; p < nprob; p++) {
        const TcProblem &g = plan.probs[p];
        voff[p] = share ? 0 : vtot;
        if (!share || p == 0) vtot += in[p].ts[in[p].ntype] / TC_KB * (share ? wide : g.n_tiles);
        const int c = (int)dgpu_cdiv(dgpu_cdiv(g.ncols, g.n_tiles), 8) * 8;
        need = c > need ? c : need;
    }
    // images pay when every one is re-read by several row tiles (a 3D grid);
    // thin planes with one or two row tiles generate V in the kernel
    double reads = 0.0, imgs = 0.0;
    for (int p = 0; p < nprob; p++) {
        const double ni = (double)(in[p].ts[in[p].ntype] / TC_KB) * plan.probs[p].n_tiles;
        if (!share || p == 0) imgs += share ? (double)(in[p].ts[in[p].ntype] / TC_KB) * wide : ni;
        reads += ni * plan.probs[p].m_tiles;
    }
    const bool reuse = imgs > 0 && reads >= 4.0 * imgs;
    // V images stream through a ring of 64-atom slots when it leaves room for
    // two U stages (N <= 64); the producers of that path hold their atoms'
    // phase data in registers, so it needs no atom slots and may use the whole
    // shared memory of the SM
    const int64_t room = (int64_t)TC_SMEM_MAX - TC_BAR_BYTES - (int64_t)TC_VSLOTS * N * 768;
    plan.vimg = vimg && vtot > 0 && vtot * N * 768 <= TC_VIMG_BUDGET && room >= 2 * 4 * TC_B_BYTES &&
                op->tc_vimg >= 0 && (reuse || op->tc_vimg > 0);
    plan.vshared = share;
    if (plan.vimg) {
        // a tile is then only as wide as the columns need, in eights (the MMAs
        // are 2N wide, and take widths in sixteens).  Tiles, slices and values
        // stay as they are; 51 columns run 56 wide, not 64: 5.85 -> 5.54 ms for
        // the 101^3 half box of 10^6 atoms.  The in-kernel V path keeps the
        // chosen width: narrower tiles were not measured there.
        N = need < N ? need : N;
        DGPU_CUDA(ctx, vimg->ensure((size_t)vtot * N * 768));
        for (int p = 0; p < nprob; p++) {
            plan.probs[p].N = N;
            plan.probs[p].vimg = vimg->as<uint8_t>() + voff[p] * N * 768;
            if (share) plan.probs[p].vstride = wide;
        }
    }
    const size_t pbytes = ((size_t)nprob * sizeof(TcProblem) + 255) & ~(size_t)255;
    DGPU_CUDA(ctx, desc.ensure(pbytes + (size_t)items * sizeof(int32_t) + 256));
    if (ctx->tc_defer) {
        // one copy from pinned memory that stays valid until the run's host wait
        char *h = static_cast<char *>(ctx->stage.take(pbytes + (size_t)items * sizeof(int32_t)));
        if (!h) return dgpu_set_error(ctx, DGPU_ERR_NOMEM, "pinned staging memory");
        memcpy(h, plan.probs.data(), (size_t)nprob * sizeof(TcProblem));
        memcpy(h + pbytes, plan.item_prob.data(), (size_t)items * sizeof(int32_t));
        DGPU_CUDA(ctx, cudaMemcpyAsync(desc.p, h, pbytes + (size_t)items * sizeof(int32_t), cudaMemcpyHostToDevice,
                                       ctx->stream));
    } else {
        DGPU_CUDA(ctx, cudaMemcpyAsync(desc.p, plan.probs.data(), (size_t)nprob * sizeof(TcProblem),
                                       cudaMemcpyHostToDevice, ctx->stream));
        DGPU_CUDA(ctx, cudaMemcpyAsync((char *)desc.p + pbytes, plan.item_prob.data(),
                                       (size_t)items * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
        // the host vectors must outlive the copies
        DGPU_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    TcLaunch &L = plan.L;
    L.probs = (const TcProblem *)desc.p;
    L.item_prob = (const int32_t *)((char *)desc.p + pbytes);
    L.nitems = items;
    L.Nmax = N;
    // TMEM: correction (2N) + main x nbuf (2N each) [+ running sum (2N)]
    L.nbuf = 2 * N * 3 <= 512 ? 2 : 1;
    L.tsum = 2 * N * (2 + L.nbuf) <= 512 ? 1 : 0;
    L.bf16 = op->split == DGPU_SPLIT_BF16;
    const uint32_t vbytes_img = 2u * 3u * N * TC_KB * 2;
    L.vring = plan.vimg ? 1 : 0;
    // V in the kernel: 64-atom stages where two of them fit (N <= 64) and the
    // drain interval is made of them, which halves the producers' waits and
    // fences per atom, else 32-atom stages
    const int64_t budget = TC_SMEM_MAX - TC_BAR_BYTES;
    const int unit = L.vring ? TC_KB : TC_KA;
    const int flush = op->tc_flush > 0 ? (int)dgpu_cdiv(op->tc_flush, unit) * unit : TC_FLUSH_ATOMS;   // atoms
    const bool wide64 = 2 * (4ll * TC_B_BYTES + vbytes_img) <= budget && flush % TC_KB == 0;
    L.ks = L.vring || wide64 ? TC_KB : TC_KA;
    L.flush = flush / L.ks;                                        // stages
    const uint32_t vbytes = 2u * 3u * N * L.ks * 2;
    const uint32_t stage_bytes = 4u * TC_M * L.ks * 2 + (L.vring ? 0u : vbytes);
    const int64_t ring = L.vring ? (int64_t)TC_VSLOTS * vbytes : 0;
    const int stages = (int)((budget - ring) / stage_bytes);
    L.stages = stages > 4 ? 4 : stages;
    L.tmem_cols = pow2_cols(2 * N * (1 + L.nbuf + L.tsum));
    if (L.stages < 2 || L.tmem_cols > 512) return dgpu_set_error(ctx, DGPU_ERR_ARG, "tile does not fit");
    plan.smem = (size_t)L.stages * stage_bytes + (size_t)ring + TC_BAR_BYTES;
    if (!ctx->tc_attr) {              // once per context (and device), outside any stream capture
        for (int v = 0; v < 6; v++) {
            const void *k = (const void *)tc_kernel(v & 1, v < 4 ? TC_KB : TC_KA, v < 2);
            DGPU_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_MAX));
            // a build that launched with fewer registers would leave the producers waiting for more
            cudaFuncAttributes a;
            DGPU_CUDA(ctx, cudaFuncGetAttributes(&a, k));
            if (a.numRegs * (TC_THREADS / 128) < 4 * TC_REG_PROD + TC_REG_EPI + TC_REG_MMA)
                return dgpu_set_error(ctx, DGPU_ERR_CUDA, "k_tc: %d registers per thread, too few to share out",
                                      a.numRegs);
        }
        ctx->tc_attr = true;
    }
    DGPU_CUDA(ctx, ctx->flag.ensure(64));
    L.err = ctx->flag.as<int32_t>() + 8;
    L.timeout_ns = op->tc_wait_us > 0 ? (uint64_t)op->tc_wait_us * 1000ull : TC_TIMEOUT_NS;
    return DGPU_OK;
}

int dgpu_tc_launch(dgpu_ctx *ctx, const TcPlan &plan, bool timed)
{
    if (!ctx->tc_defer) DGPU_CUDA(ctx, cudaMemsetAsync(plan.L.err, 0, sizeof(int32_t), ctx->stream));
    ctx->tc_timed = false;
    if (plan.L.nitems < 1) return DGPU_OK;
    if (plan.vimg)
        for (const TcProblem &g : plan.probs) {
            const int64_t nimg = (g.ts[g.ntype] / TC_KB) * g.vstride;
            if (nimg < 1) continue;
            if (plan.L.bf16)
                k_tc_vgen<true><<<(unsigned)nimg, 256, 0, ctx->stream>>>(g.dac, g.N, g.vstride, g.vimg);
            else
                k_tc_vgen<false><<<(unsigned)nimg, 256, 0, ctx->stream>>>(g.dac, g.N, g.vstride, g.vimg);
            if (plan.vshared) break;                        // one set for all problems
        }
    const int grid = (int)(plan.L.nitems < ctx->nsm ? plan.L.nitems : ctx->nsm);
    if (timed) DGPU_CUDA(ctx, cudaEventRecord(ctx->ev[6], ctx->stream));
    tc_kernel(plan.L.bf16, plan.L.ks, plan.L.vring)<<<grid, TC_THREADS, plan.smem, ctx->stream>>>(plan.L);
    DGPU_CUDA(ctx, cudaGetLastError());
    if (timed) DGPU_CUDA(ctx, cudaEventRecord(ctx->ev[7], ctx->stream));
    ctx->tc_timed = timed;
    return DGPU_OK;
}

int dgpu_tc_check(dgpu_ctx *ctx)
{
    int32_t herr = 0;
    DGPU_CUDA(ctx, cudaMemcpyAsync(&herr, ctx->flag.as<int32_t>() + 8, sizeof(int32_t), cudaMemcpyDeviceToHost,
                                   ctx->stream));
    DGPU_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (herr) return dgpu_set_error(ctx, DGPU_ERR_TIMEOUT, "tensor-core kernel wait gave up (site %d)", herr);
    return DGPU_OK;
}

int dgpu_tc_mult_async(dgpu_ctx *ctx, const uint64_t *du, const uint64_t *dv, const uint64_t *dw, int64_t n,
                       int64_t stride, float2 *out, int mask)
{
    if (n < 1 || !(mask & 7)) return DGPU_OK;
    k_tc_mult<<<(unsigned)dgpu_cdiv(n, 256), 256, 0, ctx->stream>>>(du, dv, dw, n, stride,
                                                                      ctx->tc_tab.as<double2>(), out, mask & 7);
    DGPU_CUDA(ctx, cudaGetLastError());
    return DGPU_OK;
}

#define TC_TUNE_GAIN 0.97f                     // a later candidate wins if it takes less than this of the best's time

#define TC_WIDE_ATOMS 16384                    // atoms per type up to which tiles above 64 columns are tried

// Candidate configurations: every column axis and tile width whose padded
// MMA area is within 25% of the smallest, at two slicings.  Above 64 columns
// every drain goes through global memory: 34 to 40 ms a launch against 4.4 on
// the 500 000-atom, 101^3 volume, where trying eight of them was 0.3 s of the
// first call; with few drains it costs nothing to try.
static void tc_candidates(const BoxSpec &box, int want_n, int kslice, int64_t maxn, TcChoice *out, int &n)
{
    auto skip = [&](int N) { return want_n ? N != want_n : N < 48 || (N > 64 && maxn > TC_WIDE_ATOMS); };
    double best = 1e300;
    for (int a = 0; a < 3; a++)
        for (int N = 16; N <= 128; N += 16) {
            if (skip(N)) continue;
            const double ar = tc_area(box, a, N);
            if (ar >= 0 && ar < best) best = ar;
        }
    n = 0;
    for (int a = 0; a < 3; a++)
        for (int N = 16; N <= 128; N += 16) {
            if (skip(N)) continue;
            const double ar = tc_area(box, a, N);
            if (ar < 0 || ar > 1.25 * best) continue;
            for (int m : {4, 8}) {
                if (n >= 64) return;
                if (kslice > 0 && m != 4) continue;     // the slicing is given: one candidate per tile
                out[n].axis = a;
                out[n].N = N;
                out[n].slice_mult = m;
                n++;
            }
        }
}

extern "C" double dgpu_tc_last_kernel_ms(const dgpu_ctx *ctx) { return ctx ? ctx->tc_kernel_ms : 0.0; }

int dgpu_tc_sums(dgpu_ctx *ctx, const uint64_t *ph0, const uint64_t *du, const uint64_t *dv, const uint64_t *dw,
                 const float *w, const int64_t *h_type_start, int32_t ntype, const BoxSpec &box,
                 const dgpu_opts *op, DevBuf &part, PartRef *ref)
{
    if (ntype < 1 || ntype > 64) return dgpu_set_error(ctx, DGPU_ERR_ARG, "ntype=%d", ntype);
    const int want_n = op->tc_tile_n;
    if (want_n && (want_n % 16 || want_n < 16 || want_n > 128))
        return dgpu_set_error(ctx, DGPU_ERR_ARG, "tc_tile_n=%d (multiple of 16 in 16..128)", want_n);
    int64_t maxn = 0;
    for (int t = 0; t < ntype; t++) {
        const int64_t n = h_type_start[t + 1] - h_type_start[t];
        maxn = n > maxn ? n : maxn;
    }
    const int64_t npad = h_type_start[ntype];
    DGPU_CUDA(ctx, ctx->tc_mult.ensure((size_t)TC_MULT_ARRAYS * (npad > 0 ? npad : 1) * sizeof(float2)));
    int rc;
    int lg = 0;
    while ((1LL << lg) < maxn) lg++;
    const TcKey key(box.f[0], box.f[1], box.f[2], ntype, lg, op->split * 1000 + want_n,
                    op->tc_kslice * 7 + op->tc_flush);
    TcInput in;
    in.ph0 = ph0;
    in.du = du;
    in.dv = dv;
    in.dw = dw;
    in.w = w;
    in.mult = ctx->tc_mult.as<float2>();
    in.mult_stride = npad;
    in.ts = h_type_start;
    in.ntype = ntype;
    in.box = box;
    TcChoice choice;
    auto hit = ctx->tc_tuned.find(key);
    const bool cached = hit != ctx->tc_tuned.end();
    if (cached) {
        choice = hit->second;
    } else {
        // the candidates use every axis as row or column axis: all step factors
        rc = dgpu_tc_mult_async(ctx, du, dv, dw, npad, npad, ctx->tc_mult.as<float2>(), 7);
        if (rc) return rc;
        TcChoice cand[64];
        int nc = 0;
        tc_candidates(box, want_n, op->tc_kslice, maxn, cand, nc);
        if (nc == 0) return dgpu_set_error(ctx, DGPU_ERR_ARG, "no tensor-core tile fits the box");
        float best = 1e30f;
        choice = cand[0];
        for (int c = 0; c < nc && nc > 1; c++) {
            in.axis = cand[c].axis;
            TcPlan plan;
            if (dgpu_tc_plan(ctx, 1, &in, op, cand[c].N, cand[c].slice_mult, plan, part, ctx->tc_part,
                             &ctx->tc_vimg))
                continue;
            DGPU_CUDA(ctx, cudaEventRecord(ctx->ev[4], ctx->stream));
            rc = dgpu_tc_launch(ctx, plan);
            if (rc) return rc;
            DGPU_CUDA(ctx, cudaEventRecord(ctx->ev[5], ctx->stream));
            rc = dgpu_tc_check(ctx);
            if (rc) return rc;
            float ms = 0.f;
            DGPU_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev[4], ctx->ev[5]));
            // nearly equal candidates (a cube's axes) must not change places with
            // the timing noise, and the rounding of the sums with them
            if (ms < TC_TUNE_GAIN * best) {
                best = ms;
                choice = cand[c];
            }
        }
        ctx->tc_tuned[key] = choice;
    }
    in.axis = choice.axis;
    TcPlan plan;
    rc = dgpu_tc_plan(ctx, 1, &in, op, choice.N, choice.slice_mult, plan, part, ctx->tc_part, &ctx->tc_vimg);
    if (rc) return rc;
    if (cached) {
        // the factors this plan reads: the row axis ra (the producers' steps),
        // on the in-kernel V path also the column axis
        const TcProblem &g = plan.probs[0];
        rc = dgpu_tc_mult_async(ctx, du, dv, dw, npad, npad, ctx->tc_mult.as<float2>(),
                                (1 << g.ra) | (plan.vimg ? 0 : 1 << g.ac));
        if (rc) return rc;
    }
    rc = dgpu_tc_launch(ctx, plan, ctx->tc_defer != 1);
    if (rc) return rc;
    if (!ctx->tc_defer) {
        rc = dgpu_tc_check(ctx);
        if (rc) return rc;
        float ms = 0.f;
        if (ctx->tc_timed) DGPU_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev[6], ctx->ev[7]));
        ctx->tc_kernel_ms = ms;
    }
    ctx->tc_last[0] = plan.probs[0].ac;
    ctx->tc_last[1] = choice.N;              // as tc_tile_n asks for it; with V images the tiles run narrower
    ctx->tc_last[2] = plan.L.nbuf;
    ctx->tc_last[3] = (int32_t)plan.probs[0].slice_len;
    dgpu_tc_partref(plan.probs[0], part.as<float2>(), *ref);
    return DGPU_OK;
}
