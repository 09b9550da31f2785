// Allocation-free per-type structure-factor sum.
//
// Some callers of the per-type sum cannot allocate device memory: a reverse
// Monte Carlo loop that re-evaluates the contribution of a few atoms after
// every move (thousands of calls per second, where cudaMalloc/cudaFree would
// synchronise the device each time), code that runs inside a memory budget
// owned by another allocator, or code that enqueues work on a stream it does
// not own.  dgpu_four_strucf_noalloc serves them: the caller passes device
// inputs and outputs and a stream, and the library's working memory is one
// file-scope __device__ array of fixed size (2 MiB, for the phase data of more
// than 128 atoms, or of atoms that share memory with the result) that every GPU loading the library holds until the process
// exits.
//
// Limits: at most NOALLOC_MAX_ATOMS atoms (the array's size) and
// NOALLOC_MAX_POINTS computed points (fnum(1)*fnum(2)*fnum(3), a limit of the
// interface: the points need no working memory) per call; larger requests
// return DGPU_ERR_SCRATCH_SIZE.  All calls share the array, so calls whose work
// overlaps on the GPU (two streams, or two host threads) race; calls queued
// on one stream are ordered and safe.  Every call rewrites the parts of the
// array it reads, so nothing carries over from one call to the next.
//
// Set-up: the device address of the array is looked up once per device
// (cudaGetSymbolAddress, with that device current) on the first call made on
// that device; make that first call before any stream capture begins.  The
// address is kept with the CUDA context it belongs to and looked up again
// when a later call finds a different context current on that device (for
// instance a new primary context after cudaDeviceReset).  The stream must
// belong to the device that is current at the call.
#include <cuda.h>

#include <mutex>

#include "dgpu_internal.h"

#define NOALLOC_MAX_ATOMS 131072
#define NOALLOC_MAX_POINTS 262144
#define NOALLOC_NT 128
// phase data of one atom: four 32-bit words
#define NOALLOC_BYTES ((size_t)NOALLOC_MAX_ATOMS * 16)

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

namespace {

std::mutex g_mu;
struct Cached {
    CUcontext ctx;
    void *addr;
};
Cached g_addr[256];

// cuCtxGetCurrent of the CUDA driver API, looked up through the runtime
// (the library does not link libcuda itself)
typedef CUresult (*CtxGetCurrentFn)(CUcontext *);
CtxGetCurrentFn ctx_get_current()
{
    static CtxGetCurrentFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<CtxGetCurrentFn>(p);
    }
    return fn;
}

// device address of the scratch array for the current device and context
int scratch_address(void **out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return DGPU_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_mu);
    const CtxGetCurrentFn get = ctx_get_current();
    if (!get) return DGPU_ERR_CUDA;
    CUcontext cur = nullptr;              // null before the runtime's first use on this thread
    if (get(&cur) != CUDA_SUCCESS) return DGPU_ERR_CUDA;
    if (!cur || !g_addr[dev].addr || g_addr[dev].ctx != cur) {
        void *p = nullptr;
        // the look-up also makes the device's primary context current
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return DGPU_ERR_CUDA;
        if (get(&cur) != CUDA_SUCCESS || !cur) return DGPU_ERR_CUDA;
        g_addr[dev].addr = p;
        g_addr[dev].ctx = cur;
    }
    *out = g_addr[dev].addr;
    return DGPU_OK;
}

struct Geo {
    double u[3], v[3], w[3], off[9];
    int32_t lmn[6];
    int32_t num[3], fnum[3];
};

__device__ __forceinline__ double na_dot(const double *a, double x0, double x1, double x2)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(a[0], x0), __dmul_rn(a[1], x1)), __dmul_rn(a[2], x2));
}

// NINT(2^22 * (x - INT(x))), four_strucf_OMP_mod.f90:143-148
__device__ __forceinline__ int64_t na_inc22(double x)
{
    return (int64_t)llround(__dmul_rn(4194304.0, __dadd_rn(__dsub_rn(x, trunc(x)), 0.0)));
}

// REF22 phase data of one atom in units of 2^-32 turn: origin phase and the
// increments along the three axes.  They are multiples of 2^-22 turn, so the
// 32 bits hold them exactly.
__device__ __forceinline__ uint4 na_phase(const double *__restrict__ xat, int64_t n, const Geo &g, int64_t k)
{
    const double x0 = xat[k], x1 = xat[n + k], x2 = xat[2 * n + k];
    const int64_t iu = na_inc22(na_dot(g.u, x0, x1, x2)), iv = na_inc22(na_dot(g.v, x0, x1, x2));
    const int64_t iw = na_inc22(na_dot(g.w, x0, x1, x2));
    const int64_t ju = na_inc22(na_dot(g.off + 0, x0, x1, x2)), jv = na_inc22(na_dot(g.off + 3, x0, x1, x2));
    const int64_t jw = na_inc22(na_dot(g.off + 6, x0, x1, x2));
    const int64_t base = (int64_t)g.lmn[0] * iu + (int64_t)g.lmn[1] * iv + (int64_t)g.lmn[2] * iw +
                         (int64_t)g.lmn[3] * ju + (int64_t)g.lmn[4] * jv + (int64_t)g.lmn[5] * jw;
    return make_uint4((uint32_t)((uint64_t)base << 10), (uint32_t)((uint64_t)iu << 10),
                      (uint32_t)((uint64_t)iv << 10), (uint32_t)((uint64_t)iw << 10));
}

__global__ void k_na_phase(const double *__restrict__ xat, int64_t n, Geo g, uint4 *__restrict__ ph)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) ph[k] = na_phase(xat, n, g, k);
}

// tcsf(num) = cfact(istl) * sum on fnum, zero elsewhere (fourier_form.f90:147-177).
// A thread of the first nsum blocks owns Q consecutive points of fnum along
// its first axis and sums all atoms; phases keep their top 16 bits (the
// reference's 2^16-entry table index).  FP32 sums over a shared-memory chunk
// with Fast2Sum compensation (a coherent sum of nearly equal terms, as on a
// Bragg row, would otherwise round with a bias that grows with the chunk
// length), FP64 across chunks.  Up to one chunk of atoms, every block forms
// their phases itself (ph null) and the call is one launch: 8 atoms on 51 x 51
// points took 15 us in three (4.5 + 7.7 on two blocks + 2.9).  The blocks after
// them write the zeros: threads that own points of num instead, most of them
// outside fnum, left the summing warps nearly empty and formed phases for
// nothing (call and host wait, 128 atoms, 1 x 201 x 201 of 201^3 points: 734 us
// where this takes 52; 8 atoms, 63^3 of 201^3: 166 and 50).
#define NOALLOC_ZERO 4      // points per thread of the blocks that write zeros

template <int Q>
__global__ void __launch_bounds__(NOALLOC_NT) k_na_sum(const double *__restrict__ xat, const uint4 *__restrict__ ph,
                                                       int64_t n, Geo g, const double2 *__restrict__ cfact,
                                                       const int32_t *__restrict__ istl, double2 *__restrict__ tcsf,
                                                       uint32_t nsum)
{
    if (blockIdx.x >= nsum) {
        const int64_t np = (int64_t)g.num[0] * g.num[1] * g.num[2];
        int64_t p = (int64_t)(blockIdx.x - nsum) * (NOALLOC_NT * NOALLOC_ZERO) + threadIdx.x;
        for (int k = 0; k < NOALLOC_ZERO && p < np; k++, p += NOALLOC_NT) {
            int64_t i, j, l;
            if (np <= 0xFFFFFFFFll) {             // 32-bit divisions
                const uint32_t r = (uint32_t)p / (uint32_t)g.num[0];
                i = (uint32_t)p - r * (uint32_t)g.num[0];
                l = r / (uint32_t)g.num[1];
                j = r - (uint32_t)l * (uint32_t)g.num[1];
            } else {
                i = p % g.num[0];
                j = p / g.num[0] % g.num[1];
                l = p / g.num[0] / g.num[1];
            }
            if (i >= g.fnum[0] || j >= g.fnum[1] || l >= g.fnum[2]) tcsf[p] = make_double2(0.0, 0.0);
        }
        return;
    }
    __shared__ uint4 s_ph[NOALLOC_NT];
    // at most NOALLOC_MAX_POINTS slots
    const uint32_t nq = (uint32_t)(g.fnum[0] + Q - 1) / Q, nslots = nq * g.fnum[1] * g.fnum[2];
    const uint32_t slot = blockIdx.x * NOALLOC_NT + threadIdx.x, sl = slot < nslots ? slot : 0;
    const uint32_t i0 = sl % nq * Q, j = sl / nq % g.fnum[1], l = sl / nq / g.fnum[1];
    double accd[Q][2];
#pragma unroll
    for (int k = 0; k < Q; k++) accd[k][0] = accd[k][1] = 0.0;
    for (int64_t a0 = 0; a0 < n; a0 += NOALLOC_NT) {
        const int cnt = (int)min((int64_t)NOALLOC_NT, n - a0);
        __syncthreads();
        if (threadIdx.x < cnt)
            s_ph[threadIdx.x] = ph ? ph[a0 + threadIdx.x] : na_phase(xat, n, g, a0 + threadIdx.x);
        __syncthreads();
        float accf[Q][2], cmpf[Q][2];
#pragma unroll
        for (int k = 0; k < Q; k++) accf[k][0] = accf[k][1] = cmpf[k][0] = cmpf[k][1] = 0.f;
#pragma unroll 2
        for (int a = 0; a < cnt; a++) {
            const uint4 d = s_ph[a];
            uint32_t p = d.x + i0 * d.y + j * d.z + l * d.w;
#pragma unroll
            for (int k = 0; k < Q; k++) {
                const float x = (float)(int32_t)(p & 0xFFFF0000u) * 4.656612873077393e-10f;
                float sn, cs;
                sincospif(x, &sn, &cs);
                const float t0 = accf[k][0] + cs, t1 = accf[k][1] + sn;
                cmpf[k][0] += cs - (t0 - accf[k][0]);
                cmpf[k][1] += sn - (t1 - accf[k][1]);
                accf[k][0] = t0;
                accf[k][1] = t1;
                p += d.y;
            }
        }
#pragma unroll
        for (int k = 0; k < Q; k++) {
            accd[k][0] += (double)accf[k][0] + (double)cmpf[k][0];
            accd[k][1] += (double)accf[k][1] + (double)cmpf[k][1];
        }
    }
    if (slot >= nslots) return;
#pragma unroll
    for (int k = 0; k < Q; k++) {
        const uint32_t i = i0 + k;
        if (i >= (uint32_t)g.fnum[0]) break;
        const int64_t p = i + (int64_t)g.num[0] * (j + (int64_t)g.num[1] * l);
        const double2 s = make_double2(accd[k][0], accd[k][1]);
        double2 out = s;
        if (cfact) {
            const int32_t q = istl[p];
            if (q < 0 || q > DGPU_CFPKT) {      // not a table index: flag the point, read nothing
                out = make_double2(__longlong_as_double(0x7ff8000000000000ll), 0.0);
            } else {
                const double2 c = cfact[q];
                out = make_double2(s.x * c.x - s.y * c.y, s.x * c.y + s.y * c.x);
            }
        }
        tcsf[p] = out;
    }
}

}  // namespace

extern "C" int dgpu_four_strucf_noalloc(void *stream, const double *d_xat, int64_t nxat, const double uin[3],
                                        const double vin[3], const double win[3], const double off_shift[9],
                                        const int32_t lmn[6], const int32_t num[3], const int32_t fnum[3],
                                        const double *d_cfact, const int32_t *d_istl, double *d_tcsf)
{
    if (!uin || !vin || !win || !off_shift || !lmn || !num || !fnum || !d_tcsf) return DGPU_ERR_ARG;
    if (nxat < 0 || (nxat > 0 && !d_xat) || (d_cfact && !d_istl)) return DGPU_ERR_ARG;
    for (int k = 0; k < 3; k++)
        if (num[k] < 1 || fnum[k] < 1 || fnum[k] > num[k]) return DGPU_ERR_ARG;
    const int64_t npts = (int64_t)fnum[0] * fnum[1] * fnum[2];
    if (nxat > NOALLOC_MAX_ATOMS || npts > NOALLOC_MAX_POINTS) return DGPU_ERR_SCRATCH_SIZE;
    void *base = nullptr;
    int rc = scratch_address(&base);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (st) {
        // the scratch address and the launches belong to the current device
        int sdev = -1, dev = -2;
        if (cudaStreamGetDevice(st, &sdev) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) return DGPU_ERR_ARG;
        if (sdev != dev) return DGPU_ERR_ARG;
    }
    Geo g;
    for (int k = 0; k < 3; k++) {
        g.u[k] = uin[k];
        g.v[k] = vin[k];
        g.w[k] = win[k];
        g.num[k] = num[k];
        g.fnum[k] = fnum[k];
    }
    for (int k = 0; k < 9; k++) g.off[k] = off_shift[k];
    for (int k = 0; k < 6; k++) g.lmn[k] = lmn[k];
    const int64_t np = (int64_t)num[0] * num[1] * num[2];
    const double2 *cf = reinterpret_cast<const double2 *>(d_cfact);
    double2 *out = reinterpret_cast<double2 *>(d_tcsf);
    uint4 *ph = nullptr;
    // a block that forms the phases itself reads xat while others write tcsf:
    // a caller that lets them share memory gets the phases of all atoms first
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(d_xat), t0 = reinterpret_cast<uintptr_t>(d_tcsf);
    const bool shared = x0 < t0 + (uint64_t)np * 16 && t0 < x0 + (uint64_t)nxat * 24;
    if (nxat > NOALLOC_NT || (nxat > 0 && shared)) {
        ph = reinterpret_cast<uint4 *>(base);
        k_na_phase<<<(unsigned)((nxat + NOALLOC_NT - 1) / NOALLOC_NT), NOALLOC_NT, 0, st>>>(d_xat, nxat, g, ph);
    }
    // one point per thread until there are more than fill the chip
    const int q = npts > 131072 ? 2 : 1;
    const uint32_t nslots = (uint32_t)((fnum[0] + q - 1) / q) * fnum[1] * fnum[2];
    const uint32_t nsum = (nslots + NOALLOC_NT - 1) / NOALLOC_NT;
    const int64_t nzero = npts < np ? (np + NOALLOC_NT * NOALLOC_ZERO - 1) / (NOALLOC_NT * NOALLOC_ZERO) : 0;
    const unsigned nblk = (unsigned)(nsum + nzero);
    if (q == 1) k_na_sum<1><<<nblk, NOALLOC_NT, 0, st>>>(d_xat, ph, nxat, g, cf, d_istl, out, nsum);
    else k_na_sum<2><<<nblk, NOALLOC_NT, 0, st>>>(d_xat, ph, nxat, g, cf, d_istl, out, nsum);
    return cudaGetLastError() == cudaSuccess ? DGPU_OK : DGPU_ERR_CUDA;
}
