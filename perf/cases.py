"""The work that users of the library have it do, as cases to measure.

Each case is one call (or one training step) through a public entry point:
the C-ABI on device arrays, or the Python mirror on host arrays.  Every size
is of a kind that the tests, the benchmark or the synthetic workloads of this
repository use; positions, disorder and targets come from the seed.

Cases on the tensor-core engine give `tc_kslice`, the number of atoms summed
before a partial sum is written: a program that wants the same rounding from
one process to the next fixes it, because the engine otherwise picks the
slicing by timing candidates the first time it sees a shape.  For the same
reason their grids have one clearly best column axis (or, as the benchmark's
cube, one that every process picks).
"""
import ctypes as C
import math

import numpy as np
import torch

from diffusecode_gb300 import _abi
from diffusecode_gb300 import fourier as FR
from diffusecode_gb300 import structures as S
from diffusecode_gb300._lib import default_context

DEV = "cuda:0"

# Scattering factors c, a1, b1, ..., a4, b4 of four generic atom types.
FORM = [
    [0.20, 8.0, 2.0, 5.0, 9.0, 3.0, 0.7, 1.5, 40.0],
    [1.10, 6.5, 5.5, 4.0, 0.9, 2.2, 21.0, 0.8, 33.0],
    [0.35, 3.0, 13.3, 2.3, 5.7, 1.5, 0.3, 0.9, 32.9],
    [0.80, 9.5, 1.2, 2.6, 11.0, 4.4, 27.0, 1.2, 48.0],
]
B_ISO = 0.5


def listed():
    return [
        # Reverse Monte Carlo: after a move, the contribution of the few moved
        # atoms to a plane, on device arrays, without allocation; launch latency.
        dict(name="rmc-move", kind="noalloc", atoms=8, n1=51, n2=51, n3=1),
        # The drop-in for four_strucf as the host program calls it for one atom
        # type: host arrays in and out, the reference's integer phases.
        dict(name="type-sum", kind="strucf", atoms=1500, n1=101, n2=101, n3=1),
        # calc_hkl: the reflections of a small crystal for an HKLF4 / CIF list.
        dict(name="reflections", kind="hkl", cells=6, hmax=6, refl=1200),
        # The `fourier` menu's run of a vacancy-disordered perovskite plane with
        # the reference's own phase arithmetic, host arrays (5000 sites).
        dict(name="plane-menu", kind="menu", cells=10, n=201),
        # Anisotropic displacements, CUDA-core engine with exact phases (the
        # choice where 1e-7 is wanted), a 3D volume on device arrays.
        dict(name="anisotropic-volume", kind="aniso", cells=20, n1=61, n2=45, n3=31),
        # A 3D volume through the host entry, tensor-core engine.
        dict(name="volume-host", kind="volume", cells=30, n1=125, n2=81, n3=75, kslice=8192, host=True),
        # The 3D volume of the benchmark: 500 000 atoms of an alloy on 101^3
        # points, device arrays.
        dict(name="volume", kind="volume", cells=50, n1=101, n2=101, n3=101, kslice=32768, host=False),
        # Layered crystal with stacking faults, average structure factor
        # subtracted (set aver 1), a large h0l plane.
        dict(name="layers-average", kind="average", na=100, nc=20, n=881, kslice=16384),
        # Diffuse intensity averaged over lots of a large crystal.
        dict(name="lots", kind="lots", cells=40, ls=9, lots=75, n1=121, n2=91, n3=85, kslice=8192),
        # One refinement step: chi^2 and its gradient for positions and
        # occupancies through autograd.
        dict(name="refine-step", kind="gradient", c1=25, c2=25, c3=20, n1=143, n2=47, n3=33, kslice=8192),
        # One generation of a population refinement with gradients: crystals of
        # 2000 to 60 000 atoms, each with a plane of its own.
        dict(name="population", kind="population", members=16, amin=2000, amax=60000, nmin=129, nmax=257),
        # Powder pattern by the complete integration of reciprocal space.
        dict(name="powder", kind="powder", cells=35, dhk=0.05, dl=0.02, dsmax=0.8, qmax=5.0, dq=0.001),
    ]


def _odd(rng, lo, hi):
    """An odd number of [lo, hi], even over the logarithm."""
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))) // 2 * 2 + 1


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "strucf", "hkl", "menu", "aniso", "volume", "average", "lots", "gradient",
                       "population", "powder"])
    if kind == "noalloc":
        return dict(kind=kind, atoms=_log(rng, 1, 400), n1=_odd(rng, 21, 151), n2=_log(rng, 20, 150), n3=1)
    if kind == "strucf":
        return dict(kind=kind, atoms=_log(rng, 40, 6000), n1=_odd(rng, 41, 201), n2=_log(rng, 40, 200), n3=1)
    if kind == "hkl":
        return dict(kind=kind, cells=rng.randint(3, 9), hmax=rng.randint(3, 9), refl=_log(rng, 50, 3000))
    if kind == "menu":
        return dict(kind=kind, cells=rng.randint(5, 14), n=_log(rng, 80, 300))
    if kind == "aniso":
        return dict(kind=kind, cells=rng.randint(8, 20), n1=_odd(rng, 21, 61), n2=_odd(rng, 21, 61),
                    n3=_odd(rng, 9, 31))
    if kind == "volume":
        return dict(kind=kind, cells=rng.randint(24, 40), n1=rng.choice([121, 123, 125, 127]), n2=_odd(rng, 67, 93),
                    n3=_odd(rng, 67, 93), kslice=8192, host=rng.random() < 0.5)
    if kind == "average":
        return dict(kind=kind, na=rng.randint(40, 90), nc=rng.randint(8, 20), n=_odd(rng, 865, 893),
                    kslice=8192)
    if kind == "lots":
        return dict(kind=kind, cells=rng.randint(20, 40), ls=rng.randint(5, 9), lots=_log(rng, 10, 75),
                    n1=rng.choice([121, 123, 125, 127]), n2=_odd(rng, 67, 91), n3=_odd(rng, 67, 85), kslice=8192)
    if kind == "gradient":
        return dict(kind=kind, c1=rng.randint(12, 25), c2=rng.randint(12, 25), c3=rng.randint(12, 20),
                    n1=rng.choice([139, 141, 143]), n2=rng.choice([45, 47]), n3=rng.choice([31, 33, 35]), kslice=8192)
    if kind == "population":
        lo = _log(rng, 1000, 8000)
        return dict(kind=kind, members=rng.randint(3, 16), amin=lo, amax=_log(rng, lo, 60000), nmin=_odd(rng, 81, 129),
                    nmax=_odd(rng, 133, 257))
    return dict(kind=kind, cells=rng.randint(12, 34), dhk=round(rng.uniform(0.05, 0.12), 3),
                dl=round(rng.uniform(0.02, 0.06), 3), dsmax=round(rng.uniform(0.5, 0.8), 2), qmax=5.0, dq=0.001)


# ---------------------------------------------------------------------------
# crystals and grids

def _metric(a):
    """Reciprocal metric of a cell with orthogonal axes a, or of the hexagonal cell ("hex", a, c)."""
    if a[0] == "hex":
        ar, cr = 2.0 / (math.sqrt(3.0) * a[1]), 1.0 / a[2]
        return np.array([[ar * ar, ar * ar / 2, 0.0], [ar * ar / 2, ar * ar, 0.0], [0.0, 0.0, cr * cr]])
    return np.diag([1.0 / (x * x) for x in a])


def _atoms(rng, sites, types, icc, sigma):
    """Atoms cell after cell (x fastest), displaced by sigma (lattice units), FP32-representable."""
    i, j, k = np.meshgrid(*(np.arange(n) for n in icc), indexing="ij")
    cells = np.stack([x.ravel(order="F") for x in (i, j, k)], 1).astype(np.float64)
    pos = (cells[:, None, :] + np.asarray(sites, np.float64)[None]).reshape(-1, 3)
    if sigma > 0:
        pos = pos + rng.normal(size=pos.shape) * sigma
    return pos.astype(np.float32).astype(np.float64), np.tile(np.asarray(types, np.int32), len(cells))


def _crystal(pos, iscat, nscat, icc, ncatoms, a, occ=None, **kw):
    scat = np.zeros((nscat + 1, 11))
    for t in range(nscat):
        scat[t + 1, :9] = FORM[t]
    dw = np.full(nscat + 1, B_ISO)
    dw[0] = 0.0
    return S.CrystalData(pos=pos, iscat=iscat, nscat=nscat, ncatoms=ncatoms, icc=icc, rten=_metric(a), scat=scat,
                         occ=np.ones(nscat + 1), dw=dw, atom_occ=occ, **kw)


def _grid(n, hmax):
    """A grid of n points about the origin: h_a from -hmax to hmax along axis a (one point: h_a = 0)."""
    h = [hmax[k] if n[k] > 1 else 0.0 for k in range(3)]
    ll = [-x for x in h]
    c = [list(ll) for _ in range(3)]
    for k in range(3):
        c[k][k] = h[k]
    return S.GridData.from_corners(ll, c[0], c[1], c[2], inc=tuple(n))


FCC = [[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]
SALT = [[x % 1.0, y, z] for dx in (0.0, 0.5) for x, y, z in ([p[0] + dx, p[1], p[2]] for p in FCC)]
PEROVSKITE = [[0, 0, 0], [0.5, 0.5, 0.5], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]


def _perovskite(rng, cells):
    pos, isc = _atoms(rng, PEROVSKITE, [1, 2, 3, 3, 3], (cells,) * 3, 0.01 / 4.0)
    isc[(isc == 2) & (rng.random(isc.shape[0]) < 0.3)] = 0
    return _crystal(pos, isc, 3, (cells,) * 3, 5, (4.0, 4.0, 4.0))


def _alloy(rng, cells):
    """fcc, 50/50 of two types at random, sigma = 0.02 A."""
    pos, isc = _atoms(rng, FCC, [1, 1, 1, 1], (cells,) * 3, 0.02 / 3.6)
    isc[rng.permutation(isc.shape[0])[: isc.shape[0] // 2]] = 2
    return _crystal(pos, isc, 2, (cells,) * 3, 4, (3.6, 3.6, 3.6))


def _layers(rng, na, nc):
    """Hexagonal cell, each layer moved by (1/3, 2/3, 0) with probability 0.1, 2 % vacancies."""
    pos, isc = _atoms(rng, [[0, 0, 0], [1 / 3, 2 / 3, 0.5]], [1, 2], (na, na, nc), 0.0)
    moved = np.cumsum(rng.random(nc) < 0.1)
    layer = np.clip(np.floor(pos[:, 2]).astype(np.int64), 0, nc - 1)
    pos = pos + moved[layer][:, None] * np.array([1 / 3, 2 / 3, 0.0])
    isc[rng.random(isc.shape[0]) < 0.02] = 0
    return _crystal(pos.astype(np.float32).astype(np.float64), isc, 2, (na, na, nc), 2, ("hex", 2.46, 6.7))


def _salt(rng, icc, sigma, occ):
    pos, isc = _atoms(rng, SALT, [1] * 4 + [2] * 4, icc, sigma / 5.64)
    o = (1.0 + rng.uniform(-occ, occ, isc.shape[0])).astype(np.float32)
    return _crystal(pos, isc, 2, icc, 8, (5.64, 5.64, 5.64), occ=o)


ADP = np.array([[0.010, 0.014, 0.008, 0.002, -0.001, 0.003], [0.020, 0.012, 0.016, -0.003, 0.002, 0.001],
                [0.006, 0.006, 0.006, 0.0, 0.0, 0.0]])


def _aniso(rng, cells):
    a = (4.0, 4.5, 5.0)
    pos, isc = _atoms(rng, [[0.1, 0.2, 0.3], [0.55, 0.45, 0.6]], [1, 2], (cells,) * 3, 0.01)
    adp = np.where(isc == 2, 2, np.where(rng.random(isc.shape[0]) < 0.4, 3, 1)).astype(np.int32)
    return _crystal(pos, isc, 2, (cells,) * 3, 2, a, ianis=adp, anis_full=ADP, ar=tuple(1 / x for x in a))


def _member_sizes(case):
    """(kind of cell, cells, points, hmax) of every member: fixed for the case, a population keeps its shape."""
    g = np.random.default_rng(17)
    out = []
    for _ in range(case["members"]):
        kind = int(g.integers(0, 2))
        n = math.exp(g.uniform(math.log(case["amin"]), math.log(case["amax"])))
        pts = int(g.integers(case["nmin"], case["nmax"] + 1)) // 2 * 2 + 1
        out.append((kind, max(1, round((n / (4 if kind else 8)) ** (1 / 3))), min(pts, case["nmax"]),
                    float(g.uniform(2.0, 6.0))))
    return out


def _population(rng, case):
    crs, grids = [], []
    for kind, cells, pts, hmax in _member_sizes(case):
        sites, types, a = (FCC, [1, 2, 1, 2], 3.6) if kind else (SALT, [1] * 4 + [2] * 4, 5.64)
        pos, isc = _atoms(rng, sites, types, (cells,) * 3, 0.03 / a)
        crs.append(_crystal(pos, isc, 2, (cells,) * 3, len(sites), (a, a, a)))
        grids.append(_grid((pts, pts, 1), (hmax, hmax, 0.0)))
    return crs, grids


def _build(case, seed):
    """(crystal or crystals, grid or grids, options) of a case; the same for prepare() and exact()."""
    rng = np.random.default_rng([seed, 91])
    k = case["kind"]
    exact, ref = _abi.PHASE_EXACT64, _abi.PHASE_REF22
    if k in ("noalloc", "strucf"):
        pos = rng.uniform(0.0, 10.0, (case["atoms"], 3))
        n = (case["n1"], case["n2"], case["n3"])
        return pos, _grid(n, (5.0, 5.0, 0.0)), None
    if k == "hkl":
        cr = _perovskite(rng, case["cells"])
        m = case["hmax"]
        every = np.stack(np.meshgrid(*[np.arange(-m, m + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
        hkl = rng.permutation(every[np.any(every != 0, 1)])[: case["refl"]]
        hkl[0], hkl[1] = -m, m                        # the list spans its box whatever the seed
        return cr, hkl, _abi.default_opts(ldbw=1, phase=ref)
    if k == "menu":
        return _perovskite(rng, case["cells"]), _grid((case["n"], case["n"], 1), (5.0, 5.0, 0.0)), None
    if k == "aniso":
        return (_aniso(rng, case["cells"]), _grid((case["n1"], case["n2"], case["n3"]), (3.0, 2.2, 1.5)),
                _abi.default_opts(ldbw=1, phase=exact, engine=_abi.ENGINE_DIRECT))
    if k == "volume":
        n = (case["n1"], case["n2"], case["n3"])
        return (_alloy(rng, case["cells"]), _grid(n, tuple(0.08 * (x - 1) / 2 for x in n)),
                _abi.default_opts(ldbw=1, phase=exact, tc_kslice=case["kslice"]))
    if k == "average":
        return (_layers(rng, case["na"], case["nc"]),
                S.GridData.from_corners((-10, 0, -10), (10, 0, -10), (-10, 0, 10), inc=(case["n"], case["n"], 1)),
                _abi.default_opts(ldbw=1, phase=exact, fave=1.0, tc_kslice=case["kslice"]))
    if k == "lots":
        cr = _alloy(rng, case["cells"])
        n = (case["n1"], case["n2"], case["n3"])
        op = _abi.default_opts(ldbw=1, phase=exact, ilots=_abi.LOT_BOX, tc_kslice=case["kslice"])
        for a in range(3):
            op.ls_xyz[a] = case["ls"]
        op.kept = FR.attach_selections(op, lot_origins=rng.integers(1, case["cells"] + 1, (case["lots"], 3)))
        return cr, _grid(n, tuple(0.08 * (x - 1) / 2 for x in n)), op
    if k == "gradient":
        icc = (case["c1"], case["c2"], case["c3"])
        n = (case["n1"], case["n2"], case["n3"])
        return (_salt(rng, icc, 0.05, 0.1), _grid(n, tuple(0.1 * (x - 1) / 2 for x in n)),
                _abi.default_opts(ldbw=1, phase=exact, tc_kslice=case["kslice"]))
    if k == "population":
        crs, grids = _population(rng, case)
        return crs, grids, _abi.default_opts(ldbw=1, phase=exact)
    cr = _alloy(rng, case["cells"])
    pw = S.PowderSpec(a0=(3.6, 3.6, 3.6), gten=np.diag([3.6 ** 2] * 3),
                      hkl_del=(case["dhk"], case["dhk"], case["dl"]), ds_max=case["dsmax"], qmin=0.5,
                      qmax=case["qmax"], deltaq=case["dq"])
    return cr, pw, _abi.default_opts(ldbw=1, phase=exact)


def _targets(case, seed):
    """Target intensities and weights of a refinement: smooth in h, with noise, of the size of the data."""
    rng = np.random.default_rng([seed, 92])
    if case["kind"] == "gradient":
        np_ = case["n1"] * case["n2"] * case["n3"]
        it = case["c1"] * case["c2"] * case["c3"] * rng.gamma(1.0, 900.0, np_)
        return it, 1.0 / (it + 1.0)
    its = [8.0 * cells ** 3 * rng.gamma(1.0, 90.0, (pts, pts, 1)) for _, cells, pts, _ in _member_sizes(case)]
    return its, [1.0 / (t + 1.0) for t in its]


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def prepare(case, seed):
    cr, grid, op = _build(case, seed)
    k = case["kind"]
    st = dict(kind=k, cr=cr, grid=grid, op=op, ctx=default_context())
    if k in ("noalloc", "strucf"):
        n = grid.inc
        _, lmn, off = FR.fourier_lmn(grid.eck, grid.vi, n)
        _, istl = FR.four_stltab(grid, _metric((4.0, 4.0, 4.0)))
        one = _crystal(np.zeros((1, 3)), np.ones(1, np.int32), 1, (1, 1, 1), 1, (4.0, 4.0, 4.0))
        cf = FR.four_formtab(one, _abi.default_opts(ldbw=1))[0]
        fnum = ((n[0] + 1) // 2, n[1], n[2])
        st.update(lmn=np.asarray(lmn, np.int32), off=off, istl=istl, cf=cf, fnum=fnum)
        if k == "noalloc":
            st.update(x=_device(cr.T.copy()), cfd=_device(cf), istld=_device(istl.reshape(-1, order="F")),
                      out=torch.empty(grid.npoints, dtype=torch.complex128, device=DEV),
                      uvw=[np.ascontiguousarray(grid.vi[:, i]) for i in range(3)],
                      offf=off.reshape(-1, order="F").copy(), num=np.asarray(n, np.int32),
                      fn=np.asarray(fnum, np.int32))
    elif k == "menu":
        f = FR.Fourier(cr)
        f.ll, f.lr, f.ul = (-5, -5, 0), (5, -5, 0), (-5, 5, 0)
        f.nabs = f.nord = case["n"]
        f.temp, f.phase = "use", _abi.PHASE_REF22
        st["menu"] = f
    elif k in ("aniso", "average", "lots") or (k == "volume" and not case["host"]):
        st.update(pos=_device(cr.pos), isc=_device(cr.iscat), info=_abi.Info())
        for name in ("csf", "acsf"):
            st[name] = torch.empty(grid.npoints, dtype=torch.complex128, device=DEV)
        st["dsi"] = torch.empty(grid.npoints, dtype=torch.float64, device=DEV)
        adp = None
        if cr.is_anis:
            st["adp"] = _device(cr.ianis)
            adp = C.cast(st["adp"].data_ptr(), C.POINTER(C.c_int32))
        st["c"] = cr.to_c(pos_ptr=C.cast(st["pos"].data_ptr(), C.POINTER(C.c_double)),
                          iscat_ptr=C.cast(st["isc"].data_ptr(), C.POINTER(C.c_int32)), ianis_ptr=adp)
        st["g"] = grid.to_c()
    elif k == "gradient":
        it, wt = _targets(case, seed)
        shape = grid.inc
        st.update(pos=_device(cr.pos).requires_grad_(True), occ=_device(cr.atom_occ).requires_grad_(True),
                  it=_device(it).view(shape), wt=_device(wt).view(shape))
    elif k == "population":
        st["targets"], st["weights"] = _targets(case, seed)
    torch.cuda.synchronize()
    return st


def run(st):
    k, cr, grid, op, ctx = st["kind"], st["cr"], st["grid"], st["op"], st["ctx"]
    if k == "noalloc":
        u, v, w = st["uvw"]
        rc = ctx.lib.dgpu_four_strucf_noalloc(
            C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_void_p(st["x"].data_ptr()), cr.shape[0],
            _abi.dptr(u), _abi.dptr(v), _abi.dptr(w), _abi.dptr(st["offf"]), _abi.iptr(st["lmn"]),
            _abi.iptr(st["num"]), _abi.iptr(st["fn"]), C.c_void_p(st["cfd"].data_ptr()),
            C.c_void_p(st["istld"].data_ptr()), C.c_void_p(st["out"].data_ptr()))
        if rc:
            raise RuntimeError("four_strucf_noalloc: %d" % rc)
        return st["out"]
    if k == "strucf":
        return FR.four_strucf(cr, grid.vi[:, 0], grid.vi[:, 1], grid.vi[:, 2], st["off"], st["lmn"], grid.inc,
                              st["fnum"], st["cf"], st["istl"])
    if k == "hkl":
        return FR.calc_hkl(cr, op, grid, scale=0.5, exti=10.0)
    if k == "menu":
        r = st["menu"].run()
        return r.csf, r.dsi
    if k == "volume" and "pos" not in st:
        r = FR.four_run(cr, grid, op)
        return r.csf, r.dsi
    if k == "gradient":
        from diffusecode_gb300.autograd import chi2
        st["pos"].grad = st["occ"].grad = None
        loss = chi2(st["pos"], st["occ"], cr, grid, op, st["it"], st["wt"])
        loss.backward()
        return loss.detach(), st["pos"].grad, st["occ"].grad
    if k == "population":
        dsi, c2, gp, go, _ = FR.batch_run(cr, grid, op, st["targets"], st["weights"])
        return dsi, c2, gp, go
    if k == "powder":
        return FR.powder_complete(cr, grid, op)[0]
    ctx.check(ctx.lib.dgpu_four_run_device(
        ctx.h, C.byref(st["c"]), C.byref(st["g"]), C.byref(op), C.c_void_p(st["csf"].data_ptr()),
        C.c_void_p(st["acsf"].data_ptr()), C.c_void_p(st["dsi"].data_ptr()), C.byref(st["info"])))
    return st["csf"], st["dsi"]


# ---------------------------------------------------------------------------
# what a pass cannot do without: the inputs read and the outputs written once,
# and 8 floating-point operations (one complex multiply-add) for every pair of
# an atom and a point that Friedel's law does not give away

def _half(n):
    return (n[0] + 1) // 2 * n[1] * n[2] if all(x % 2 for x in n) else n[0] * n[1] * n[2]


def work(case):
    k = case["kind"]
    if k in ("noalloc", "strucf"):
        n = (case["n1"], case["n2"], case["n3"])
        pts = n[0] * n[1] * n[2]
        return {"bytes": 24 * case["atoms"] + 20 * pts // 2 + 16 * pts, "flops": 8 * case["atoms"] * (pts // 2)}
    if k == "hkl":
        m = 2 * case["hmax"] + 1
        atoms = 4.7 * case["cells"] ** 3
        return {"bytes": 28 * 5 * case["cells"] ** 3 + 36 * case["refl"], "flops": 8 * atoms * _half((m, m, m))}
    if k == "menu":
        n = (case["n"], case["n"], 1)
        atoms = 5 * case["cells"] ** 3
        return {"bytes": 28 * atoms + 40 * case["n"] ** 2, "flops": 8 * 0.94 * atoms * _half(n)}
    if k == "powder":
        atoms = 4 * case["cells"] ** 3
        pts = 2 / 3 * math.pi * (3.6 * case["dsmax"]) ** 3 / (case["dhk"] ** 2 * case["dl"])
        return {"bytes": 28 * atoms + 8 * (case["qmax"] - 0.5) / case["dq"], "flops": 8 * atoms * pts}
    if k == "population":
        b = f = 0
        for kind, cells, pts, _ in _member_sizes(case):
            atoms = (4 if kind else 8) * cells ** 3
            b += (28 + 32) * atoms + 24 * pts ** 2
            f += (8 + 32) * atoms * _half((pts, pts, 1))
        return {"bytes": b, "flops": f}
    if k == "gradient":
        atoms, n = 8 * case["c1"] * case["c2"] * case["c3"], (case["n1"], case["n2"], case["n3"])
        return {"bytes": (32 + 28) * atoms + 16 * n[0] * n[1] * n[2], "flops": (8 + 32) * atoms * _half(n)}
    if k == "average":
        n = (case["n"], case["n"], 1)
        atoms = 2 * case["na"] ** 2 * case["nc"]
        return {"bytes": 28 * atoms + 40 * case["n"] ** 2, "flops": 2 * 8 * 0.98 * atoms * _half(n)}
    n = (case["n1"], case["n2"], case["n3"])
    pts = n[0] * n[1] * n[2]
    atoms = (2 if k == "aniso" else 4) * case["cells"] ** 3
    summed = 4 * case["ls"] ** 3 * case["lots"] if k == "lots" else atoms
    return {"bytes": (32 if k == "aniso" else 28) * atoms + 24 * pts, "flops": 8 * summed * _half(n)}


# ---------------------------------------------------------------------------
# the same values in 64 bits, from the definitions

def _turn(x):
    """exp(2 pi i x)."""
    x = 2 * math.pi * (x - torch.round(x))
    return torch.complex(torch.cos(x), torch.sin(x))


def _axes(x, grid):
    """exp(2 pi i phase) of the atoms x (n, 3) split over the grid's axes: (n1, n), (n2, n), (n3, n)."""
    e = [torch.from_numpy(np.ascontiguousarray(grid.vi[:, a])).to(DEV) for a in range(3)]
    o = torch.from_numpy(np.ascontiguousarray(grid.eck[:, 0])).to(DEV)
    out = []
    for a in range(3):
        i = torch.arange(grid.inc[a], dtype=torch.float64, device=DEV)
        ph = i[:, None] * (x @ e[a])[None]
        out.append(_turn(ph + (x @ o)[None] if a == 1 else ph))
    return out


def _sums(x, grid, w=None):
    """sum_j w_j exp(2 pi i h.x_j) on the grid, shaped (n3, n2, n1)."""
    x = torch.as_tensor(x, device=DEV)
    n1, n2, n3 = grid.inc
    s = torch.zeros((n3 * n2, n1), dtype=torch.complex128, device=DEV)
    step = max(64, int(1e9 / 16 / (n2 * n3)))
    for a in range(0, x.shape[0], step):
        v, u, t = _axes(x[a:a + step], grid)
        if w is not None:
            u = u * torch.as_tensor(w[a:a + step], device=DEV, dtype=torch.float64)[None]
        s += (t[:, None, :] * u[None]).reshape(n3 * n2, -1) @ v.T
    return s.view(n3, n2, n1)


def _h(grid):
    h = grid.eck[:, 0][:, None, None, None] + sum(
        grid.vi[:, a][:, None, None, None] * np.arange(grid.inc[a]).reshape([-1 if b == a else 1 for b in (2, 1, 0)])
        for a in range(3))
    return torch.from_numpy(np.broadcast_to(h, (3,) + grid.inc[::-1]).copy()).to(DEV)


def _factor(cr_form, s2, b):
    f = cr_form[0] + sum(cr_form[2 * i - 1] * torch.exp(-cr_form[2 * i] * s2) for i in range(1, 5))
    return f * torch.exp(-b * s2)


def _table_s2(h, rten):
    """(sin theta / lambda)^2 on the 0.001 grid of the form-factor table, h rounded to single precision."""
    h = h.float().double()
    q = sum(h[a] * float(rten[a, b]) * h[b] for a in range(3) for b in range(3)) / 4
    return (torch.floor(torch.sqrt(q) * 1000 + 0.5) * 0.001) ** 2


def _structure_factor(cr, grid):
    """sum_t f_t(h) sum_j occ_j exp(2 pi i h.x_j), shaped (n3, n2, n1), and the factors."""
    s2 = _table_s2(_h(grid), cr.rten)
    f, fac = 0, []
    for t in range(cr.nscat):
        on = cr.iscat == t + 1
        fac.append(_factor(FORM[t], s2, B_ISO))
        f = f + fac[-1] * _sums(cr.pos[on], grid, None if cr.atom_occ is None else cr.atom_occ[on])
    return f, fac


def _laue(x):
    """sum of exp(2 pi i h k) for k = 0 .. n-1 is a plain sum here: x = (h, n)."""
    h, n = x
    return sum(_turn(h * k) for k in range(n))


def _chi2(cr, grid, it, wt):
    """chi^2 = sum w (|F|^2 - I_t)^2 and its gradients; it, wt shaped (n3, n2, n1)."""
    f, fac = _structure_factor(cr, grid)
    d = f.abs() ** 2 - it
    value = (wt * d * d).sum()
    h, (n1, n2, n3) = _h(grid), grid.inc
    gp = torch.zeros((cr.natoms, 3), dtype=torch.float64, device=DEV)
    go = torch.zeros(cr.natoms, dtype=torch.float64, device=DEV)
    for t in range(cr.nscat):
        q = 4 * wt * d * f.conj() * fac[t]
        on = np.nonzero(cr.iscat == t + 1)[0]
        step = max(64, int(5e8 / 16 / (n2 * n3)))
        for a in range(0, on.size, step):
            at = torch.from_numpy(on[a:a + step]).to(DEV)
            v, u, s = _axes(torch.from_numpy(cr.pos[on[a:a + step]]).to(DEV), grid)
            us = (s[:, None, :] * u[None]).reshape(n3 * n2, -1)
            w = 1.0 if cr.atom_occ is None else torch.from_numpy(cr.atom_occ[on[a:a + step]]).to(DEV).double()
            for c in range(4):
                m = q if c == 3 else q * h[c]
                r = (us * (m.reshape(n3 * n2, n1) @ v)).sum(0)
                if c == 3:
                    go[at] = r.real
                else:
                    gp[at, c] = -2 * math.pi * r.imag * w
    return value, gp, go


def _powder(cr, pw):
    """The rods inside the sphere, |F|^2 split over the two nearest bins of Q; a cubic cell, half space doubled."""
    ar = 1.0 / pw.a0[0]
    dh, dk, dl = pw.hkl_del
    qsp = np.zeros(int(math.floor((pw.qmax + pw.deltaq - pw.qmin) / pw.deltaq + 0.5)) + 3)
    for ih in range(int(pw.a0[0] * pw.ds_max / dh) + 1):
        hh = ih * dh
        u2 = (ar / hh) ** 2 if hh else 0.0            # the plane hh is placed at 1/hh (the reference's projection)
        rr = pw.ds_max ** 2 - u2
        if rr <= 0:
            continue
        kmax = int(math.sqrt(rr) / ar / dk)
        rods = []
        for ik in range(0 if ih == 0 else -kmax, kmax + 1):
            disc = pw.ds_max ** 2 / ar ** 2 - hh ** 2 - (ik * dk) ** 2
            if disc > 0:
                hi = int(math.sqrt(disc) / dl)
                rods.append((ik, 0 if ih == 0 and ik == 0 else -hi, hi))
        if not rods:
            continue
        k0, l0 = rods[0][0], min(r[1] for r in rods)
        nk, nl = rods[-1][0] - k0 + 1, max(r[2] for r in rods) - l0 + 1
        g = S.GridData(eck=np.repeat([[hh], [k0 * dk], [l0 * dl]], 4, 1), inc=(nl, nk, 1),
                       vi=np.array([[0, 0, 0], [0, dk, 0], [dl, 0, 0]], float))
        f, _ = _structure_factor(cr, g)
        inten = (f.abs() ** 2).cpu().numpy()[0]
        for ik, lo, hi in rods:
            ll = lo * dl + np.arange(hi - lo + 1) * dl
            q = 2 * math.pi * np.sqrt(hh * hh + (ik * dk) ** 2 + ll * ll) * ar
            i = inten[ik - k0, lo - l0: hi - l0 + 1]
            on = (q >= pw.qmin) & (q <= pw.qmax + pw.deltaq)
            x = (q[on] - pw.qmin) / pw.deltaq
            at = x.astype(np.int64)
            np.add.at(qsp, at, i[on] * (1 - (x - at)))
            np.add.at(qsp, at + 1, i[on] * (x - at))
    return 2 * qsp


def _flat(t):
    """(n3, n2, n1) as the library lays it out, first axis fastest."""
    return t.reshape(-1)


def _shaped(t):
    """(n3, n2, n1) as the array (n1, n2, n3) that the Python entries return."""
    return t.permute(2, 1, 0).contiguous()


def exact(case, seed):
    cr, grid, op = _build(case, seed)
    k = case["kind"]
    if k in ("noalloc", "strucf"):
        s2 = _table_s2(_h(grid), _metric((4.0, 4.0, 4.0)))
        f = _factor(FORM[0], s2, B_ISO) * _sums(cr, grid)
        f[:, :, (grid.inc[0] + 1) // 2:] = 0
        return _flat(f) if k == "noalloc" else _shaped(f)
    if k == "hkl":
        m = case["hmax"]
        g = _grid((2 * m + 1,) * 3, (m, m, m))
        f = _structure_factor(cr, g)[0].cpu().numpy()
        h = np.asarray(grid)
        fr = f[h[:, 2] + m, h[:, 1] + m, h[:, 0] + m]
        amp = np.abs(fr) / case["cells"] ** 3
        lam = 0.70932
        tth = 2 * np.arcsin(0.5 * lam * np.sqrt((h * h).sum(1)) / 4.0)
        amp = amp * (1 / (1 + 0.001 * 10.0 * amp ** 2 * lam ** 3 / np.sin(tth))) ** 0.25
        icalc = amp ** 2 * 0.5
        return icalc, np.sqrt(icalc), None            # a weak reflection's phase may sit at +-180
    if k == "aniso":
        h = _h(grid)
        s2 = _table_s2(h, cr.rten)
        ar = cr.ar
        f = 0
        for t in (1, 2):
            for a in (1, 2, 3):
                on = (cr.iscat == t) & (cr.ianis == a)
                if not on.any():
                    continue
                u = ADP[a - 1]
                arg = sum(w * u[c] * ar[i] * ar[j] * h[i] * h[j] for c, (i, j, w) in enumerate(
                    [(0, 0, 1), (1, 1, 1), (2, 2, 1), (1, 2, 2), (0, 2, 2), (0, 1, 2)]))
                f = f + _factor(FORM[t - 1], s2, 0.0) * torch.exp(-2 * math.pi ** 2 * arg) * _sums(cr.pos[on], grid)
        return _flat(f), _flat(f.abs() ** 2)
    if k in ("menu", "volume"):
        f, _ = _structure_factor(cr, grid)
        if k == "menu" or case["host"]:
            return _shaped(f), _shaped(f.abs() ** 2)
        return _flat(f), _flat(f.abs() ** 2)
    if k == "average":
        f, fac = _structure_factor(cr, grid)
        i = np.arange(cr.natoms) // 2
        na, nc = case["na"], case["nc"]
        cell = np.stack([i % na, i // na % na, i // (na * na)], 1)
        h = _h(grid)
        lat = _laue((h[0], na)) * _laue((h[1], na)) * _laue((h[2], nc)) / (na * na * nc)
        for t in range(2):
            on = cr.iscat == t + 1
            f = f - fac[t] * lat * _sums((cr.pos - cell)[on], grid)
        return _flat(f), _flat(f.abs() ** 2)
    if k == "lots":
        n, ls = case["cells"], case["ls"]
        origins = np.random.default_rng([seed, 91])
        _alloy(origins, n)                            # the draws before the origins
        origins = origins.integers(1, n + 1, (case["lots"], 3)) - 1
        s2 = _table_s2(_h(grid), cr.rten)
        fac = [_factor(FORM[t], s2, B_ISO) for t in range(2)]
        box = np.stack(np.meshgrid(*[np.arange(ls)] * 3, indexing="ij"), -1).reshape(-1, 3)
        dsi = 0
        for o in origins:
            c = (o + box) % n
            at = (c[:, 0] + n * (c[:, 1] + n * c[:, 2]))[:, None] * 4 + np.arange(4)
            pos = cr.pos[at] - c[:, None, :] + box[:, None, :]
            f = sum(fac[t] * _sums(pos[cr.iscat[at] == t + 1], grid) for t in range(2))
            dsi = dsi + f.abs() ** 2
        return None, _flat(dsi * (n ** 3 / (ls ** 3 * case["lots"])))
    if k == "gradient":
        it, wt = (_device(x).view(grid.inc).permute(2, 1, 0) for x in _targets(case, seed))
        return _chi2(cr, grid, it, wt)
    if k == "population":
        its, wts = _targets(case, seed)
        dsi, c2, gp, go = [], [], [], []
        for c, g, it, wt in zip(cr, grid, its, wts):
            f, _ = _structure_factor(c, g)
            dsi.append(_shaped(f.abs() ** 2))
            v, p, o = _chi2(c, g, _device(it).permute(2, 1, 0), _device(wt).permute(2, 1, 0))
            c2.append(v.item())
            gp.append(p)
            go.append(o)
        return dsi, np.array(c2), gp, go
    return _powder(cr, grid)
