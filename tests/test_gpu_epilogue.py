"""The epilogue in one pass (combine, Friedel mirror, statistics): grids whose
halved axis is the first, second or third, single points and rows, and grids
that are not halved, against the oracle's four_run (csf, dsi) and against
four_qinfo's definition evaluated here on the returned dsi.  Tolerances: the
engine's intensity bound 1e-5 for dsi; the statistics are FP64 sums, minima and
maxima of the same numbers, 1e-12."""
import numpy as np
import pytest

import kat_cases as K
from diffusecode_gb300 import _abi
from diffusecode_gb300 import fourier as FR
from diffusecode_gb300 import structures as S

pytestmark = pytest.mark.gpu


def _centred(inc, step):
    """About the origin, slightly sheared: fourier_lmn takes no row along b or
    c alone."""
    vi = np.diag(step) + (1.0 - np.eye(3)) / 64.0
    lo = -0.5 * vi @ (np.asarray(inc) - 1)
    eck = np.repeat(lo[:, None], 4, axis=1)
    for a in range(3):
        eck[:, a + 1] += vi[:, a] * (inc[a] - 1)
    return S.GridData(eck=eck, vi=vi, inc=inc)


@pytest.mark.parametrize("engine", [_abi.ENGINE_DIRECT, _abi.ENGINE_TC], ids=["direct", "tc"])
@pytest.mark.parametrize("inc", [(1, 1, 1), (9, 1, 1), (1, 9, 1), (1, 1, 7), (1, 5, 7), (5, 1, 7), (3, 5, 7),
                                 (4, 5, 3), (65, 33, 9)])
def test_epilogue_one_pass(oracle, ctx, inc, engine):
    cr, _ = S.small_random(seed=61, natoms=150, nscat=2)
    g = _centred(inc, (0.5, 0.25, 1.0 / 3.0))
    op = K.opts(phase=_abi.PHASE_EXACT64, engine=engine, diff_scale=1.7)
    rc, csf, acsf, dsi, info = oracle.four_run(cr, g, op)
    r = FR.four_run(cr, g, op, ctx=ctx)
    odd = all(n % 2 for n in inc)
    assert r.info.friedel_dim == (next(a + 1 for a in range(3) if inc[a] > 1) if odd and max(inc) > 1 else 0)
    floor = 1.7 * K.incoherent_floor(cr, g, op)
    assert K.rel_err(r.dsi, dsi, floor) <= 1e-5
    np.testing.assert_allclose(np.abs(r.csf) ** 2, r.dsi, rtol=1e-12, atol=1e-12 * r.dsi.max())
    assert np.all(np.abs(r.csf - csf) <= 1e-5 * np.abs(csf) + 1e-5 * np.sqrt(floor))
    assert not np.any(r.acsf)
    h = g.hkl()
    bragg = np.all(h == np.trunc(h), axis=0)
    dif = r.dsi[~bragg]
    res = list(r.info.res)
    assert res[0] == 6.0
    if dif.size:
        np.testing.assert_allclose(res[1:4], [dif.min(), dif.max(), dif.mean()], rtol=1e-12)
        np.testing.assert_allclose(res[4] ** 2, max(0.0, np.mean(dif ** 2) - dif.mean() ** 2),
                                   rtol=1e-9, atol=1e-12 * np.mean(dif ** 2))
    if bragg.any():
        np.testing.assert_allclose(res[5:7], [r.dsi[bragg].min(), r.dsi[bragg].max()], rtol=1e-12)


@pytest.mark.parametrize("engine", [_abi.ENGINE_DIRECT, _abi.ENGINE_TC], ids=["direct", "tc"])
@pytest.mark.parametrize("vi", [np.diag([0.21, 0.17, 0.33]), np.array([[0, 0, 0.21], [0.17, 0, 0], [0, 0.33, 0]]),
                                np.array([[0.21, 0.03, 0], [0, 0.17, 0], [0, 0, 0.33]])],
                         ids=["axes", "permuted", "sheared"])
def test_average_lattice_sum(oracle, ctx, vi, engine):
    """<F> with the lattice sum's series tabulated per component of h (grids
    along the reciprocal axes, in any order) and evaluated per point (a
    component that changes along two axes); cells from a shifted origin.
    Tolerance: the intensity bound of the other <F> comparisons, 1e-5."""
    cr, _ = S.small_lots_anis(anis=False, nextra=0)
    inc = (12, 9, 7)
    lo = np.array([-1.1, -0.7, -0.9])
    eck = np.repeat(lo[:, None], 4, axis=1)
    for a in range(3):
        eck[:, a + 1] += vi[:, a] * (inc[a] - 1)
    g = S.GridData(eck=eck, vi=vi, inc=inc)
    op = K.opts(phase=_abi.PHASE_EXACT64, engine=engine, fave=1.0)
    rc, csf, acsf, dsi, info = oracle.four_run(cr, g, op)
    r = FR.four_run(cr, g, op, ctx=ctx)
    assert K.rel_err(r.dsi, dsi, K.incoherent_floor(cr, g, op)) <= 1e-5
    assert np.max(np.abs(r.acsf - acsf)) <= 1e-5 * np.abs(acsf).max()


@pytest.mark.parametrize("cells", [5, 12])
@pytest.mark.parametrize("inc", [(131, 1, 1), (41, 37, 1), (41, 1, 37), (1, 41, 37), (21, 19, 17)])
def test_refined_points(oracle, ctx, inc, cells):
    """Points listed for the exact sums along a row, on planes across every
    axis and in a box: groups of eight that are one run, that start new lines
    and that the list's end cuts short; types of 125 to 5184 atoms, less than a
    block's threads and more than one FP32 chunk.  Tolerances as for <F>
    elsewhere: 1e-5 of the intensity bound, 1e-6 of max |<F>|."""
    cr, _ = S.perovskite_plane(cells=cells, vacancy=0.3)
    g = _centred(inc, (0.05, 0.06, 0.07))
    op = K.opts(phase=_abi.PHASE_EXACT64, fave=1.0, engine=_abi.ENGINE_TC)
    rc, csf, acsf, dsi, info = oracle.four_run(cr, g, op)
    r = FR.four_run(cr, g, op, ctx=ctx)
    assert r.info.refined > 0
    assert np.max(np.abs(r.acsf - acsf)) <= 1e-6 * np.abs(acsf).max()
    assert K.rel_err(r.dsi, dsi, K.incoherent_floor(cr, g, op)) <= 1e-5


@pytest.mark.parametrize("ano", [0, 1])
@pytest.mark.parametrize("form", [_abi.FORM_TABLE, _abi.FORM_ANALYTIC], ids=["table", "analytic"])
@pytest.mark.parametrize("kslice,scale", [(0, 1.0), (64, 2.25)])
def test_combine_factors(oracle, ctx, form, ano, kslice, scale):
    """Real and complex form factors from the table and from the formula, one
    K slice and more than a round of eight, with and without an intensity
    scale.  Tolerances as above."""
    cr, _ = S.small_random(seed=67, natoms=1500, nscat=2)
    cr.delfr[:] = [0.0, 0.3, -1.2]
    cr.delfi[:] = [0.0, 0.7, 2.1]
    g = _centred((9, 7, 5), (0.5, 0.25, 1.0 / 3.0))
    op = K.opts(phase=_abi.PHASE_EXACT64, engine=_abi.ENGINE_TC, form=form, ano=ano, tc_kslice=kslice,
                diff_scale=scale)
    rc, csf, acsf, dsi, info = oracle.four_run(cr, g, op)
    r = FR.four_run(cr, g, op, ctx=ctx)
    assert K.rel_err(r.dsi, dsi, scale * K.incoherent_floor(cr, g, op)) <= 1e-5
    dif = r.dsi[~np.all(g.hkl() == np.trunc(g.hkl()), axis=0)]
    np.testing.assert_allclose(list(r.info.res)[1:4], [dif.min(), dif.max(), dif.mean()], rtol=1e-12)


@pytest.mark.parametrize("cell", [(4.0, 4.0, 4.0, 90.0, 90.0, 90.0), (5.1, 7.3, 9.7, 70.0, 110.0, 55.0),
                                  (1000.0, 3.0, 0.5, 90.0, 90.0, 120.0)])
def test_stltab_estimate(oracle, ctx, cell):
    """The table index where its FP32 estimate decides it and where it does
    not: the origin, half integers hit exactly (cubic, a = 4: 1000 |h| / 8),
    a metric whose mixed terms nearly cancel the others, and one with axes of
    very different length.  Whole numbers: equal."""
    r = S.reciprocal_metric(*cell)
    top = 8.0 / np.sqrt(max(r[k, k] for k in range(3)))
    g = _centred((81, 61, 41), (top / 81, top / 61, top / 41))
    for vi in (g.vi, np.diag([0.004, 0.012, 0.02])):
        h = S.GridData(eck=g.eck if vi is g.vi else np.zeros((3, 4)), vi=vi, inc=g.inc)
        rc_o, a = oracle.stltab(h, r)
        rc_g, b = FR.four_stltab(h, r, ctx=ctx)
        assert rc_o == rc_g == 0
        np.testing.assert_array_equal(b, a)


@pytest.mark.parametrize("engine", [_abi.ENGINE_DIRECT, _abi.ENGINE_TC], ids=["direct", "tc"])
@pytest.mark.parametrize("n", [1, 3], ids=["one-point", "row-about-bragg"])
def test_sigma_of_equal_values(ctx, n, engine):
    """res(4) where all diffuse points have one value: a single point off the
    Bragg positions, and the two of a row about one that are each other's
    Friedel mates.  sqrt(mean v^2 - (mean v)^2) is then sqrt of a rounding
    error: at most two roundings of the squares, 2^-52 v^2, either sign; never
    NaN."""
    for seed in range(12):
        cr, _ = S.small_random(seed=seed, natoms=60, nscat=2)
        if n == 1:
            g = S.GridData.from_corners((0.3, 0.2, 0.1), (0.3, 0.2, 0.1), (0.3, 0.2, 0.1), inc=(1, 1, 1))
        else:
            g = S.GridData.from_corners((-0.25, 0, 0), (0.25, 0, 0), (-0.25, 0, 0), inc=(3, 1, 1))
        r = FR.four_run(cr, g, K.opts(phase=_abi.PHASE_EXACT64, engine=engine), ctx=ctx)
        dif = r.dsi[~np.all(g.hkl() == np.trunc(g.hkl()), axis=0)]
        assert dif.size == (1 if n == 1 else 2) and np.all(dif == dif[0])
        assert 0.0 <= r.info.res[4] <= np.sqrt(2.0 ** -52) * dif[0]
