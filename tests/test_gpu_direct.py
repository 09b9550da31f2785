"""CUDA-core engine at the edges of its work split: the 128-atom chunks, the
2, 4 or 8 points of a thread, and the groups of chunks, against the oracle.
Tolerance: the engine's intensity bound, max |I - I_ref| / (I_ref + N<|f|^2>)
<= 1e-5 (its FP32 phasors are good to 1e-7, and the oracle follows the same
phase arithmetic)."""
import numpy as np
import pytest

import kat_cases as K
from diffusecode_gb300 import _abi
from diffusecode_gb300 import fourier as FR
from diffusecode_gb300 import structures as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phase", [_abi.PHASE_REF22, _abi.PHASE_EXACT64], ids=["ref22", "exact64"])
@pytest.mark.parametrize("inc,natoms", [((1, 1, 1), 1), ((3, 1, 2), 127), ((7, 5, 1), 129), ((1, 9, 1), 700),
                                        ((33, 17, 1), 513), ((66, 9, 65), 260), ((5, 130, 63), 2050)])
def test_direct_work_split(oracle, ctx, inc, natoms, phase):
    cr, g = S.small_random(seed=51, natoms=natoms, nscat=2, inc=inc)
    cr.atom_occ = np.linspace(0.5, 1.5, natoms).astype(np.float32) if phase == _abi.PHASE_EXACT64 else None
    op = K.opts(phase=phase, engine=_abi.ENGINE_DIRECT)
    rc, csf, acsf, dsi, info = oracle.four_run(cr, g, op)
    r = FR.four_run(cr, g, op, ctx=ctx)
    assert r.info.engine_used == _abi.ENGINE_DIRECT
    floor = K.incoherent_floor(cr, g, op)
    assert K.rel_err(r.dsi, dsi, floor + 1e-30) <= 1e-5


@pytest.mark.parametrize("natoms,nscat", [(128, 8), (129, 9), (1025, 9), (16384, 3), (65536, 2), (65537, 2)])
def test_preparation_block_edges(oracle, ctx, natoms, nscat):
    """The gather by type with 128 or 1024 atoms per block (at most 65 536
    atoms of at most 8 types, or more), whole and broken last blocks, on a few
    points; same tolerance."""
    cr, g = S.small_random(seed=52, natoms=natoms, nscat=nscat, inc=(3, 2, 1))
    op = K.opts(phase=_abi.PHASE_EXACT64, engine=_abi.ENGINE_DIRECT)
    rc, csf, acsf, dsi, info = oracle.four_run(cr, g, op)
    r = FR.four_run(cr, g, op, ctx=ctx)
    assert K.rel_err(r.dsi, dsi, K.incoherent_floor(cr, g, op)) <= 1e-5


@pytest.mark.parametrize("natoms", [1, 2, 63, 64, 65, 128, 129, 1000])
def test_one_type_preparation(oracle, ctx, natoms):
    """four_strucf's own preparation of one type's atoms around the padding
    (64) and a block (128).  Tolerance: that of the per-type entry, 1e-5 of the
    largest sum."""
    cr, g = S.small_random(seed=71, natoms=natoms, nscat=1, inc=(13, 11, 3))
    _, lmn, off = oracle.fourier_lmn(g.eck, g.vi, g.inc)
    args = (cr.pos, g.vi[:, 0], g.vi[:, 1], g.vi[:, 2], off, lmn, g.inc, (7, 11, 3))
    _, istl = oracle.stltab(g, cr.rten)
    cf = oracle.formtab(cr, K.opts())[0]
    a = oracle.four_strucf(*args, cf, istl)
    b = FR.four_strucf(*args, cf, istl, ctx=ctx)
    assert np.all(b[7:] == 0)
    assert np.max(np.abs(b - a)) <= 1e-5 * np.abs(a).max()
