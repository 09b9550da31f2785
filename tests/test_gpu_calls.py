"""What a call leaves behind and takes: runs that are cancelled while the GPU
works, arguments that a call reports and another takes back."""
import ctypes as C

import numpy as np
import pytest

from diffusecode_gb300 import _abi
from diffusecode_gb300 import structures as S

pytestmark = pytest.mark.gpu


def _volume(inc):
    """108 000 atoms on inc^3 points: about 0.1 s of CUDA-core sums at inc 121,
    0.5 s at inc 201."""
    return S.fcc_alloy_volume(cells=30, sweeps=0, inc=inc, step=8.0 / inc)


class _Device:
    """A crystal's arrays and a grid's outputs on the device, and the call."""

    def __init__(self, cr, g):
        import torch
        dev = torch.device("cuda:0")
        self.cr, self.g = cr, g            # cr: the arrays that c points to
        self.pos = torch.from_numpy(np.ascontiguousarray(cr.pos)).to(dev)
        self.isc = torch.from_numpy(np.ascontiguousarray(cr.iscat, dtype=np.int32)).to(dev)
        self.c = cr.to_c(pos_ptr=C.cast(self.pos.data_ptr(), C.POINTER(C.c_double)),
                         iscat_ptr=C.cast(self.isc.data_ptr(), C.POINTER(C.c_int32)))
        self.out = [torch.zeros(n * g.npoints, dtype=torch.float64, device=dev) for n in (2, 2, 1)]

    def run(self, ctx, op):
        import torch
        torch.cuda.synchronize()
        info = _abi.Info()
        p = [C.c_void_p(t.data_ptr()) for t in self.out]
        return ctx.lib.dgpu_four_run_device(ctx.h, C.byref(self.c), C.byref(self.g.to_c()), C.byref(op), *p,
                                            C.byref(info))

    def reuse(self, value):
        """The outputs as another user of the memory finds them: filled on
        torch's stream, and whether the values last."""
        import torch
        for t in self.out:
            t.fill_(value)
        torch.cuda.synchronize()
        torch.cuda._sleep(10**8)           # 50 ms for anything still on its way
        torch.cuda.synchronize()
        return all(bool((t == value).all()) for t in self.out)


@pytest.mark.parametrize("engine", [_abi.ENGINE_DIRECT, _abi.ENGINE_TC], ids=["direct", "tc"])
@pytest.mark.parametrize("kind", ["plain", "average", "lots"])
def test_cancelled_run_has_left_the_outputs(ctx, engine, kind):
    """A run that returns DGPU_ERR_CANCELLED writes nothing afterwards: the
    flag is up from the start, and is polled with the first sums on the
    device."""
    d = _Device(*_volume(121))
    flag = C.c_int32(1)
    op = _abi.default_opts(ldbw=1, phase=_abi.PHASE_EXACT64, engine=engine, fave=float(kind == "average"),
                           tc_kslice=8192)
    if kind == "lots":
        op.ilots, op.lot_all = _abi.LOT_BOX, 1
    op.cancel = C.pointer(flag)
    assert d.run(ctx, op) == _abi.DGPU_ERR_CANCELLED
    assert d.reuse(3.0)


@pytest.mark.parametrize("fave", [0.0, 1.0])
def test_cancel_while_the_sums_run(ctx, fave):
    """A flag that goes up while the first sums of a run are on the device
    (half a second of CUDA-core sums, the flag after a tenth) ends the run:
    neither the combine nor, with <F>, the main sums follow.  Nothing of the
    result is written then."""
    import threading
    import time
    small = _Device(*_volume(21))
    op = _abi.default_opts(ldbw=1, phase=_abi.PHASE_EXACT64, engine=_abi.ENGINE_DIRECT, fave=fave)
    assert small.run(ctx, op) == 0                # kernels loaded
    d = _Device(*_volume(201))
    for t in d.out:
        t.fill_(7.0)
    flag = C.c_int32(0)
    op.cancel = C.pointer(flag)
    timer = threading.Timer(0.1, lambda: setattr(flag, "value", 1))
    timer.start()
    t0 = time.perf_counter()
    rc = d.run(ctx, op)
    assert time.perf_counter() - t0 > 0.1
    timer.join()
    assert rc == _abi.DGPU_ERR_CANCELLED
    assert bool((d.out[0] == 7.0).all()) and bool((d.out[2] == 7.0).all())
    assert d.reuse(3.0)


def test_reported_tile_can_be_asked_for(ctx):
    """info.tc_config of a run goes back into the options of the next (tile
    width and atoms per K slice): 51 columns, which the kernel runs 56 wide."""
    from diffusecode_gb300 import fourier as FR
    cr, g = S.fcc_alloy_volume(cells=8, sweeps=0, inc=101)
    a = FR.four_run(cr, g, _abi.default_opts(ldbw=1, engine=_abi.ENGINE_TC, tc_vimg=1), ctx=ctx)
    axis, n, nbuf, kslice = a.info.tc_config
    assert n in range(16, 129, 16)
    b = FR.four_run(cr, g, _abi.default_opts(ldbw=1, engine=_abi.ENGINE_TC, tc_vimg=1, tc_tile_n=n, tc_kslice=kslice),
                    ctx=ctx)
    assert list(b.info.tc_config)[1:] == [n, nbuf, kslice]


@pytest.mark.parametrize("lots", [False, True])
@pytest.mark.parametrize("engine", [_abi.ENGINE_DIRECT, _abi.ENGINE_TC], ids=["direct", "tc"])
def test_gradient_into_the_positions(ctx, engine, lots):
    """chi2_grad_device may write its gradient over the positions it was given
    (they are read before anything is written): equal to the gradient in an
    array of its own up to the order of the lots' atomic sums, 1e-12."""
    import torch
    dev = torch.device("cuda:0")
    cr, g = S.small_lots_anis(anis=False)
    op = _abi.default_opts(ldbw=1, phase=_abi.PHASE_EXACT64, engine=engine, tc_kslice=64)
    if lots:
        op.ilots, op.lot_all = _abi.LOT_BOX, 1
        for k, n in enumerate((3, 2, 2)):
            op.ls_xyz[k] = n
    target = torch.from_numpy(np.random.default_rng(4).uniform(0, 100, g.npoints)).to(dev)

    def grad(shared):
        d = _Device(cr, g)
        gp = d.pos if shared else torch.zeros_like(d.pos)
        go = torch.zeros(cr.natoms, dtype=torch.float64, device=dev)
        chi2 = np.zeros(1)
        info = _abi.Info()
        torch.cuda.synchronize()
        ctx.check(ctx.lib.dgpu_chi2_grad_device(ctx.h, C.byref(d.c), C.byref(g.to_c()), C.byref(op),
                                                C.c_void_p(target.data_ptr()), None, _abi.dptr(chi2),
                                                C.c_void_p(gp.data_ptr()), C.c_void_p(go.data_ptr()), C.byref(info)))
        return chi2[0], gp.cpu().numpy(), go.cpu().numpy()

    a, b = grad(False), grad(True)
    assert np.abs(a[1]).max() > 0
    for x, y in zip(a, b):
        np.testing.assert_allclose(y, x, rtol=1e-12, atol=1e-12 * np.abs(x).max())
