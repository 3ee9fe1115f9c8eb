"""Device memory of a context whose batch runs and one-call stage use different product grids.

A context that prepares before its q slots are loaded, and then runs, holds no more
than one that never left the plain grid: what prepare made for the other grid is
handed over or given back.  Results are the bits of the usual order's."""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

CELL = dict(kind="l12", a=7.1, fft=(48, 48, 48), kgrid=(2, 2, 2), qpts=[(0.5, 0.5, 0.5)], nbnds=8, npw=2500, ls=(0, 1))


def _load(ctx, s):
    ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])


def _run(ctx, s):
    return ctx.run([0] * s.nk_bz, list(range(s.nk_bz)))


@pytest.mark.parametrize("route", ["real", "gspace"])
def test_prepare_before_the_slots(route, monkeypatch):
    s = synth.make_system("case", CELL)
    with LelphGPU(s, "mixed", route=route) as ctx:
        _load(ctx, s)
        ref = _run(ctx, s)
        assert ctx.grid()["copies"] > 1
        usual = ctx.stats()["device_bytes"]
    with LelphGPU(s, "mixed", route=route) as ctx:
        ctx.prepare()
        _load(ctx, s)
        g = _run(ctx, s)
        again = _run(ctx, s)
        assert ctx.stats()["device_bytes"] <= usual
    monkeypatch.setenv("LELPH_PLAIN_GRID", "1")
    with LelphGPU(s, "mixed", route=route) as ctx:
        _load(ctx, s)
        _run(ctx, s)
        assert usual <= ctx.stats()["device_bytes"]
    assert np.array_equal(g, ref) and np.array_equal(again, ref)
