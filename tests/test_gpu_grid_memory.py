"""Device memory of a context whose batch runs and one-call stage use different product grids.

A context that prepares before its q slots are loaded, and then runs, holds no more
than one that never left the plain grid: what prepare made for the other grid is
handed over or given back.  One that alternates between the two holds one set of
operands where two would take more than an eighth of the memory it may hold, and
gives the inactive grid's up when another allocation needs it.  Results are the bits
of the usual order's throughout."""
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


def _alternate(ctx, s):
    args = (s.qpts[0], s.eigVec[0], s.dVscf[0])
    return [x for _ in range(2) for x in (ctx.compute_elphq(*args), _run(ctx, s))]


def test_alternating_grids_share_one_set(monkeypatch):
    s = synth.make_system("case", CELL)
    with LelphGPU(s, "mixed", route="real") as ctx:
        ref = _alternate(ctx, s)
    monkeypatch.setenv("LELPH_PLAIN_GRID", "1")
    with LelphGPU(s, "mixed", route="real") as ctx:
        ctx.compute_elphq(s.qpts[0], s.eigVec[0], s.dVscf[0])
        one = ctx.stats()["device_bytes"]
        pts = ctx.grid()["points"]
    monkeypatch.delenv("LELPH_PLAIN_GRID")
    second = 24 * 8 * pts * s.nk_bz        # operands of 8 bands on the plain grid
    limit = one + second // 2
    monkeypatch.setenv("LELPH_DEVICE_LIMIT", str(limit))
    with LelphGPU(s, "mixed", route="real") as ctx:
        got = _alternate(ctx, s)
        assert ctx.stats()["device_bytes"] <= limit
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))


def test_the_inactive_grid_gives_way(monkeypatch):
    s = synth.make_system("case", CELL)
    args = (s.qpts[0], s.eigVec[0], s.dVscf[0])
    with LelphGPU(s, "mixed", route="real") as ctx:
        ref = _alternate(ctx, s)
        held = ctx.stats()["device_bytes"]
    nslots = 60
    new = nslots * 16 * s.nmodes * int(np.prod(s.fft_dims))  # the slot arrays grow to this, beside the old ones
    limit = held + new - (20 << 20)
    monkeypatch.setenv("LELPH_DEVICE_LIMIT", str(limit))
    with LelphGPU(s, "mixed", route="real") as ctx:
        got = _alternate(ctx, s)
        assert ctx.stats()["device_bytes"] >= held          # both sets are kept
        ctx.set_q(nslots - 1, *args)
        assert ctx.stats()["device_bytes"] < held + new - (60 << 20)  # one set (over 60 MB) and the old slots are gone
        got += _alternate(ctx, s)
    assert all(np.array_equal(a, b) for a, b in zip(got, ref + ref))
