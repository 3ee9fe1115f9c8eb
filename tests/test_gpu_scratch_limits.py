"""Scratch that only makes a call faster is done without where there is no room for it.

Under a limit a few hundred kilobytes above what the context needs, the FP64 sandwich
takes its whole K range in one chunk instead of many (agreement to the FP64 bar of the
other tests, 1e-10 of max|g|), and the dV windows of eight q slots are made one slot at a
time instead of together (the same bits)."""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu


def test_fp64_chunk_partials(monkeypatch):
    s = synth.make_system("case", dict(kind="l12", a=7.1, fft=(32, 32, 32), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], nbnds=16,
                                       npw=800, ls=(0,), nsym_max=1))

    def run(ctx):
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        return ctx.run([0, 0], [0, 1], non_loc=False)

    with LelphGPU(s, "fp64", route="real") as ctx:
        ref = run(ctx)
        held = ctx.stats()["device_bytes"]
    one = 16 * 2 * s.nmodes * 16 * 16       # the partial sums of one chunk; there are several
    monkeypatch.setenv("LELPH_DEVICE_LIMIT", str(held - 2 * one))
    with LelphGPU(s, "fp64", route="real") as ctx:
        g = run(ctx)
        assert ctx.stats()["device_bytes"] <= held - 2 * one
    assert np.abs(g - ref).max() < 1e-10 * np.abs(ref).max()


def test_windows_of_many_slots(monkeypatch):
    s = synth.make_system("case", dict(kind="l12", a=7.1, fft=(48, 48, 48), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], nbnds=2,
                                       npw=800, ls=(0,), nsym_max=1))
    n = 8

    def run(ctx):
        for i in reversed(range(n)):
            ctx.set_q(i, s.qpts[0], s.eigVec[0], (i + 1) * s.dVscf[0])
        return ctx.run(list(range(n)), [0] * n, non_loc=False)

    with LelphGPU(s, "mixed", route="real") as ctx:
        ref = run(ctx)
        held = ctx.stats()["device_bytes"]
    box = 8 * s.nmodes * int(np.prod(s.fft_dims))       # one slot's dV in FP32; the scratch holds eight
    monkeypatch.setenv("LELPH_DEVICE_LIMIT", str(held - 3 * box))
    with LelphGPU(s, "mixed", route="real") as ctx:
        g = run(ctx)
        assert ctx.stats()["device_bytes"] <= held - 3 * box
    assert np.array_equal(g, ref)
