"""The fused wavefunction boxes are the ones that run.

Under profiling the passes' time of the preparation is zero where one CTA transforms
a whole box, and positive where the projections are held off the tensor cores and with
them the boxes in their passes.  The systems cover one, two and four copies and eight
of the ten box lengths; both preparations agree to the norm 2e-6 of the mixed form.
(27- and 30-point lengths and three copies do not occur together with boxes that fit
in shared memory in the cells at hand.)"""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

BASE = dict(kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], nbnds=3, ls=(0,), nsym_max=1)
FCC = dict(BASE, kind="diamond", a=10.26, fft=(48, 48, 48))
SC = dict(BASE, kind="l12", a=7.1, fft=(64, 64, 64))
SYSTEMS = [dict(FCC, npw=260), dict(FCC, npw=700), dict(FCC, npw=900), dict(FCC, npw=1200), dict(FCC, npw=1600),
           dict(SC, npw=520), dict(SC, npw=1200), dict(SC, npw=3000), dict(SC, npw=4200)]


def _run(s):
    with LelphGPU(s, "mixed", route="real") as ctx:
        ctx.set_profiling(True)
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        return ctx.run([0] * s.nk_bz, list(range(s.nk_bz)), non_loc=False), ctx.stats()["prep_fft_ms"], ctx.grid()


def test_fused_boxes_run(monkeypatch):
    lengths, copies = set(), set()
    for o in SYSTEMS:
        s = synth.make_system("case", o)
        monkeypatch.delenv("LELPH_PROJ_TC", raising=False)
        fused, ms, grid = _run(s)
        assert ms == 0
        monkeypatch.setenv("LELPH_PROJ_TC", "0")
        passes, ms, _ = _run(s)
        assert ms > 0
        assert np.linalg.norm(fused - passes) < 2e-6 * np.linalg.norm(passes)
        lengths |= set(grid["n"])
        copies.add(grid["copies"])
    assert lengths >= {12, 15, 16, 18, 20, 24, 25, 32} and copies >= {1, 2, 4}, (lengths, copies)
