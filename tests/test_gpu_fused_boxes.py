"""Wavefunction boxes transformed in shared memory, and windows of several q slots.

One CTA per box (k_box_fft_split) against the pass-by-pass preparation, which a
context takes when its projections do not run on the tensor cores: the local
term of both, for box lengths from 12 to 32, one to four copies, spinors and
two spins, ragged spheres.  Both transform in FP32, so they agree to the norm
2e-6 that the mixed form keeps to FP64.  The dV windows of a batch of q slots
with a gap are the bits of the windows built for one slot at a time.
"""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

BASE = dict(kgrid=(2, 2, 2), qpts=[(0.5, 0, 0), (0.5, 0.5, 0), (0.5, 0.5, 0.5)], nbnds=3, ls=(0,))
SYSTEMS = {
    "small": dict(BASE, kind="diamond", a=10.26, fft=(18, 18, 18), npw=(90, 110)),
    "two copies": dict(BASE, kind="l12", a=7.1, fft=(48, 48, 48), npw=2500),
    "largest": dict(BASE, kind="l12", a=7.1, fft=(64, 64, 64), npw=4200),
    "spinors": dict(BASE, kind="rocksalt8", a=8.0, fft=(32, 32, 32), npw=(500, 700), nspinor=2, nmag=4, soc=True,
                    ls=(0, 1), nsym_max=1, kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)]),
    "two spins": dict(BASE, kind="zincblende", a=10.2, fft=(30, 30, 32), npw=(350, 700), nspin=2, nmag=2,
                      timerev=True),
}


def _run(ctx, s, slots):
    for iq in slots:
        ctx.set_q(iq, s.qpts[iq], s.eigVec[iq], s.dVscf[iq])
    return ctx.run(np.repeat(slots, s.nk_bz), np.tile(np.arange(s.nk_bz), len(slots)), non_loc=False)


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_fused_boxes_equal_the_passes(name, monkeypatch):
    s = synth.make_system("case", SYSTEMS[name])
    with LelphGPU(s, "mixed", route="real") as ctx:
        fused = _run(ctx, s, [0])
    monkeypatch.setenv("LELPH_PROJ_TC", "0")
    with LelphGPU(s, "mixed", route="real") as ctx:
        passes = _run(ctx, s, [0])
    assert np.linalg.norm(fused - passes) < 2e-6 * np.linalg.norm(passes)


def test_windows_of_slots_with_a_gap():
    s = synth.make_system("case", SYSTEMS["two copies"])
    with LelphGPU(s, "mixed", route="real") as ctx:
        both = _run(ctx, s, [0, 2]).reshape(2, s.nk_bz, *(s.nmodes, s.nspin, s.nbnds, s.nbnds))
    for i, iq in enumerate((0, 2)):
        with LelphGPU(s, "mixed", route="real") as ctx:
            one = _run(ctx, s, [iq]).reshape(both[i].shape)
        assert np.array_equal(both[i], one)
