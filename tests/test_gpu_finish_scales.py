"""Operand scales of the mixed form whose product leaves FP32's range.

Large projection sets (spinors, d projectors, 40 bands: one atom's projections at a
time in the finish kernel) with a dV of 2^-100 and wavefunctions of 2^-12 times the
usual: every operand scale is a power of two, so the local matrix elements are
2^-124 times the usual ones.  Wavefunctions of 2^-70 times the usual: the nonlocal
ones are 2^-140 times the usual ones.  Within the mixed form's bar (norm 2e-6)."""
import dataclasses

import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu


def _run(s, non_loc=False):
    with LelphGPU(s, "mixed", route="real") as ctx:
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        return ctx.run([0] * s.nk_bz, list(range(s.nk_bz)), non_loc=non_loc)


SOC = dict(kind="rocksalt8", a=8.0, fft=(32, 32, 32), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=700, nbnds=40,
           ls=(0, 1, 2), nspinor=2, nmag=4, soc=True, nsym_max=1)


def test_small_dv_and_wavefunctions():
    s = synth.make_system("case", SOC)
    g = _run(s)
    t = dataclasses.replace(s, dVscf=s.dVscf * 2.0 ** -100, wfc=[w * 2.0 ** -12 for w in s.wfc])
    h = _run(t) * 2.0 ** 124
    assert np.linalg.norm(h - g) < 2e-6 * np.linalg.norm(g)


def test_small_projections():
    s = synth.make_system("case", SOC)
    s = dataclasses.replace(s, dVscf=0 * s.dVscf)
    g = _run(s, non_loc=True)
    h = _run(dataclasses.replace(s, wfc=[w * 2.0 ** -70 for w in s.wfc]), non_loc=True) * 2.0 ** 140
    assert np.linalg.norm(h - g) < 2e-6 * np.linalg.norm(g)
