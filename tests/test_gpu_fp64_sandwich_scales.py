"""Scales of the FP64 sandwich's fixed-point operands.

Each (mode, spin) has its own: a NaN or an infinity in the dV of one spin (with
products dV psi above 1, which a scale of 1 would not hold), or a dV of one spin
2^40 times the other's, leaves the other spin's matrix elements
at the FP64 bar of the other tests (1e-10 of their own max|g|).  A row's scale is
that of the products it holds: components of dV 2^60 above the rest that meet only
zeros of psi change nothing."""
import dataclasses

import numpy as np
import pytest

import elph_oracle as O
from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

TOL = 1e-10
LSDA = dict(kind="zincblende", a=10.2, fft=(18, 20, 16), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=150, nbnds=4,
            ls=(0, 1), nsym_max=1, nspin=2, nmag=2)


def _gpu(s, non_loc=False):
    ks = list(range(s.nk_bz))
    with LelphGPU(s, "fp64", route="real") as ctx:
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        return ctx.run([0] * len(ks), ks, non_loc=non_loc)


@pytest.mark.parametrize("bad", [np.nan, np.inf, 2.0 ** 40])
@pytest.mark.parametrize("spin", [0, 1])
def test_one_spin_does_not_touch_the_other(spin, bad):
    s = synth.make_system("case", LSDA)
    dv = 1024 * s.dVscf
    ref = O.compute_elphq(s, 0, dVscfq=dv[0], non_loc=False)
    if np.isfinite(bad):
        dv[:, :, spin] *= bad
        ref[:, :, spin] *= bad
    else:
        dv[0, 2, spin, 3, 4, 5] = bad
    g = _gpu(dataclasses.replace(s, dVscf=dv))
    other = 1 - spin
    assert np.abs(g[:, :, other] - ref[:, :, other]).max() < TOL * np.abs(ref[:, :, other]).max()
    if np.isfinite(bad):
        assert np.abs(g[:, :, spin] - ref[:, :, spin]).max() < TOL * np.abs(ref[:, :, spin]).max()
    else:
        hit = np.zeros(s.nmodes, bool)
        hit[2] = True
        assert not np.isfinite(g[:, hit, spin]).any()
        rest = np.abs(g[:, ~hit, spin] - ref[:, ~hit, spin]).max()
        assert rest < TOL * np.abs(ref[:, ~hit, spin]).max()


def test_scale_of_the_products_not_of_the_maxima():
    s = synth.make_system("case", dict(LSDA, kind="diamond", a=10.26, nspin=1, nspinor=2, nmag=4, ls=(0,)))
    w = [x.copy() for x in s.wfc]
    for x in w:
        x[:, :, 1] = 0
    s = dataclasses.replace(s, wfc=w)
    ref = O.compute_elphq(s, 0, non_loc=False)
    dv = s.dVscf.copy()
    dv[:, :, [1, 3]] *= 2.0 ** 60  # [up, down] and [down, down] multiply psi's second component
    g = _gpu(dataclasses.replace(s, dVscf=dv))
    assert np.abs(g - ref).max() < TOL * np.abs(ref).max()
