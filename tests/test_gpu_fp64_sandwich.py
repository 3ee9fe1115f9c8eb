"""The FP64 sandwich on the tensor cores (63-bit fixed point, base-512 digits).

Edges of its tiles -- 128 (mode, band) rows, 32 bands of k+q, 32 grid points a
stage -- in the band count, spin and spinor layouts, and inputs whose magnitudes
spread widely, against the oracle at the FP64 bar of the other tests (1e-10 of
max|g|); bands of zeros; a NaN and an infinity reach exactly the matrix
elements they enter, as in FP64 arithmetic."""
import dataclasses

import numpy as np
import pytest

import elph_oracle as O
from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

TOL = 1e-10
BASE = dict(kind="diamond", a=10.26, fft=(16, 18, 20), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=150, ls=(0, 1),
            nsym_max=1)


def _gpu(s, non_loc=True):
    ks = list(range(s.nk_bz))
    with LelphGPU(s, "fp64", route="real") as ctx:
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        return ctx.run([0] * len(ks), ks, non_loc=non_loc)


def _close(s):
    ref = O.compute_elphq(s, 0)
    assert np.abs(_gpu(s) - ref).max() / np.abs(ref).max() < TOL


@pytest.mark.parametrize("nb", [1, 7, 8, 9, 21, 22, 31, 32, 33, 64, 67])
def test_band_counts(nb):
    _close(synth.make_system("case", dict(BASE, nbnds=nb)))


@pytest.mark.parametrize("ov", [dict(nspin=2, nmag=2), dict(nspinor=2, nmag=4, soc=True), dict(nspinor=2, nmag=1)])
def test_spin_layouts(ov):
    _close(synth.make_system("case", dict(BASE, nbnds=5, **ov)))


def test_wide_magnitudes():
    """dV with a peak 10^4 above the rest, modes and bands scaled by up to 10^+-30: the scales are
    per (mode, band) row, so each element keeps FP64's accuracy against its own row."""
    s = synth.make_system("case", dict(BASE, nbnds=4))
    dv = s.dVscf.copy()
    dv[0][:, :, 3, 4, 5] *= 1e4
    f = 10.0 ** np.array([0, 30, -30, 5, -7, 12])
    w = [x * (10.0 ** np.array([0, 20, -20, 3]))[None, :, None, None] for x in s.wfc]
    t = dataclasses.replace(s, wfc=w, dVscf=dv * f[None, :, None, None, None, None])
    ref, g = O.compute_elphq(t, 0, non_loc=False), _gpu(t, non_loc=False)
    rowmax = np.abs(ref).max(axis=(0, 2), keepdims=True)  # per (mode, band of k, band of k+q) over k
    assert (np.abs(g - ref) <= 1e-9 * rowmax).all()


def test_zero_band_and_mode():
    s = synth.make_system("case", dict(BASE, nbnds=4))
    w = [x.copy() for x in s.wfc]
    for x in w:
        x[:, 2] = 0
    dv = s.dVscf.copy()
    dv[0][1] = 0
    t = dataclasses.replace(s, wfc=w, dVscf=dv)
    g = _gpu(t, non_loc=False)
    assert np.isfinite(g).all() and (g[:, :, :, 2] == 0).all() and (g[:, :, :, :, 2] == 0).all() and (g[:, 1] == 0).all()
    _close(t)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_not_finite(bad):
    s = synth.make_system("case", dict(BASE, nbnds=4))
    w = [x.copy() for x in s.wfc]
    w[0][0, 1, 0, 3] = bad
    t = dataclasses.replace(s, wfc=w)
    g = _gpu(t, non_loc=False)
    kq = [O.get_kplusq_idxs(s.kbz_crys, s.qpts[0])[k] for k in range(s.nk_bz)]
    for k in range(s.nk_bz):
        hit = np.zeros(g.shape[1:], bool)
        if s.kmap[k][0] == 0:
            hit[:, :, 1, :] = True
        if s.kmap[kq[k]][0] == 0:
            hit[:, :, :, 1] = True
        assert np.array_equal(np.isfinite(g[k]), ~hit)
