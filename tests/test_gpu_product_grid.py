"""The product grid of batch runs: interleaved copies of a smaller grid.

For cells whose best grid has one to four copies, with shifts along one axis
and along several: the grid a context reports is exact for its spheres (no two
differences G' - G1 of a pair fall into one class of the grid's reciprocal
lattice, by enumeration on the host), and the matrix elements equal those on
the plain product grid -- FP64 to the FP64 bar of the other tests (1e-10 of
max|g|) on both routes, the mixed form to its bar against FP64 (norm 2e-6).
The one-call stage of the mixed form stays on the plain grid: its results are
the bits of a context that is held on it.
"""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import OUT_C64, LelphGPU

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "diamond": dict(kind="diamond", a=10.26, fft=(24, 24, 24), kgrid=(2, 2, 2), qpts=[(0.5, 0, 0), (0.5, 0.5, 0)],
                    nbnds=5, npw=400, ls=(0, 1)),
    "cubic": dict(kind="l12", a=7.1, fft=(32, 32, 32), kgrid=(2, 2, 2), qpts=[(0.5, 0.5, 0.5)], nbnds=3, npw=800,
                  ls=(0, 1)),
    "hexagonal, ragged spheres": dict(kind="hex2d", a=6.0, fft=(36, 36, 216), kgrid=(3, 3, 1),
                                      qpts=[(1 / 3, 1 / 3, 0)], nbnds=3, npw=(1800, 2600), ls=(0, 1)),
    "spinors, nmag 4": dict(kind="rocksalt8", a=8.0, fft=(32, 32, 32), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], nbnds=3,
                            npw=700, ls=(0, 1, 2), nspinor=2, nmag=4, soc=True, nsym_max=1),
    "collinear spins, time reversal": dict(kind="zincblende", a=10.2, fft=(30, 30, 32), kgrid=(2, 2, 2),
                                           qpts=[(0.5, 0, 0.5)], nbnds=3, npw=(350, 700), ls=(0, 1), nspin=2, nmag=2,
                                           timerev=True),
    # a reference box near the spheres' extent: most of its residues are needed
    "tight box": dict(kind="diamond", a=10.26, fft=(18, 20, 24), kgrid=(2, 2, 2), qpts=[(0, 0.5, 0)], nbnds=2,
                      npw=300, ls=(0,)),
}


def _run(s, prec, route, out=0):
    with LelphGPU(s, prec, route=route) as ctx:
        for iq in range(len(s.qpts)):
            ctx.set_q(iq, s.qpts[iq], s.eigVec[iq], s.dVscf[iq])
        qs = np.repeat(np.arange(len(s.qpts)), s.nk_bz)
        ks = np.tile(np.arange(s.nk_bz), len(s.qpts))
        g = ctx.run(qs, ks, out=out)
        return g, ctx.grid()


def _exact(s, grid):
    """No two differences of a pair's spheres in one class of the grid's reciprocal lattice."""
    n, p, a = np.array(grid["n"]), grid["copies"], np.array(grid["shift"])
    W = [np.rint(s.alat.T @ R @ np.linalg.inv(s.alat).T).astype(int) for R in s.sym_R]
    sph = [s.miller[ik] @ W[isym].T for ik, isym in s.kmap[:2]]
    for A in sph:
        for B in sph:
            # the extreme points of the spheres carry the extreme differences
            d = (A[:, None, :] - B[None, :, :]).reshape(-1, 3)
            d = np.unique(d, axis=0)
            m, r = np.floor_divide(d, n), np.mod(d, n)
            cls = np.mod(m @ a, p)
            key = ((r[:, 0] * n[1] + r[:, 1]) * n[2] + r[:, 2]) * p + cls
            assert len(np.unique(key)) == len(key)


@pytest.mark.parametrize("route", ["real", "gspace"])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_smaller_grid_equals_the_plain_one(name, route, monkeypatch):
    s = synth.make_system("case", SYSTEMS[name])
    g64, grid = _run(s, "fp64", route)
    _exact(s, grid)
    gm, gridm = _run(s, "mixed", route, out=OUT_C64)
    _exact(s, gridm)
    monkeypatch.setenv("LELPH_PLAIN_GRID", "1")
    ref, plain = _run(s, "fp64", route)
    assert plain["copies"] == 1 and grid["points"] <= plain["points"]
    assert np.abs(g64 - ref).max() / np.abs(ref).max() < 1e-10
    assert np.linalg.norm((gm - ref).ravel()) / np.linalg.norm(ref.ravel()) < 2e-6


def test_cases_reach_every_copy_count():
    copies = set()
    for o in SYSTEMS.values():
        s = synth.make_system("case", o)
        for prec, route in (("fp64", "real"), ("mixed", "real"), ("fp64", "gspace")):
            with LelphGPU(s, prec, route=route) as ctx:
                copies.add(ctx.grid()["copies"])
    assert {2, 3, 4} <= copies, copies


@pytest.mark.parametrize("route", ["real", "gspace"])
def test_one_call_stage_keeps_the_plain_grid(route, monkeypatch):
    s = synth.make_system("case", SYSTEMS["cubic"])
    qs, ks = np.zeros(s.nk_bz, int), np.arange(s.nk_bz)
    args = (s.qpts[0], s.eigVec[0], s.dVscf[0])
    with LelphGPU(s, "mixed", route=route) as ctx:
        ctx.prepare()
        g = ctx.compute_elphq(*args)
        assert ctx.grid()["copies"] == 1
        batch = ctx.run(qs, ks)          # the batch grid, prepared on its first use
        assert ctx.grid()["copies"] > 1
        again = ctx.compute_elphq(*args)
        ctx.set_wavefunctions([w[:, ::-1].copy() for w in s.wfc])
        ctx.set_wavefunctions(s.wfc)     # both grids are out of date
        batch2 = ctx.run(qs, ks)
        third = ctx.compute_elphq(*args)
    monkeypatch.setenv("LELPH_PLAIN_GRID", "1")
    with LelphGPU(s, "mixed", route=route) as ctx:
        ref = ctx.compute_elphq(*args)
    for x in (g, again, third):
        assert np.array_equal(x, ref)
    assert np.array_equal(batch, batch2)
    assert np.linalg.norm((batch - ref).ravel()) / np.linalg.norm(ref.ravel()) < 2e-6
