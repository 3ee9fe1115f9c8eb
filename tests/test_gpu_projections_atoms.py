"""KB projections where one block's 64 rows span many atoms.

With one projector an atom (four rows) a block holds up to 16 atoms, with three up to
six.  Every form of the projections against the oracle: FP64 to the FP64 bar of the
other tests (1e-10 of max|g|), the mixed form on and off the tensor cores to its norm
bar (2e-6)."""
import numpy as np
import pytest

import elph_oracle as O
from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

CELLS = {"8 atoms": dict(kind="rocksalt8", a=8.0), "16 atoms": dict(kind="sc16", a=10.0)}


@pytest.mark.parametrize("ls", [(0,), (1,)])
@pytest.mark.parametrize("cell", list(CELLS))
def test_many_atoms_a_block(cell, ls, monkeypatch):
    s = synth.make_system("case", dict(CELLS[cell], fft=(24, 24, 24), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=300,
                                       nbnds=4, ls=ls, nsym_max=1))
    ref = O.compute_elphq(s, 0)

    def run(prec):
        with LelphGPU(s, prec, route="real") as ctx:
            ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
            return ctx.run([0] * s.nk_bz, list(range(s.nk_bz)))

    assert np.abs(run("fp64") - ref).max() < 1e-10 * np.abs(ref).max()
    for tc in ("1", "0"):
        monkeypatch.setenv("LELPH_PROJ_TC", tc)
        assert np.linalg.norm(run("mixed") - ref) < 2e-6 * np.linalg.norm(ref)
