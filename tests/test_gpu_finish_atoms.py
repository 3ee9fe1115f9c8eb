"""The finish for projection sets that overflow shared memory (one atom's
projections at a time): spinors with d projectors and 24 modes, more than 8
atoms on the real-space route, band counts around its 16-band tiles; the mixed
form (pairs of floats, K-chunk partials) and the FP64 form against the oracle
on a few pairs.  Tolerances: the FP64 bar (1e-10 of max|g|) and the mixed
form's norm bar (2e-6)."""
import numpy as np
import pytest

import elph_oracle as O
from letzelphc_gb300 import synth
from letzelphc_gb300.elph import OUT_C64, LelphGPU

pytestmark = pytest.mark.gpu

SOC = dict(kind="rocksalt8", a=8.0, fft=(24, 24, 24), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=300, ls=(0, 1, 2),
           nspinor=2, nmag=4, soc=True, nsym_max=1)
SC16 = dict(kind="sc16", a=10.0, fft=(24, 24, 24), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=300, ls=(0, 1, 2, 3),
            nsym_max=1)


@pytest.mark.parametrize("nonlocal_", [True, False])
@pytest.mark.parametrize("base,nb", [(SOC, 15), (SOC, 17), (SOC, 33), (SC16, 9)])
def test_finish_matches_oracle(base, nb, nonlocal_):
    s = synth.make_system("case", dict(base, nbnds=nb))
    ref = O.compute_elphq(s, 0, non_loc=nonlocal_)
    ks = list(range(s.nk_bz))
    for prec, out, tol in (("fp64", 0, None), ("mixed", 0, 2e-6), ("mixed", OUT_C64, 2e-6)):
        with LelphGPU(s, prec, route="real") as ctx:
            ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
            g = ctx.run([0] * len(ks), ks, non_loc=nonlocal_, out=out)
        if tol is None:
            assert np.abs(g - ref).max() / np.abs(ref).max() < 1e-10
        else:
            assert np.linalg.norm((g - ref).ravel()) / np.linalg.norm(ref.ravel()) < tol
