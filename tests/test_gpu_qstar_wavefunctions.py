"""q-star expansion after a change of the wavefunctions: the Dmats left on the device
belong to the old ones, so the expansion equals that of a context made with the new
ones (1e-10 of max|g|, the FP64 bar of the other tests)."""
import dataclasses

import numpy as np
import pytest

from golden_util import load_star
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu


def test_resident_dmats_of_old_wavefunctions_are_not_used():
    z, s, kmq = load_star("star_c0")
    n = int(z["nqstar"][0])
    args = (s.qpts[0], s.eigVec[0], s.dVscf[0], z["qsym"][:n])
    new = [np.ascontiguousarray(w[:, ::-1]) for w in s.wfc]
    with LelphGPU(dataclasses.replace(s, wfc=new), "fp64") as ctx:
        ref = ctx.compute_elphq_star(*args)
    with LelphGPU(s, "fp64") as ctx:
        ctx.dmats(s.sym_R, s.sym_tau, s.sym_trev, host=False)
        ctx.compute_elphq_star(*args)
        ctx.set_wavefunctions(new)
        g = ctx.compute_elphq_star(*args)
    assert np.abs(g - ref).max() < 1e-10 * np.abs(ref).max()
