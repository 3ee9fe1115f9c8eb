"""Error of the mixed form's G-space route on its two product grids.

The batch runs' grid has about half the points, so its FP32 transforms average less
rounding away; the order of the GEMM's split products and windows transformed in FP64
make up for it.  Against the FP64 form, the batch run of a 16-atom cell is no further off than the one-call stage
on the plain grid."""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,npw", [(72, 4000), (130, 9000)])
def test_batch_grid_is_no_less_accurate(nb, npw):
    s = synth.make_system("case", dict(kind="sc16", a=10.0, fft=(90, 90, 90), kgrid=(2, 1, 1), qpts=[(0.5, 0, 0)], npw=npw,
                                       nbnds=nb, ls=(0, 1), nsym_max=1))
    args = (s.qpts[0], s.eigVec[0], s.dVscf[0])

    def err(g):
        return np.linalg.norm(g - ref) / np.linalg.norm(ref)

    with LelphGPU(s, "fp64", route="gspace") as ctx:
        ref = ctx.compute_elphq(*args, non_loc=False)
    with LelphGPU(s, "mixed", route="gspace", gs_gemm="tensor") as ctx:
        plain = err(ctx.compute_elphq(*args, non_loc=False))
        ctx.set_q(0, *args)
        batch = err(ctx.run([0] * s.nk_bz, list(range(s.nk_bz)), non_loc=False))
        assert ctx.grid()["copies"] > 1
    assert batch <= plain
