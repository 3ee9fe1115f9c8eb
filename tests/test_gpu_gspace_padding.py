"""G-space route: positions past a sphere in the GEMM operand.

A q with a NaN in its dV leaves NaN in the operand buffer; spheres of other sizes
then use other positions of it.  The next, finite q gives the bits of a context
that never saw the NaN, in every form of the GEMM."""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu

RAGGED = dict(kind="zincblende", a=10.2, fft=(20, 20, 20), kgrid=(2, 2, 2), qpts=[(0.5, 0, 0)], npw=(90, 160), nbnds=5,
              ls=(0,), nsym_max=1)


@pytest.mark.parametrize("prec,gemm", [("fp64", "auto"), ("mixed", "tensor"), ("mixed", "simt")])
@pytest.mark.parametrize("spin", [{}, dict(nspinor=2, nmag=4, soc=True)])
def test_a_nan_does_not_stay(prec, gemm, spin):
    s = synth.make_system("case", dict(RAGGED, **spin))
    ks = list(range(s.nk_bz))

    def run(ctx, dv):
        ctx.set_q(0, s.qpts[0], s.eigVec[0], dv)
        return ctx.run([0] * len(ks), ks, non_loc=False)

    with LelphGPU(s, prec, route="gspace", gs_gemm=gemm) as ctx:
        ref = run(ctx, s.dVscf[0])
    with LelphGPU(s, prec, route="gspace", gs_gemm=gemm) as ctx:
        assert not np.isfinite(run(ctx, np.full_like(s.dVscf[0], np.nan))).any()
        g = run(ctx, s.dVscf[0])
    assert np.array_equal(g, ref)
