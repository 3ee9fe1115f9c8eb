"""A wait of the FP64 sandwich that runs out, without a GPU fault.

With a limit of 1 ns the wait for a stage's MMAs (about a microsecond for 32 bands)
runs out: the kernel lets them finish, releases its tensor memory and reports
LELPH_GPU_ERR_TIMEOUT; with the default limit the context then gives the bits of
before."""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphError, LelphGPU

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = -4


def test_short_wait_limit_reports_timeout_and_context_recovers():
    s = synth.make_system("c0", {"kgrid": (4, 4, 4), "qpts": [(0.5, 0, 0)], "nbnds": 32})
    ks = list(range(s.nk_bz))
    with LelphGPU(s, "fp64", route="real") as ctx:
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        g0 = ctx.run([0] * len(ks), ks)
        ctx.set_wait_limit(1)
        with pytest.raises(LelphError) as e:
            ctx.run([0] * len(ks), ks)
        assert e.value.status == ERR_TIMEOUT
        ctx.set_wait_limit(0)
        g1 = ctx.run([0] * len(ks), ks)
    assert np.isfinite(g1).all()
    assert np.array_equal(g0, g1)
