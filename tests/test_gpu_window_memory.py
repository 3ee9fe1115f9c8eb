"""The plain form transforms its dV windows in place: loading a q and running it takes no
scratch of the windows' size besides them."""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU

pytestmark = pytest.mark.gpu


def test_no_second_set_of_windows():
    s = synth.make_system("case", dict(kind="l12", a=7.1, fft=(32, 32, 32), kgrid=(2, 2, 2), qpts=[(0, 0, 0)],
                                       nbnds=1, npw=800, ls=(0, 1)))
    with LelphGPU(s, "fp64", route="real") as ctx:
        ctx.prepare()
        before = ctx.stats()["device_bytes"]
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        ctx.run([0], [0])
        grown = ctx.stats()["device_bytes"] - before
        window = 16 * s.nmodes * ctx.grid()["points"]
    box = 16 * s.nmodes * int(np.prod(s.fft_dims))
    # dV and its transform on the reference box, one window (q = 0 has no umklapp) and its exponents (1/32);
    # the rest (pairs, sums, results of one pair of one band) is below a megabyte
    assert grown < 2 * box + window * 33 / 32 + (1 << 20)
