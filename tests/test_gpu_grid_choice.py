"""Which product grid prepare and the allocation-free call take.

After a one-call stage, a q slot loaded and prepared is for batch runs: the
allocation-free call then works on the batch runs' grid and returns their bits.
Without such a preparation it works on the grid that is ready."""
import ctypes as C

import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import OUT_C128, LelphGPU, load_library

pytestmark = pytest.mark.gpu

CELL = dict(kind="l12", a=7.1, fft=(32, 32, 32), kgrid=(2, 2, 2), qpts=[(0.5, 0.5, 0.5)], nbnds=3, npw=800, ls=(0, 1))


def test_after_the_one_call_stage():
    torch = pytest.importorskip("torch")
    s = synth.make_system("case", CELL)
    n = s.nk_bz
    args = (s.qpts[0], s.eigVec[0], s.dVscf[0])
    qs, ks = (C.c_int * n)(*[0] * n), (C.c_int * n)(*range(n))
    L = load_library()

    def noalloc(ctx):
        out = torch.full((n, s.nmodes, s.nspin, s.nbnds, s.nbnds), float("nan"), dtype=torch.complex128, device="cuda")
        rc = L.lelph_gpu_run_device_noalloc(ctx.h, n, qs, ks, 1, 0, OUT_C128, C.c_void_p(out.data_ptr()))
        assert rc == 0, L.lelph_gpu_last_error(ctx.h).decode()
        return out.cpu().numpy()

    with LelphGPU(s, "mixed", route="real") as ctx:
        one = ctx.compute_elphq(*args)
        assert ctx.grid()["copies"] == 1
        assert np.array_equal(noalloc(ctx), one)        # nothing else is ready
        ctx.set_q(0, *args)
        ctx.prepare()
        assert ctx.grid()["copies"] > 1
        g = noalloc(ctx)
        batch = ctx.run([0] * n, list(range(n)))
        assert np.array_equal(g, batch)
        assert np.array_equal(ctx.compute_elphq(*args), one)
        ctx.prepare()                                   # the last run's grid
        assert ctx.grid()["copies"] == 1
