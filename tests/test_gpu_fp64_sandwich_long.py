"""The FP64 sandwich over a product grid longer than its 64-bit sums hold.

One K chunk of 62,500 32-point stages (the allocation-free call always takes one
chunk), beyond the 32,768 stages after which the sums go to the output, against
the oracle and against run(), which splits the grid, at the FP64 bar of the other
tests (1e-10 of max|g|)."""
import ctypes as C

import numpy as np
import pytest

import elph_oracle as O
from letzelphc_gb300 import synth
from letzelphc_gb300.elph import OUT_C128, LelphGPU, load_library

pytestmark = pytest.mark.gpu


def test_one_chunk_of_two_million_points(monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("LELPH_FULL_BOX", "1")
    s = synth.make_system("case", dict(kind="diamond", a=10.26, fft=(128, 125, 125), kgrid=(1, 1, 1), qpts=[(0, 0, 0)],
                                       nbnds=2, npw=150, ls=(0,), nsym_max=1))
    ref = O.compute_elphq(s, 0, non_loc=False)
    L = load_library()
    with LelphGPU(s, "fp64", route="real") as ctx:
        assert ctx.grid()["points"] > 60000 * 32
        ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
        split = ctx.run([0], [0], non_loc=False)
        out = torch.full(ref.shape, float("nan"), dtype=torch.complex128, device="cuda")
        i = (C.c_int * 1)(0)
        rc = L.lelph_gpu_run_device_noalloc(ctx.h, 1, i, i, 0, 0, OUT_C128, C.c_void_p(out.data_ptr()))
        assert rc == 0, L.lelph_gpu_last_error(ctx.h).decode()
        g = out.cpu().numpy()
    for x in (split, g):
        assert np.abs(x - ref).max() < 1e-10 * np.abs(ref).max()
