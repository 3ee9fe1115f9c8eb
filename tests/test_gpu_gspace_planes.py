"""Plane passes of the G-space route on every compile-time plane size.

The mixed form against the FP64 one on the same route, for spheres whose
interleaved grid has planes of 24 to 64 points a side (an odd one among them),
with a number of modes that is no multiple of a CTA's eight, few bands, an
umklapp and ragged spheres.  The bar is the one of the other mixed tests (norm
2e-6 of FP64): TF32-split GEMM and FP32 transforms.
"""
import numpy as np
import pytest

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import OUT_C64, LelphGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npw, box, nbnds", [
    ((700, 900), 48, 3), (1500, 48, 3), ((4000, 4500), 72, 3), (5000, 72, 3), (6500, 96, 3), (7600, 96, 3),
    (9000, 96, 3), ((11500, 12000), 96, 3), (13500, 108, 3), (24000, 128, 3), (32000, 144, 3),
    (2500, 48, 260)])  # enough bands for 16 modes a CTA
def test_planes_against_fp64(npw, box, nbnds):
    s = synth.make_system("planes", dict(kind="l12", a=10.0, fft=(box,) * 3, kgrid=(2, 2, 2),
                                         qpts=[(0.5, 0.5, 0)], nbnds=nbnds, npw=npw, ls=(0,)))
    got = {}
    for prec in ("fp64", "mixed"):
        with LelphGPU(s, prec, route="gspace") as ctx:
            ctx.set_q(0, s.qpts[0], s.eigVec[0], s.dVscf[0])
            got[prec] = ctx.run(np.zeros(2, int), np.array([0, s.nk_bz - 1]), out=OUT_C64 if prec == "mixed" else 0)
    d = np.linalg.norm(got["mixed"] - got["fp64"]) / np.linalg.norm(got["fp64"])
    assert d < 2e-6
