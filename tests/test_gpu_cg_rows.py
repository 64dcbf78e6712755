"""The rows that the many-iterations solve forms for itself, for rings that lie
across warps and have few or no pairs, so that a warp that is done with its rows
could run ahead of one that still reads its ring's area.  Against the captured
per-op iterations, whose products come from the derivative kernel; both carry
the rounding of a product (1e-15) through a few iterations, and the first
iterates are the most sensitive to a wrong row.  (A solve to convergence says
nothing here: rings without pairs translate and rotate freely.)"""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth
from cudaring_b200._lib import CudaRingError

from test_gpu_cg_steps import _angles

pytestmark = pytest.mark.gpu


# one ring per CTA over two, three or four warps; rings that start inside a warp
@pytest.mark.parametrize("nv_list", [[33] * 4, [64] * 3, [65] * 3, [96] * 3, [97] * 3, [128] * 2,
                                     [20] * 30, [45, 18] * 6, [31, 33, 40, 24] * 3])
@pytest.mark.parametrize("phi", [0.05, 0.4])
def test_rows(cuda_device, nv_list, phi):
    pk = synth.make_packing(nv_list, [1.0] * len(nv_list), 1.05, phi, seed=5, jitter=0.01, placement="uniform")
    contexts = []
    for spin in (0, -1):  # a negative limit: the barrier gives up, the captured iterations run
        d = DPM2D.from_packing(pk, potential="harmonic", ea=1.0, el=1.0, eb=0.5)
        d.setRestAngles(_angles(pk))
        d.calcNeighborList(d.setDisplacementCutoff(0.5, 2 * pk.rad.mean()))
        d.setSpinLimit(spin)
        contexts.append(d)
    b = contexts[0].hvp(np.random.default_rng(3).normal(size=2 * contexts[0].numVertices))
    for iterations in (1, 2, 3, 1, 2, 3):
        out = []
        for d in contexts:
            try:
                out.append(d.hessianSolve(b, tol=1e-14, maxIter=iterations))
            except CudaRingError as e:  # overlapping rings need not be stable
                out.append(e.code)
        if isinstance(out[0], int) or isinstance(out[1], int):
            assert out[0] == out[1]
            continue
        (x, it, rr), (y, jt, ss) = out
        assert it == jt
        assert np.abs(x - y).max() <= 1e-9 * np.abs(y).max()
        assert rr == pytest.approx(ss, rel=1e-8)
    for d in contexts:
        d.close()
