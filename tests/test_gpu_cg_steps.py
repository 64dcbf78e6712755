"""Conjugate-gradient iterations in one launch against the captured per-op
iterations (which the solve falls back to when a grid barrier gives up): the
same iterates to rounding at small iteration counts, for both preconditioners,
the potentials, and the ring sizes at the edges of its CTAs; and Hessian
products written to arrays that overlap the input or are not 16-byte aligned."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth
from cudaring_b200._lib import CudaRingError

pytestmark = pytest.mark.gpu


def _context(nv=33, n=12, potential="harmonic", phi=0.4):
    pk = synth.make_packing([nv] * n, [1.0] * n, 1.05, phi, seed=2, jitter=0.01, placement="rsa")
    d = DPM2D.from_packing(pk, potential=potential, ea=1.0, el=1.0, eb=0.5, l1=0.05, l2=0.2)
    d.setRestAngles(_angles(pk))
    d.calcNeighborList(d.setDisplacementCutoff(0.5, 2 * pk.rad.mean()))
    return d


def _angles(pk):
    # the turning angles of the packing itself: no bending stress, a stable state
    x = pk.pos.reshape(-1, 2)
    first, out, a = 0, [], None
    for nv in pk.nv_list:
        r = x[first:first + nv]
        ns = np.roll(r, -1, axis=0) - r
        ps = np.roll(ns, 1, axis=0)
        a = np.arctan2(ns[:, 0] * ps[:, 1] - ns[:, 1] * ps[:, 0], (ns * ps).sum(1))
        out.append(a)
        first += nv
    return np.concatenate(out)


@pytest.mark.parametrize("iterations", [1, 2, 12])
@pytest.mark.parametrize("precond", ["block_jacobi", "none"])
@pytest.mark.parametrize("nv,n", [(33, 12), (64, 5), (65, 4), (128, 3), (4, 30)])
def test_iterates(cuda_device, iterations, precond, nv, n):
    phi = 0.4 if nv > 10 else 0.1
    b = None
    out = []
    for spin in (0, -1):
        d = _context(nv, n, phi=phi)
        d.setCGPreconditioner(precond)
        d.setSpinLimit(spin)
        if b is None:  # in the range of the Hessian: products of vectors
            b = d.hvp(np.random.default_rng(1).normal(size=2 * d.numVertices))
        try:
            out.append(d.hessianSolve(b, tol=1e-14, maxIter=iterations))
        except CudaRingError as e:  # rings of four are not stable: a direction of negative curvature
            out.append(e.code)
        d.close()
    if isinstance(out[0], int) or isinstance(out[1], int):
        assert out[0] == out[1]
        return
    (x, it, rr), (y, jt, ss) = out
    assert it == jt
    # both carry the rounding of a product (1e-15) through at most 12 iterations
    assert np.abs(x - y).max() <= 1e-9 * np.abs(y).max()
    assert rr == pytest.approx(ss, rel=1e-8)


def test_product_in_place_and_unaligned(cuda_device):
    import torch

    d = _context()
    n = 2 * d.numVertices
    v = torch.randn(n + 3, dtype=torch.float64, device=cuda_device)
    ref = torch.from_numpy(d.hvp(v[:n].cpu().numpy())).to(cuda_device)
    out = torch.zeros(n + 1, dtype=torch.float64, device=cuda_device)
    torch.cuda.synchronize()
    d.hvpDevice(v.data_ptr(), out[1:].data_ptr())
    assert torch.equal(out[1:], ref) and out[0] == 0
    w = v[:n].clone()
    torch.cuda.synchronize()
    d.hvpDevice(w.data_ptr(), w.data_ptr())
    assert torch.equal(w, ref)
    d.close()
