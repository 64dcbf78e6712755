"""A Hessian solve whose rows find no device memory runs one launch per op, with
scratch of its own, and gives the iterates of a context that had the memory."""
import numpy as np
import pytest
import torch

from cudaring_b200 import DPM2D, synth

from test_gpu_cg_steps import _angles

pytestmark = pytest.mark.gpu


def test_no_memory_for_the_rows(cuda_device):
    # every pair of 4,096 vertices listed: rows of 28 bytes at a capacity of
    # 4,096 and more, 470 MB at least
    pk = synth.make_packing([64] * 64, [1.0] * 64, 1.05, 0.4, seed=2, jitter=0.01, placement="rsa")
    contexts = []
    for _ in range(2):
        d = DPM2D.from_packing(pk, potential="harmonic", ea=1.0, el=1.0, eb=0.5)
        d.setRestAngles(_angles(pk))
        d.calcNeighborList(d.setDisplacementCutoff(1.0e3, 2 * pk.rad.mean()))
        contexts.append(d)
    full, short = contexts
    b = full.hvp(np.random.default_rng(1).normal(size=2 * full.numVertices))
    assert np.array_equal(b, short.hvp(np.random.default_rng(1).normal(size=2 * short.numVertices)))
    before = full.getLaunchCount()
    out = [full.hessianSolve(b, tol=1e-14, maxIter=5)]
    assert full.getLaunchCount() - before < 10
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - (384 << 20), dtype=torch.uint8, device=cuda_device)
    for _ in range(2):
        before = short.getLaunchCount()
        out.append(short.hessianSolve(b, tol=1e-14, maxIter=5))
        assert short.getLaunchCount() - before > 100  # a chunk of per-op iterations
    del held
    torch.cuda.empty_cache()
    (x, it, rr) = out[0]
    for y, jt, ss in out[1:]:
        assert it == jt
        # the rounding of a product (1e-15) through five iterations
        assert np.abs(x - y).max() <= 1e-9 * np.abs(x).max()
        assert rr == pytest.approx(ss, rel=1e-8)
    assert np.array_equal(out[1][0], out[2][0])
    full.close()
    short.close()
