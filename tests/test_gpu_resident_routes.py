"""Which sizes run many steps in a launch.  The grid of such a launch must be on
the GPU at once: a B200 (148 SMs) holds 3, 4 or 5 CTAs an SM of the kernels here,
with the staged lists or, one size further, without.  Rings of 100 vertices with
one lane per vertex make a tile each.  FP64 states equal those of one launch per
op bit for bit, mixed ones to the rounding that the multi-step tests state."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth
from cudaring_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _run(n, interaction, multi, precision, steps=70):
    pk = synth.make_packing([100] * n, [1.0] * n, 1.05, 0.45, seed=3, placement="rsa")
    d = DPM2D.from_packing(pk, potential="harmonic", interaction=interaction, ea=10.0, el=5.0, eb=0.1, dt=2e-3)
    d.setLanes(1)
    d.setMultistep(multi)
    d.setPrecision(precision)
    d.setSeed(1)
    d.calcNeighborList(d.setDisplacementCutoff(0.1, 2 * pk.rad.mean()))
    d.calcForceEnergy()
    d.initNVE(1e-2, readState=False)
    before = d.getLaunchCount()
    d.NVELoop(steps)
    out = d.getVertexPositions(), d.getVertexVelocities(), d.getUpdateCount(), d.getLaunchCount() - before
    assert not d.getDegraded()
    d.close()
    return out


# staged, the last staged and the first unstaged size, the last unstaged one, one launch per op
@pytest.mark.parametrize("interaction,n,many", [
    ("vertexVertex", 300, True), ("vertexVertex", 592, True), ("vertexVertex", 593, True),
    ("vertexVertex", 740, True), ("vertexVertex", 741, False),
    ("vertexSmooth", 300, True), ("vertexSmooth", 444, True), ("vertexSmooth", 445, True),
    ("vertexSmooth", 592, True), ("vertexSmooth", 593, False)])
def test_steps(cuda_device, interaction, n, many):
    a, b = _run(n, interaction, True, "fp64"), _run(n, interaction, False, "fp64")
    assert b[3] >= 2 * 70  # a step and its build
    # a launch of up to 64 steps and its build, one pair more per rebuild, and what was sized in vain
    assert (a[3] < 2 * 70) == many
    assert a[2] == b[2] and a[2] > 1
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("interaction,n", [("vertexVertex", 600), ("vertexSmooth", 450)])
def test_steps_mixed_unstaged(cuda_device, interaction, n):
    a, b = _run(n, interaction, True, "mixed", 10), _run(n, interaction, False, "mixed", 10)
    assert a[2] == b[2]
    assert np.max(np.abs(a[0] - b[0])) < 1e-9
    assert np.max(np.abs(a[1] - b[1])) < 1e-7


@pytest.mark.parametrize("interaction,lanes,n,many", [
    ("vertexVertex", 1, 592, True), ("vertexVertex", 1, 593, False), ("vertexVertex", 2, 444, True),
    ("vertexSmooth", 1, 296, True), ("vertexSmooth", 1, 297, True), ("vertexSmooth", 1, 592, True),
    ("vertexSmooth", 1, 593, False), ("vertexSmooth", 2, 296, True), ("vertexSmooth", 2, 297, True),
    ("vertexSmooth", 2, 444, True), ("vertexSmooth", 2, 445, False)])
def test_batch_fire(cuda_device, interaction, lanes, n, many):
    nv = 100 if lanes == 1 else 80
    rings = [n // 8 + (1 if s < n % 8 else 0) for s in range(8)]
    pks = [synth.make_packing([nv] * m, [1.0] * m, 1.05, 0.4, seed=s, placement="rsa") for s, m in enumerate(rings)]
    out = []
    for persistent in (True, False):
        b = Batch.from_packings(pks, potential="harmonic", interaction=interaction, ea=10.0, el=5.0, eb=0.1, ec=1.0)
        b.setTileShape(lanes, 128 if lanes == 1 else 192)
        b.setPersistent(persistent)
        b.setDisplacementCutoff(0.5)
        b.initFIRE([0.2, 0.5, 1.1, 0.99, 1e-3, 1e-2, 0.2], 20, dt=np.full(8, 1e-3))
        before = b.getLaunchCount()
        its, fmax = b.fireMinimize(1e-14, 100)
        out.append((its, fmax, b.getVertexPositions(), b.getVertexVelocities(), b.getLaunchCount() - before))
        b.close()
    p, q = out
    assert q[4] >= 2 * 100 and (p[4] < 100) == many
    for x, y in zip(p[:4], q[:4]):
        assert np.array_equal(x, y)
