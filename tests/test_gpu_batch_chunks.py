"""Batched FIRE at one launch per op: the first chunks of 64 iterations are plain
launches, the later ones replay a graph.  Runs of many chunks, in one call or
several, with growing lists and across changes that a graph would hold, against
the persistent kernel: the same iterates bit for bit."""
import numpy as np
import pytest

from cudaring_b200 import synth
from cudaring_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _run(persistent, calls, change, cutoff=0.5):
    pks = [synth.make_packing([20] * n, [1.0] * n, 1.05, 0.7, seed=n, placement="uniform") for n in (6, 25, 14)]
    b = Batch.from_packings(pks, potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, ec=1.0)
    b.setLanes(1)
    b.setPersistent(persistent)
    b.setDisplacementCutoff(cutoff)
    b.initFIRE([0.2, 0.5, 1.1, 0.99, 1e-3, 1e-2, 0.2], 20, dt=np.full(3, 1e-3))
    out = []
    for k, its in enumerate(calls):
        if k == 1 and change == "costs":
            b.setEnergyCosts(2.0, 1.0, 0.02, 1.5)
        if k == 1 and change == "init":
            b.initFIRE([0.1, 0.5, 1.1, 0.99, 1e-3, 1e-2, 0.1], 10, dt=np.full(3, 5e-4))
        if k == 1 and change == "lists":
            b.setDisplacementCutoff(3.0)
        out += list(b.fireMinimize(1e-14, its)) + [b.getVertexPositions(), b.getVertexVelocities()]
    b.close()
    return out


@pytest.mark.parametrize("calls", [(255,), (256, 64), (320, 320), (64,) * 7, (70, 500), (1000,)])
@pytest.mark.parametrize("change", ["none", "costs", "init", "lists"])
def test_chunks(cuda_device, calls, change):
    for x, y in zip(_run(True, calls, change), _run(False, calls, change)):
        assert np.array_equal(x, y)
