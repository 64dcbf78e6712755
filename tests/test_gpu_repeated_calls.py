"""Loops called a few steps at a time: the first chunks of a kind are plain
launches, from the eighth on they replay a captured graph, also over several
calls.  The same kernels in the same order: states equal those of direct
launches bit for bit, through the line, for calls of odd lengths (the position
buffers alternate) and across a change of a parameter that a graph holds."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, simControl, synth

pytestmark = pytest.mark.gpu


def _context(kind):
    pk = synth.make_packing([21] * 30 + [26] * 7, [1.0] * 30 + [1.6] * 7, 1.05, 0.42, seed=9, placement="rsa")
    d = DPM2D.from_packing(pk, potential="harmonic", interaction="vertexVertex", ea=10.0, el=5.0, eb=0.1, dt=2e-3)
    if kind == "rigid":
        d.setShapeType(simControl.shapeEnum.rigid)
    if kind == "lanes":
        d.setLanes(4)
    d.setSeed(6)
    d.calcNeighborList(d.setDisplacementCutoff(0.1, 2 * pk.rad.mean()))
    if kind == "rigid":
        d.calcParticlePositions()
        d.calcRigidForceEnergy()
        d.initRigidLangevin(1e-2, 1.0, readState=False)
        return d, d.rigidLangevinLoop
    d.calcForceEnergy()
    if kind == "rescale":
        d.initNVERescale(1e-2)
        return d, d.NVERescaleLoop
    d.initNVE(1e-2, readState=False)
    return d, d.NVELoop


@pytest.mark.parametrize("kind", ["rigid", "lanes", "rescale"])
@pytest.mark.parametrize("steps", [1, 5, 128, 130])
def test_states(cuda_device, kind, steps):
    out = []
    for graphs in (True, False):
        d, loop = _context(kind)
        d.setUseGraphs(graphs)
        states = []
        for call in range(20):
            if call == 17:
                d.setTimeStep(1e-3)
            loop(steps)
            if call in (6, 7, 8, 16, 17, 19):
                states += [d.getVertexPositions(), d.getVertexVelocities()]
        out.append((d.getUpdateCount(), states))
        d.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
