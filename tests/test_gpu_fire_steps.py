"""FIRE iterations in the multi-iteration kernel against one launch per op: the
same iterates to rounding over a few dozen iterations (both evaluate the same
expressions; separate compilations may fuse products differently), at
iteration counts inside, at and past a launch's budget, with rebuilds on the
way, and the same end at a tolerance met inside a launch and after a grid
barrier that gave up."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth

pytestmark = pytest.mark.gpu


def _context(interaction="vertexVertex", potential="harmonic", lanes=2, n=41, phi=0.8):
    pk = synth.make_packing([16] * (n // 2) + [22] * (n - n // 2), [1.0] * (n // 2) + [1.96] * (n - n // 2), 1.05, phi,
                            seed=11, placement="uniform")
    d = DPM2D.from_packing(pk, potential=potential, interaction=interaction, l1=0.05, l2=0.2)
    d.setLanes(lanes)
    d.calcNeighborList(d.setDisplacementCutoff(0.5, 2 * pk.rad.mean()))
    d.calcForceEnergy()
    d.initFIRE([0.2, 0.5, 1.1, 0.99, 2e-3, 2e-2, 0.2], 20, 0, d.numVertices)
    return d


def _close(a, b, tol):
    return np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("iterations", [1, 2, 63, 64, 65, 90])
@pytest.mark.parametrize("interaction", ["vertexVertex", "vertexSmooth"])
@pytest.mark.parametrize("lanes", [1, 2])
def test_iterates(cuda_device, iterations, interaction, lanes):
    out = []
    for multi in (True, False):
        d = _context(interaction, lanes=lanes)
        d.setMultistep(multi)
        d.vertexFIRELoop(iterations)
        out.append((d.getVertexPositions(), d.getVertexVelocities(), d.getVertexForces(), d.getFIREState(),
                    d.getUpdateCount(), d.getPotentialEnergy()))
        d.close()
    a, b = out
    assert a[4] == b[4]
    # rounding of one iteration (1e-16) grown over 90 steps of bounded forces
    assert _close(a[0], b[0], 1e-10) and _close(a[1], b[1], 1e-9) and _close(a[2], b[2], 1e-9)
    assert np.allclose(a[3], b[3], rtol=1e-12)
    assert a[5] == pytest.approx(b[5], rel=1e-10)


def test_tolerance_inside_a_launch(cuda_device):
    out = []
    for multi in (True, False):
        d = _context(phi=0.7)
        d.setMultistep(multi)
        it, fmax = d.minimizeFIRE(1e-2, 5000)
        assert fmax <= 1e-2 and 0 < it < 5000
        again, _ = d.minimizeFIRE(1e-2, 5000)
        assert again == 0  # converged: nothing to do
        out.append(it)
        d.close()
    assert out[0] == out[1]


def test_barrier_that_gives_up(cuda_device):
    ref = _context()
    ref.vertexFIRELoop(40)
    d = _context()
    d.setSpinLimit(-1)
    d.vertexFIRELoop(40)
    assert d.getDegraded()
    assert _close(d.getVertexPositions(), ref.getVertexPositions(), 1e-10)
    d.close()
    ref.close()
