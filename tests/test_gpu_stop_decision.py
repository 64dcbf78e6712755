"""Sequences whose launches end often: every step of a hot, dilute run moves some
vertex past the displacement cutoff, so each launch of the multi-step kernels
stops after a step or two, at even and odd barriers, with CTAs of little work
running ahead of the others.  No barrier may give up (the context would go back
to one launch per op), and states equal those of one launch per op."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth

pytestmark = pytest.mark.gpu


def _context(potential, interaction, lanes, multi, cutoff, dt):
    # rings of uneven sizes and numbers of pairs: uneven work per CTA
    nv = [8] * 200 + [40] * 30 + [24] * 60
    pk = synth.make_packing(nv, [1.0] * 200 + [6.0] * 30 + [3.0] * 60, 1.05, 0.3, seed=9, placement="rsa")
    d = DPM2D.from_packing(pk, potential=potential, interaction=interaction, ea=10.0, el=5.0, eb=0.1, dt=dt)
    d.setLanes(lanes)
    d.setMultistep(multi)
    d.setSeed(7)
    d.calcNeighborList(d.setDisplacementCutoff(cutoff, 2 * pk.rad.mean()))
    d.calcForceEnergy()
    return d


@pytest.mark.parametrize("interaction", ["vertexVertex", "vertexSmooth"])
@pytest.mark.parametrize("lanes", [1, 2])
def test_rebuilds_every_few_steps(cuda_device, interaction, lanes):
    out = []
    for multi in (True, False):
        d = _context("harmonic", interaction, lanes, multi, cutoff=0.02, dt=2e-3)
        d.initNVE(1.0, readState=False)
        d.NVELoop(400)
        assert not d.getDegraded()
        out.append((d.getUpdateCount(), d.getVertexPositions(), d.getVertexVelocities()))
        d.close()
    assert out[0][0] == out[1][0] and out[0][0] > 100
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("interaction", ["vertexVertex", "vertexSmooth"])
def test_fire_rebuilds(cuda_device, interaction):
    d = _context("harmonic", interaction, 2, True, cutoff=0.02, dt=2e-3)
    d.initFIRE([0.2, 0.5, 1.1, 0.99, 1e-2, 1e-1, 0.2], 20, 0, d.numVertices)
    d.vertexFIRELoop(300)
    assert not d.getDegraded()
    assert d.getUpdateCount() > 5
    d.close()
