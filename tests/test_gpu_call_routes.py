"""Routes that a call takes by its size: host copies of 8 MB and more through
pinned chunks, step sequences of one step and of few or many chunks, and the
batched list build over systems of few and many cells.  Copies are exact; the
step sequences run the same kernels in the same order, so FP64 states are
identical; the batch evaluates the lists of the single-system build with the
same arithmetic, so forces agree to FP64 rounding (1e-12 of the largest)."""
import numpy as np
import pytest
import torch

from cudaring_b200 import DPM2D, synth
from cudaring_b200.batch import Batch

from conftest import rel_inf

pytestmark = pytest.mark.gpu


# 16 bytes a vertex: one vertex under 8 MB, 8 MB, one over, and a last chunk of 48 bytes after 21
@pytest.mark.parametrize("nv", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1, 21 * (1 << 16) + 3])
@pytest.mark.parametrize("pinned", [False, True])
def test_large_copies(cuda_device, nv, pinned):
    d = DPM2D([32] * (nv // 32 - 1) + [32 + nv % 32])
    rng = np.random.default_rng(nv)
    x = torch.from_numpy(rng.standard_normal(2 * nv + 1))[1:]  # 8-byte aligned
    y = torch.zeros(2 * nv, dtype=torch.float64)
    if pinned:
        x, y = x.pin_memory(), y.pin_memory()
    d.setVertexVelocities(x.numpy())
    got = d.getVertexVelocities(out=y.numpy())
    assert np.array_equal(np.asarray(got).ravel(), x.numpy())
    assert np.array_equal(y.numpy(), x.numpy())
    d.close()


def _packing(seed):
    return synth.make_packing([21] * 30 + [26] * 7, [1.0] * 30 + [1.6] * 7, 1.05, 0.42, seed=seed, placement="rsa")


@pytest.mark.parametrize("integrator", ["nve", "langevin"])
@pytest.mark.parametrize("lanes", [1, 2, 4])
def test_single_step_calls(cuda_device, integrator, lanes):
    out = []
    for multi in (True, False):
        d = DPM2D.from_packing(_packing(8), potential="lennardJones", interaction="vertexSmooth", ea=10.0, el=5.0,
                               eb=0.1, dt=0.002)
        d.setLanes(lanes)
        d.setMultistep(multi)
        d.setSeed(5)
        d.calcNeighborList(d.setDisplacementCutoff(0.3, 2 * d.getMeanVertexRadius()))
        d.calcForceEnergy()
        if integrator == "nve":
            d.initNVE(1e-1, readState=False)
        else:
            d.initLangevin(1e-1, 1.0, readState=False)
        for n in (1, 1, 2, 1, 3, 1):
            (d.NVELoop if integrator == "nve" else d.langevinLoop)(n)
        out.append((d.getVertexPositions(), d.getVertexVelocities(), d.getVertexForces(), d.getUpdateCount()))
        d.close()
    assert out[0][3] == out[1][3]
    for a, b in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(a, b)


# chunks of 128 steps: one, two, the last plain call (7 chunks) and the first graph (8)
@pytest.mark.parametrize("steps", [1, 130, 896, 1000])
def test_plain_and_captured_sequences(cuda_device, steps):
    out = []
    for graphs in (True, False):
        d = DPM2D.from_packing(_packing(9), potential="harmonic", interaction="vertexVertex", dt=0.005)
        d.setUseGraphs(graphs)
        d.setSeed(6)
        d.calcNeighborList(d.setDisplacementCutoff(0.3, 2 * d.getMeanVertexRadius()))
        d.calcParticlePositions()
        d.calcRigidForceEnergy()
        d.initRigidLangevin(1e-2, 1.0, readState=False)
        d.rigidLangevinLoop(steps)
        out.append((d.getVertexPositions(), d.getParticleAngles(), d.getParticleVelocities(), d.getUpdateCount()))
        d.close()
    assert out[0][3] == out[1][3]
    for a, b in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(a, b)


# list cutoffs that leave many cells per side, about three, and one
@pytest.mark.parametrize("cutoff", [0.3, 8.0, 30.0])
def test_batch_lists(cuda_device, cutoff):
    sizes = [(1, 20), (3, 40), (60, 37), (9, 114)]  # 20 to 2220 vertices, rings up to most of a tile
    pks = [synth.make_packing([nv] * n, [1.0] * n, 1.05, 0.40 if n > 1 else 0.2, seed=70 + n, placement="rsa")
           for n, nv in sizes]
    kw = dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, ec=1.0)
    for pk in pks:
        pk.rad = pk.rad * 1.6
    b = Batch.from_packings(pks, **kw)
    b.setDisplacementCutoff(cutoff)
    b.calcNeighborLists()
    b.calcForceEnergy()
    f = b.getVertexForces()
    for s, pk in enumerate(pks):
        d = DPM2D.from_packing(pk, **kw)
        d.calcNeighborList(d.setDisplacementCutoff(cutoff, 2 * d.getMeanVertexRadius()))
        d.calcForceEnergy()
        fs = d.getVertexForces()
        assert rel_inf(f[b.system_slice(s)], fs) < 1e-12
        d.close()
    b.close()
