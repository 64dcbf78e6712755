"""The multi-step kernel's staged neighbourhood against one launch per step at
the edges of the stage: every potential with both lane counts, lists too long
for it, a box that its marking pass must not trust (rings a good part of the
box), coordinates beyond its fixed-point range, and rings of the largest and
smallest size.  The sums are formed in the same order, so FP64 states are
identical bit for bit."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth

pytestmark = pytest.mark.gpu


def _states(pk, potential, interaction, lanes, cutoff=0.5, steps=12, shift=0.0, dt=0.002):
    out = []
    for multi in (True, False):
        d = DPM2D.from_packing(pk, potential=potential, interaction=interaction, ea=10.0, el=5.0, eb=0.1, l1=0.05,
                               l2=0.2, dt=dt)
        d.setVertexPositions(pk.pos + shift)
        d.setLanes(lanes)
        d.setMultistep(multi)
        d.setSeed(3)
        d.calcNeighborList(d.setDisplacementCutoff(cutoff, 2 * pk.rad.mean()))
        d.calcForceEnergy()
        d.initNVE(1e-2, readState=False)
        d.NVELoop(steps)
        out.append((d.getVertexPositions(), d.getVertexVelocities(), d.getUpdateCount()))
        d.close()
    return out


def _same(out):
    assert out[0][2] == out[1][2]
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("potential", ["harmonic", "lennardJones", "adhesive", "wca"])
@pytest.mark.parametrize("interaction", ["vertexVertex", "vertexSmooth"])
@pytest.mark.parametrize("lanes", [1, 2])
def test_potentials(cuda_device, potential, interaction, lanes):
    n = 23  # a ragged last tile
    pk = synth.make_packing([17] * 12 + [23] * (n - 12), [1.0] * 12 + [1.9] * (n - 12), 1.05, 0.42, seed=4,
                            placement="rsa")
    _same(_states(pk, potential, interaction, lanes))


@pytest.mark.parametrize("cutoff", [4.0, 9.0])
@pytest.mark.parametrize("interaction", ["vertexVertex", "vertexSmooth"])
def test_lists_beyond_the_stage(cuda_device, cutoff, interaction):
    # 40 to 150 entries per vertex: some tiles or all of them read global memory
    pk = synth.make_packing([30] * 40, [1.0] * 40, 1.05, 0.45, seed=5, placement="rsa")
    _same(_states(pk, "harmonic", interaction, 2, cutoff=cutoff))


def test_rings_a_good_part_of_the_box(cuda_device):
    # four coarse rings: segments of a fifth of the box and more
    pk = synth.make_packing([5, 4, 6, 3], [1.0, 1.0, 1.0, 1.0], 1.0, 0.35, seed=6, placement="uniform")
    _same(_states(pk, "harmonic", "vertexSmooth", 2, dt=1e-3))


@pytest.mark.parametrize("boxes", [3.0e5, 9.0e5])
def test_coordinates_far_out(cuda_device, boxes):
    pk = synth.make_packing([20] * 12, [1.0] * 12, 1.05, 0.42, seed=7, placement="rsa")
    _same(_states(pk, "harmonic", "vertexSmooth", 2, shift=boxes * float(pk.box[0])))


@pytest.mark.parametrize("nv,lanes", [(96, 2), (95, 2), (128, 1), (3, 1), (3, 2)])
def test_ring_sizes(cuda_device, nv, lanes):
    pk = synth.make_packing([nv] * 9, [1.0] * 9, 1.05, 0.35 if nv > 10 else 0.06, seed=8, placement="rsa")
    _same(_states(pk, "wca", "vertexSmooth", lanes, dt=2e-4))


@pytest.mark.parametrize("interaction", ["vertexVertex", "vertexSmooth"])
def test_queue_in_parts(cuda_device, interaction):
    # far out, so that every listed slot is marked: 1,000 entries and more per
    # tile, several times what the queue holds at once
    pk = synth.make_packing([30] * 24, [1.0] * 24, 1.05, 0.45, seed=12, placement="rsa")
    for _ in range(3):  # the marking rounds end in another order each time
        _same(_states(pk, "harmonic", interaction, 2, cutoff=1.5, shift=9.0e5 * float(pk.box[0])))


@pytest.mark.parametrize("nv", [3, 31, 32, 33, 64, 65, 127, 128])
def test_ring_areas(cuda_device, nv):
    pk = synth.make_packing([nv] * 3, [1.0] * 3, 1.05, 0.2, seed=13)
    d = DPM2D.from_packing(pk)
    d.setLanes(1)
    d.calcNeighborList(d.setDisplacementCutoff(0.5, 2 * pk.rad.mean()))
    d.calcForceEnergy()
    x = pk.pos.reshape(3, nv, 2)
    x = x - x[:, :1]
    n = np.roll(x, -1, axis=1)
    area = 0.5 * np.abs((x[..., 0] * n[..., 1] - x[..., 1] * n[..., 0]).sum(1))
    # per term and side: two products of up to 4 R^2 and their difference, three
    # roundings of 2^-53, halved, R^2 = area / pi (2 area 2^-53); the sum adds
    # as much as 2^-53 area per term: 3 nv 2^-52 area for both sides
    assert np.abs(d.getAreas() - area).max() <= 4 * nv * 2.0 ** -52 * area.max()
    d.close()
