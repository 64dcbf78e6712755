"""The batched list build with its cells by one CTA per system and by clusters of
2, 4 and 8 (few large systems): lists and forces of each system against its own
context, whose build is the single-system one; and rebuilds inside FIRE."""
import numpy as np
import pytest

from cudaring_b200 import DPM2D, synth
from cudaring_b200.batch import Batch

from conftest import rel_inf

pytestmark = pytest.mark.gpu

KW = dict(potential="harmonic", interaction="vertexVertex", ea=10.0, el=5.0, eb=0.1, ec=1.0)


def _lattice(rings, nv, seed):
    # jittered rings on a square lattice (no rejection sampling at large sizes)
    small = synth.make_packing([nv] * 2, [1.0] * 2, 1.05, 0.1, seed=seed)
    m = int(np.ceil(np.sqrt(rings)))
    l0, rad = small.l0[0], small.rad[0]
    r = l0 / (2 * np.sin(np.pi / nv))
    L = m * 2.05 * (r + rad)
    th = 2 * np.pi * np.arange(nv) / nv
    i = np.random.default_rng(seed).permutation(m * m)[:rings]
    rng = np.random.default_rng(seed + 1)
    x = ((i % m + 0.5) * L / m)[:, None] + r * np.cos(th) + rng.normal(0, 0.1 * rad, (rings, nv))
    y = ((i // m + 0.5) * L / m)[:, None] + r * np.sin(th) + rng.normal(0, 0.1 * rad, (rings, nv))
    n = rings * nv
    return synth.Packing(nv_list=np.full(rings, nv), pos=np.stack([x, y], -1).reshape(-1), vel=np.zeros(2 * n),
                         rad=np.full(n, rad), l0=np.full(n, l0), theta0=np.full(n, small.theta0[0]),
                         a0=np.full(rings, 1.0), box=np.array([L, L]), centres=np.zeros((rings, 2)))


# vertices of the systems: at and past the line of one CTA, clusters of 8, 4 and 2
# (one, 37 and 74 systems a chip of 148 SMs), small and large ones together, few cells
@pytest.mark.parametrize("rings", [[102], [103], [500], [4000], [500, 3, 60, 120], [103] * 37, [103] * 74])
@pytest.mark.parametrize("cutoff", [0.5, 40.0])
def test_lists(cuda_device, rings, cutoff):
    if cutoff > 1 and max(rings) > 200:
        pytest.skip("every pair listed")
    kinds = {n: _lattice(n, 20, seed=n) for n in set(rings)}
    pks = [kinds[n] for n in rings]
    b = Batch.from_packings(pks, **KW)
    b.setDisplacementCutoff(cutoff)
    forces = []
    for _ in range(2):  # the second build starts from the first one's cells
        b.calcNeighborLists()
        b.calcForceEnergy()
        forces.append(b.getVertexForces())
    assert np.array_equal(forces[0], forces[1])
    single = {}
    for n, pk in kinds.items():
        d = DPM2D.from_packing(pk, **KW)
        d.calcNeighborList(d.setDisplacementCutoff(cutoff, 2 * d.getMeanVertexRadius()))
        d.calcForceEnergy()
        single[n] = d.getVertexForces()
        d.close()
    for s, n in enumerate(rings):
        # the same pairs summed in another order
        assert rel_inf(forces[0][b.system_slice(s)], single[n]) < 1e-12
    b.close()


def test_rebuilds_in_a_run(cuda_device):
    # a small displacement cutoff: rebuilds of one system of the batch and of the other
    pks = [_lattice(500, 20, seed=1), _lattice(120, 20, seed=2)]
    out = []
    for cutoff in (0.02, 0.5):
        b = Batch.from_packings(pks, **KW)
        b.setDisplacementCutoff(cutoff)
        b.initFIRE([0.2, 0.5, 1.1, 0.99, 1e-3, 1e-2, 0.2], 20, dt=np.full(2, 1e-3))
        b.fireMinimize(1e-14, 50)
        out.append(b.getVertexPositions())
        b.close()
    # the force does not depend on when its list was built, beyond the order of
    # its terms: 50 iterations of FP64 rounding
    assert rel_inf(out[0], out[1]) < 1e-11
