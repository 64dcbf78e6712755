"""Smooth interaction with short lists read from global memory (one launch per
op; no stage): every lane count against the CPU oracle.  A vertex's unit as a
segment end needs the length of its predecessor's segment, which another warp
forms (always with eight lanes per vertex, at warp edges and where a ring
closes with one), and short lists leave the least time between the two."""
import numpy as np
import pytest

import oracle
from cudaring_b200 import DPM2D, synth
from oracle.integrators import OracleState

from conftest import rel_inf

pytestmark = pytest.mark.gpu


def _state(nv, cutoff, seed):
    # overlapping rings: units in range, whatever the list's reach
    n = 400 // nv + 2
    pk = synth.make_packing([nv] * n, [1.0] * n, 1.05, 0.6, seed=seed, placement="uniform")
    S = oracle.System(pk.nv_list, pk.box, "harmonic", "vertexSmooth", 10.0, 5.0, 0.1, 1.0)
    return pk, S, S.cut_distance(cutoff)


def _context(pk, lanes, cutoff, precision="fp64"):
    d = DPM2D.from_packing(pk, potential="harmonic", interaction="vertexSmooth", ea=10.0, el=5.0, eb=0.1, ec=1.0,
                           dt=1e-3)
    d.setLanes(lanes)
    d.setMultistep(False)
    d.setPrecision(precision)
    d.calcNeighborList(d.setDisplacementCutoff(cutoff, 2 * pk.rad.mean()))
    return d


# rings that fill a tile of the lane count, leave a remainder, span warps or close inside one
@pytest.mark.parametrize("lanes,nv", [(1, 31), (1, 33), (1, 128), (2, 17), (2, 33), (2, 96), (4, 16), (4, 33),
                                      (4, 64), (8, 5), (8, 31), (8, 32)])
@pytest.mark.parametrize("cutoff", [0.0, 0.5])
def test_forces(cuda_device, lanes, nv, cutoff):
    pk, S, cut = _state(nv, cutoff, seed=20 + nv)
    S.neighbor_list(pk.pos, pk.rad, cut)
    ref = S.force_energy(pk.pos, pk.rad, pk.a0, pk.l0, pk.theta0)
    d = _context(pk, lanes, cutoff)
    for _ in range(3):  # the lengths left in shared memory are another tile's
        d.calcForceEnergy()
        # FP64 in another order of the sums: the bar of the parity tests
        assert rel_inf(d.getVertexForces(), ref["force"]) < 1e-12
    d.setPrecision("mixed")
    d.calcForceEnergy()
    f = d.getVertexForces()
    # FP32 pair units: the bar of the mixed-precision tests on overlapping packings
    assert np.linalg.norm(f - ref["force"]) <= 2e-6 * np.linalg.norm(ref["force"])
    d.close()


@pytest.mark.parametrize("lanes,nv", [(1, 33), (2, 33), (4, 33), (8, 31)])
def test_steps(cuda_device, lanes, nv):
    pk, S, _ = _state(nv, 0.5, seed=40 + nv)
    st = OracleState(S, pk)
    d = _context(pk, lanes, 0.5)
    d.calcForceEnergy()
    d.initNVE(0.0, readState=True)
    d.NVELoop(10)
    for _ in range(10):
        st.nve_step(1e-3)
    # ten steps of FP64 rounding, as the trajectory tests
    assert rel_inf(d.getVertexPositions(), st.pos) < 1e-12
    d.close()
