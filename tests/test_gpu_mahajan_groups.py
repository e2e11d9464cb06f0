"""Mahajan's steep nodes (|dV/dt| > 20: ten sub-steps) run in groups of 32 with
the rates split over four warps: none, one, a full and an overfull group in a
CTA, and more nodes than one wave of CTAs takes.  (Several sub-steps a step run in
test_gpu_tissue.py's Mahajan case.)"""
import numpy as np
import pytest

from oracle import oracle as O
from ucla_cmg_b200 import capi
from ucla_cmg_b200.simulation import ionic_step

pytestmark = pytest.mark.gpu

REST = np.array([-81.4359, 0.002789, 0.96679, 0.97859, 0.014994, 0.044487, 0.091992, 2.1933, 0.23277, 0.24868, 101.6418,
                 95.4278, 0.009495, 3.7e-005, 0.96094, 0.003718, 6.7e-005, 0.010571, 0.024659, 11.5909, 0.00533, 0.99047,
                 0.005333, 0.17488, 21.5955, 20.0206])


@pytest.mark.parametrize("n,share", [(1, 1.0), (31, 1.0), (33, 1.0), (127, 0.0), (128, 1.0), (129, 0.3), (1000, 0.25),
                                     (70001, 0.02)])
def test_steep_cells_against_the_oracle(gpu, n, share):
    rng = np.random.default_rng(n)
    m = min(n, 257)
    S = REST[None, :] * rng.uniform(0.98, 1.0, (m, 26))
    V = rng.uniform(-85.0, -75.0, m)
    steep = rng.random(m) < share
    S[steep, 1] = 0.9                                # open sodium gates
    V[steep] = rng.uniform(-40.0, 0.0, steep.sum())
    types = rng.integers(0, 9, m).astype(np.uint8)
    ist = np.zeros(m)
    c = O.Cells(O.MAHAJAN, m, types=types)
    c.state[:] = S
    ref = c.compute_ion(V, ist, 0.02)
    assert (np.abs(ref[steep]) > 20).all()
    at = np.arange(n) % m
    st = np.ascontiguousarray(S[at])
    dv = ionic_step(capi.MAHAJAN, V[at], ist[at], st, 0.02, node_type=types[at])
    # the FP64 tolerance of the cell models' golden vectors
    assert np.max(np.abs(dv - ref[at]) / np.maximum(np.abs(ref[at]), 1.0)) < 1e-8
    assert np.max(np.abs(st - c.state[at])[:, 1:] / np.maximum(np.abs(c.state[at][:, 1:]), 1e-12)) < 1e-8
