"""Mahajan's nodes have the same bits alone, in a group of steep nodes and beside others
(FP32 and FP64, one and several sub-steps a step): grouping moves work, not results."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_mahajan_groups import REST
from ucla_cmg_b200 import capi
from ucla_cmg_b200.capi import check, ptr

pytestmark = pytest.mark.gpu


def _phase(prec, V, S, dt, ionic_dt):
    V, S, n = V.copy(), np.array(S, order="C"), len(V)
    mo = capi.ModelDesc()
    mo.model, mo.n_types = capi.MAHAJAN, 1
    ist = np.zeros(n)
    check(capi.lib().ep_ionic_phase(C.byref(mo), prec, n, dt, ionic_dt, 1.0, ptr(V), ptr(ist), ptr(S)))
    return np.column_stack([V, S[:, 1:]])


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("dt,ionic_dt", [(0.02, 0.02), (0.05, 0.02), (0.05, 0.01)])
def test_every_node_as_alone(gpu, prec, dt, ionic_dt):
    rng = np.random.default_rng(7)
    m = 41
    S = REST[None, :] * rng.uniform(0.98, 1.0, (m, 26))
    V = rng.uniform(-85.0, -75.0, m)
    steep = np.arange(m) % 3 == 0
    S[steep, 1] = 0.9                                # open sodium gates
    V[steep] = rng.uniform(-40.0, 0.0, steep.sum())
    alone = np.concatenate([_phase(prec, V[k:k + 1], S[k:k + 1], dt, ionic_dt) for k in range(m)])
    assert np.all(np.isfinite(alone)) and np.ptp(alone[:, 0]) > 10
    for n in (m, 500, 3000):
        at = rng.permutation(n) % m
        assert np.array_equal(_phase(prec, V[at], S[at], dt, ionic_dt), alone[at])
