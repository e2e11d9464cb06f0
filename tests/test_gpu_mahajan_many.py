"""Mahajan's steep nodes in long runs, as a front along the node order leaves them: the
CTAs' lists of 65 to 1024 nodes, which FP64 takes one thread a node, give every node the
result that it has alone, and the same bits in every run."""
import numpy as np
import pytest

from test_gpu_mahajan_alone import _phase
from test_gpu_mahajan_groups import REST
from ucla_cmg_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("dt,ionic_dt", [(0.02, 0.02), (0.05, 0.02)])
def test_long_lists(gpu, prec, dt, ionic_dt):
    rng = np.random.default_rng(11)
    m = 36
    S = REST[None, :] * rng.uniform(0.98, 1.0, (m, 26))
    V = rng.uniform(-85.0, -75.0, m)
    steep = np.arange(m) % 4 != 3
    S[steep, 1] = 0.9                                # open sodium gates
    V[steep] = rng.uniform(-40.0, 0.0, steep.sum())
    alone = np.concatenate([_phase(prec, V[k:k + 1], S[k:k + 1], dt, ionic_dt) for k in range(m)])
    # up to one CTA per SM, and beyond, with one to eight chunks of 128 nodes a CTA
    for n, run in ((300, 300), (15000, 1024), (20000, 97), (40000, 128), (40000, 77), (131072, 1024), (131072, 31)):
        at = np.arange(n) // run % m
        got = _phase(prec, V[at], S[at], dt, ionic_dt)
        assert np.array_equal(got, _phase(prec, V[at], S[at], dt, ionic_dt))
        if prec == capi.FP32:
            assert np.array_equal(got, alone[at]), (n, run)
        # FP64's two ways round differently: a hundredth of the tolerance to the oracle
        # (test_gpu_mahajan_groups.py)
        floor = np.r_[1.0, np.full(25, 1e-12)]
        assert np.max(np.abs(got - alone[at]) / np.maximum(np.abs(alone[at]), floor)) < 1e-10, (n, run)
