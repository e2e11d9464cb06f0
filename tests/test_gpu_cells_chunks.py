"""The plugin-level entries over more cells than one chunk of their buffers
holds (131072), each option in turn: every cell's result is the one of a short
call, whatever chunk and place it falls in."""
import numpy as np
import pytest

from ucla_cmg_b200 import capi, workloads as W
from ucla_cmg_b200.simulation import ionic_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("model,types,gks", [(capi.TUSSCHER, True, True), (capi.TUSSCHER, False, False),
                                             (capi.MAHAJAN, False, False), (capi.LUORUDY, False, False)])
def test_chunks_give_every_cell_its_own_result(gpu, prec, model, types, gks):
    n, m = (1 << 17) + 37, 211
    ns = capi.model_nstate(model)
    rest = {capi.TUSSCHER: [-85.423, 136.89, 8.604, 0.000126, 0.00621, 0.4712, 0.0095, 0.00172, 0.7444, 0.7045, 0.00036,
                            3.373e-5, 0.7888, 0.9755, 0.9953, 0.999998, 2.42e-8, 3.64, 0.9073],
            capi.MAHAJAN: [-81.4359, 0.002789, 0.96679, 0.97859, 0.014994, 0.044487, 0.091992, 2.1933, 0.23277, 0.24868,
                           101.6418, 95.4278, 0.009495, 3.7e-005, 0.96094, 0.003718, 6.7e-005, 0.010571, 0.024659, 11.5909,
                           0.00533, 0.99047, 0.005333, 0.17488, 21.5955, 20.0206],
            capi.LUORUDY: [.001, 0.0001, 0.99, .001, 0.9, .001, 0.0000001, -80.0]}[model]
    rng = np.random.default_rng(4)
    S = np.array(rest)[None, :] * rng.uniform(0.98, 1.0, (m, ns))
    V = rng.uniform(-85.0, -60.0, m)
    ist = rng.uniform(0.0, 1e4, m)
    kw = {}
    if types:
        kw = dict(node_type=rng.integers(0, 3, m).astype(np.uint8), type_consts=W.tt_type_consts())
    if gks:
        kw["gks_scale"] = rng.uniform(0.5, 1.5, m)
    s0 = S.copy()
    d0 = ionic_step(model, V, ist, s0, 0.01, precision=prec, tt_jacobian=capi.TT_JAC_TRUE, **kw)
    at = np.arange(n) % m
    big = {k: (v[at] if k != "type_consts" else v) for k, v in kw.items()}
    s1 = np.ascontiguousarray(S[at])
    d1 = ionic_step(model, V[at], ist[at], s1, 0.01, precision=prec, tt_jacobian=capi.TT_JAC_TRUE, **big)
    assert np.all(np.isfinite(d0)) and np.ptp(d0) > 0
    assert np.array_equal(d1, d0[at])
    assert np.array_equal(s1, s0[at])
