"""Rounding errors of the ten Tusscher gates of the time steps (csrc/tt_step.cuh, one
division a gate) against the model's formulas in long double, beside those of the
reference's order of operations (csrc/tt.cuh), on the host."""
import ctypes as C
import os

import numpy as np
import pytest

from test_tt_step_host import HERE, lib  # noqa: F401
from ucla_cmg_b200 import capi

GATES = (4, 5, 6, 7, 8, 9, 11, 12, 13, 14, 15, 16)      # Xr1 Xr2 Xs m h j d f f2 fCass s r


def _gates(V, cass):
    """(steady state, time constant) of the epicardial cell's gates (Tusscher.cc:5-55)."""
    e = np.exp
    f = lambda a: 1 / (1 + e(a))  # noqa: E731
    lo = V < -40
    ah = np.where(lo, c("0.057") * e(-(V + 80) / c("6.8")), 0)
    bh = np.where(lo, c("2.7") * e(c("0.079") * V) + 310000 * e(c("0.3485") * V),
                  c("0.77") / (c("0.13") * (1 + e(-(V + c("10.66")) / c("11.1")))))
    aj = np.where(lo, (-25428 * e(c("0.2444") * V) - c("6.948e-06") * e(c("-0.04391") * V)) * (V + c("37.78"))
                  * f(c("0.311") * (V + c("79.23"))), 0)
    bj = np.where(lo, c("0.02424") * e(c("-0.01052") * V) * f(c("-0.1378") * (V + c("40.14"))),
                  c("0.6") * e(c("0.057") * V) * f(c("-0.1") * (V + 32)))
    hj = f((V + c("71.55")) / c("7.43")) ** 2
    q = 1 / (1 + (20 * cass) ** 2)
    v27 = (V + 27) ** 2
    return [(f((-26 - V) / 7), 2700 * f((-45 - V) / 10) * f((V + 30) / c("11.5"))),
            (f((V + 88) / 24), c("3.36") * f((-60 - V) / 20) * f((V - 60) / 20)),
            (f((-5 - V) / 14), 1400 / np.sqrt(1 + e((5 - V) / 6)) * f((V - 35) / 15) + 80),
            (f((c("-56.86") - V) / c("9.03")) ** 2, f((-60 - V) / 5) * c("0.1") * (f((V + 35) / 5) + f((V - 50) / 200))),
            (hj, 1 / (ah + bh)), (hj, 1 / (aj + bj)),
            (f((-8 - V) / c("7.5")), (c("1.4") * f((-35 - V) / 13) + c("0.25")) * c("1.4") * f((V + 5) / 5) + f((50 - V) / 20)),
            (f((V + 20) / 7), c("1102.5") * e(-v27 / 225) + 200 * f((13 - V) / 10) + 180 * f((V + 30) / 10) + 20),
            (c("0.67") * f((V + 35) / 7) + c("0.33"), 562 * e(-v27 / 240) + 31 * f((25 - V) / 10) + 80 * f((V + 30) / 10)),
            (c("0.6") * q + c("0.4"), 80 * q + 2),
            (f((V + 20) / 5), 85 * e(-(V + 45) ** 2 / 320) + 5 * f((V - 20) / 5) + 3),
            (f((20 - V) / 6), c("9.5") * e(-(V + 40) ** 2 / 1800) + c("0.8"))]


def c(text):
    """A constant of the sources: the double that stands there."""
    return np.longdouble(float(text))


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("dt", [0.005, 0.02, 0.1])
def test_gate_errors_are_no_larger_than_the_reference_orders(lib, fp32, dt):  # noqa: F811
    g = np.load(os.path.join(HERE, "golden", "kat_tt.npz"))
    rng = np.random.default_rng(1)
    k = rng.integers(0, len(g["V"]), 6000)
    S = g["states_in"][k] * (1 + 1e-3 * rng.uniform(-1, 1, (len(k), 19)))
    V = g["V"][k] + rng.uniform(-1, 1, len(k))
    if fp32:
        S, V, dt = S.astype(np.float32).astype(float), V.astype(np.float32).astype(float), float(np.float32(dt))
    S, V = np.ascontiguousarray(S), np.ascontiguousarray(V)
    consts = np.ascontiguousarray(capi.default_consts(capi.TUSSCHER, 0))
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    exact = np.stack([(S[:, j] + dt * inf / tau) / (1 + dt / tau)
                      for j, (inf, tau) in zip(GATES, _gates(V.astype(np.longdouble), S[:, 10].astype(np.longdouble)))], 1)
    err = []
    for step in (0, 1):
        out, dv = S.copy(), np.zeros(len(V))
        lib.tt_step_host(step, fp32, len(V), C.c_double(dt), p(consts), C.c_double(1e-6 if fp32 else 1e-12), p(V), p(out),
                         p(dv))
        err.append(np.linalg.norm((out[:, GATES] - exact).astype(float), axis=0))
    # 6000 roundings a gate: the norms' own scatter is 1 %; five times that
    assert np.all(err[1] <= 1.05 * err[0]), err[1] / err[0]
