"""A NaN voltage reaches every gate that depends on it, in the time steps' ten Tusscher
source (csrc/tt_step.cuh) as in the reference's order of operations (csrc/tt.cuh)."""
import ctypes as C
import os

import numpy as np
import pytest

from test_tt_step_host import HERE, lib  # noqa: F401
from ucla_cmg_b200 import capi


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("V", [np.nan, 20.0])
def test_nan_voltage_in_both_orders(lib, fp32, V):  # noqa: F811
    S0 = np.load(os.path.join(HERE, "golden", "kat_tt.npz"))["states_in"][:4]
    consts = np.ascontiguousarray(capi.default_consts(capi.TUSSCHER, 0))
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    Vs, out = np.full(len(S0), V), []
    for step in (0, 1):
        S, dv = np.array(S0), np.zeros(len(S0))
        lib.tt_step_host(step, fp32, len(S0), C.c_double(0.02), p(consts), C.c_double(1e-6), p(Vs), p(S), p(dv))
        out.append((np.isnan(S[:, 1:]), np.isnan(dv)))
    # (the six concentrations' Newton runs stop at once or with NaN: not compared)
    gates = [k - 1 for k in (4, 5, 6, 7, 8, 9, 11, 12, 13, 14, 15, 16)]
    assert np.array_equal(out[0][0][:, gates], out[1][0][:, gates])
    assert np.array_equal(out[0][1], out[1][1])
    assert out[1][0][:, gates].any() == np.isnan(V)
