"""The ten Tusscher source of the time steps (csrc/tt_step.cuh: one division per
gate, Jacobian written out) against the one in the reference's order (csrc/tt.cuh),
on the host, over the golden vectors' states; and the quotient of the FP32 kernels
(csrc/common.cuh, dv) against the true one."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from ucla_cmg_b200 import capi

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "native", "tt_step_host.cu")
OUT = os.path.join(HERE, "native", "_build", "libtt_step_host.so")
DEPS = [SRC] + [os.path.join(ROOT, "ucla_cmg_b200", "csrc", f) for f in ("tt.cuh", "tt_step.cuh", "common.cuh")]
CONC = [1, 2, 3, 10, 17, 18]                     # Ki, Nai, Cai, Cass, CaSR, R'


@pytest.fixture(scope="module")
def lib():
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    nvcc = nvcc if os.path.exists(nvcc) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("nvcc not available to build the host harness")
    if not os.path.exists(OUT) or os.path.getmtime(OUT) < max(os.path.getmtime(d) for d in DEPS):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                        "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-I", os.path.join(ROOT, "include"),
                        "-o", OUT, SRC], check=True, capture_output=True)
    return C.CDLL(OUT)


@pytest.mark.parametrize("dt", [0.005, 0.02, 0.1])
def test_time_step_source_equals_the_reference_order(lib, dt):
    g = np.load(os.path.join(HERE, "golden", "kat_tt.npz"))
    V = np.ascontiguousarray(g["V"])
    consts = np.ascontiguousarray(capi.default_consts(capi.TUSSCHER, 0))
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    out = {}
    for step, fp32 in ((0, 0), (1, 0), (1, 1)):
        S, dv = np.array(g["states_in"]), np.zeros(len(V))
        lib.tt_step_host(step, fp32, len(V), C.c_double(dt), p(consts), C.c_double(1e-6 if fp32 else 1e-12), p(V), p(S),
                         p(dv))
        out[step, fp32] = S[:, 1:], dv
    gates = [k - 1 for k in range(1, 19) if k not in CONC]
    ref, dref = out[0, 0]
    S, dv = out[1, 0]
    # gates: the same formula, some twenty roundings.  Concentrations: both Newton
    # runs end at a residual of 1e-12, 1e-8 of the smallest (Cai), tenfold for safety
    assert np.max(np.abs(S - ref)[:, gates] / np.abs(ref[:, gates])) < 1e-13
    assert np.max(np.abs(S - ref) / np.abs(ref)) < 1e-7
    assert np.max(np.abs(dv - dref) / np.maximum(np.abs(dref), 1.0)) < 1e-6
    # FP32 gates: arguments of exponentials up to 20, four of them, each rounded
    S32 = out[1, 1][0]
    assert np.max(np.abs(S32 - ref)[:, gates] / np.maximum(np.abs(ref[:, gates]), 1e-6)) < 2e-5
    assert np.all(np.isfinite(S32)) and np.all(np.isfinite(out[1, 1][1]))


def test_quotient_is_within_half_an_ulp():
    """dv's steps with the reciprocal estimate off by up to one ulp either way; the
    products of two FP32 numbers are exact in FP64."""
    rng = np.random.default_rng(1)
    f = np.float32
    a, b = (np.exp2(rng.uniform(-20, 20, 400000)) * rng.choice([-1, 1], 400000)).astype(f), \
        np.exp2(rng.uniform(-20, 20, 400000)).astype(f)
    exact = a.astype(np.float64) / b
    ulp = np.spacing(np.abs(exact).astype(f)).astype(np.float64)
    for off in (-1, 0, 1):
        r = (1.0 / b.astype(np.float64)).astype(f)
        r = r if off == 0 else np.nextafter(r, f(off * np.inf))
        q = a * r
        rem = (a.astype(np.float64) - b.astype(np.float64) * q).astype(f)
        got = (q.astype(np.float64) + rem.astype(np.float64) * r).astype(f)
        assert np.max(np.abs(got - exact) / ulp) <= 0.51
