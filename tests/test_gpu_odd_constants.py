"""Cell constants at their limits: zero and infinite denominators of Mahajan's rates in
FP32 as in FP64, ten Tusscher fluxes switched off by an infinite or very large constant,
and the device's quotients (csrc/common.cuh, dv and dvc) against FP64 ones."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from test_gpu_mahajan_groups import REST
from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Monodomain, ionic_step

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _mahajan(prec, k, value):
    c = np.array([capi.default_consts(capi.MAHAJAN, 0)])
    c[0, k] = value
    V = np.array([-81.4, -60.0, -20.0, 10.0])
    S = np.tile(REST, (len(V), 1))
    dv = ionic_step(capi.MAHAJAN, V, 0.0, S, 0.01, precision=prec, type_consts=c)
    return np.column_stack([S[:, 1:], dv])


@pytest.mark.parametrize("k", [14, 16, 17, 19])
def test_mahajan_denominators(gpu, k):
    # an infinite denominator is one of 1e30 to the last bit of every state
    big = _mahajan(capi.FP32, k, 1e30)
    assert np.all(np.isfinite(big))
    assert np.array_equal(_mahajan(capi.FP32, k, np.inf), big)
    # a zero one gives infinities and NaN where FP64's division does
    a, b = _mahajan(capi.FP64, k, 0.0), _mahajan(capi.FP32, k, 0.0)
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b))
    assert np.array_equal(np.sign(a[np.isinf(a)]), np.sign(b[np.isinf(b)]))
    assert np.isfinite(a).any() and not np.all(np.isfinite(a))


@pytest.mark.parametrize("k", [23, 31, 42])                   # K_mNa, K_pCa, K_up
@pytest.mark.parametrize("value", [np.inf, 1e30])
@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
def test_ten_tusscher_fluxes_switched_off(gpu, k, value, prec):
    """An infinite half-saturation constant is one of 9e5 to every digit that counts."""
    m = M.slab(3, 3, 2, 0.02, 0.02, 0.01)
    out = []
    for v in (value, 9e5):
        c = np.array([capi.default_consts(capi.TUSSCHER, 0)])
        c[0, k] = v
        g = Monodomain(m, capi.TUSSCHER, prec, dt=0.02, ionic_dt=0.02, D=(1e-3,) * 3, type_consts=c,
                       tt_jacobian=capi.TT_JAC_TRUE)
        g.set_voltage(-80.0)
        g.step(5)
        out.append(np.column_stack([g.states()[:, 1:], g.voltage()]))
        g.close()
    assert np.all(np.isfinite(out[0]))
    # a flux 1e-5 of its ordinary size against none over 0.1 ms, and FP32's Newton stop (1e-6)
    assert np.max(np.abs(out[0] - out[1]) / np.maximum(np.abs(out[1]), 1e-6)) < (1e-5 if prec == capi.FP64 else 1e-4)


@pytest.fixture(scope="module")
def quotients():
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    nvcc = nvcc if os.path.exists(nvcc) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("nvcc not available to build the harness")
    src, out = (os.path.join(HERE, "native", f) for f in ("quotient.cu", "_build/libquotient.so"))
    deps = [src, os.path.join(ROOT, "ucla_cmg_b200", "csrc", "common.cuh")]
    if not os.path.exists(out) or os.path.getmtime(out) < max(os.path.getmtime(d) for d in deps):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-Xcompiler", "-fPIC",
                        "-shared", "-I", os.path.join(ROOT, "include"), "-o", out, src], check=True, capture_output=True)
    lib = C.CDLL(out)

    def f(a, b):
        ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        y = torch.empty(2, len(a), device="cuda")
        torch.cuda.synchronize()
        assert lib.quotients(len(a), C.c_void_p(ta.data_ptr()), C.c_void_p(tb.data_ptr()), C.c_void_p(y.data_ptr())) == 0
        return y.cpu().numpy()
    return f


def test_device_quotients(gpu, quotients):
    rng = np.random.default_rng(2)
    f32, n = np.float32, 200000
    s = lambda k: rng.choice([-1.0, 1.0], k)  # noqa: E731
    a = (np.exp2(rng.uniform(-40, 40, n)) * s(n)).astype(f32)
    b = (np.exp2(rng.uniform(-40, 40, n)) * s(n)).astype(f32)
    # the ends of the denominators' range, with quotients and remainders that stay normal
    a = np.concatenate([a, (np.exp2(rng.uniform(30, 40, 2000)) * s(2000)).astype(f32),
                        (np.exp2(rng.uniform(-60, -50, 2000)) * s(2000)).astype(f32)])
    b = np.concatenate([b, (np.exp2(rng.uniform(125, 125.99, 2000)) * s(2000)).astype(f32),
                        (np.exp2(rng.uniform(-125.9, -125, 2000)) * s(2000)).astype(f32)])
    exact = a.astype(np.float64) / b
    ulp = np.spacing(np.abs(exact).astype(f32)).astype(np.float64)
    assert np.min(np.abs(exact)) > 2.0 ** -126
    for got in quotients(a, b):
        assert np.max(np.abs(got - exact) / ulp) <= 0.51
    # dvc: zero, infinite and NaN operands as with /
    v = np.array([0.0, -0.0, 1.0, -2.5, np.inf, -np.inf, np.nan, 3e38], f32)
    a, b = (x.ravel().copy() for x in np.meshgrid(v, v[:-1]))
    with np.errstate(all="ignore"):
        want = a / b
    assert np.array_equal(quotients(a, b)[1], want, equal_nan=True)


@pytest.mark.parametrize("k", [23, 31])
def test_learned_step_with_a_flux_switched_off(gpu, k):
    """The nodes the network takes advance V by the current balance, which an infinite
    constant leaves finite."""
    from ucla_cmg_b200.surrogate import Surrogate
    m = M.slab(5, 5, 3, 0.04, 0.04, 0.02)
    out = []
    for v in (np.inf, 9e5):
        c = np.array([capi.default_consts(capi.TUSSCHER, 0)])
        c[0, k] = v
        g = Monodomain(m, capi.TUSSCHER, capi.SURROGATE, dt=0.1, ionic_dt=0.02, D=(1e-3,) * 3, type_consts=c,
                       tt_jacobian=capi.TT_JAC_TRUE)
        Surrogate.load().deploy(g)
        g.set_voltage(-85.2)
        st = g.step(1)
        out.append(g.voltage())
        assert st["fallback_nodes"] < m.n
        g.close()
    # a current of at most 1 uA/uF, 1e-4 of it, over 0.1 ms, and FP32's digits of V
    assert np.all(np.isfinite(out[0])) and np.max(np.abs(out[0] - out[1])) < 1e-4
