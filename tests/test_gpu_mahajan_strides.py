"""Mahajan's steep nodes where a step has strides of the node's own (backward Euler and
explicit splittings), against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Monodomain

pytestmark = pytest.mark.gpu
D = M.sigma_to_D(1.2, 0.2)


@pytest.mark.parametrize("scheme", [capi.SCHEME_BE, capi.SCHEME_EXPLICIT])
def test_strides_against_the_oracle(gpu, scheme):
    m = M.slab(11, 11, 4, 0.2, 0.2, 0.06)
    dt, idt = 0.05, 0.005                           # (strides that fill a step exactly end in one of length 0: NaN)
    types = (np.arange(m.n) % 9).astype(np.uint8)
    cells = O.Cells(O.MAHAJAN, m.n, types=types)
    s = O.Sim(O.Csr(m.xyz, m.tets, m.fibers, D, 1.0, dt), cells, dt, idt, cg_tol=1e-12, cg_maxit=2000, jacobi_steps=1)
    s.set_scheme(scheme)
    s.V[:] = V0 = cells.initial_voltage()
    g = Monodomain(m, capi.MAHAJAN, capi.FP64, dt=dt, ionic_dt=idt, D=D, cg_tol=1e-12 if scheme == capi.SCHEME_BE else 0.0,
                   cg_maxit=2000, node_type=types, scheme=scheme)
    g.set_voltage(V0)
    blk = M.corner_block(m, 3, 3)
    amp = 50.0 * 1.55e-4 / 2.58e-8
    g.set_stimulus(blk, 0.0, 2.0, amp)
    worst = 0.0
    for k in range(200):
        s.istim[:] = 0.0
        if k < 40:
            s.istim[blk] = amp
        s.step()
        if k % 50 == 49:
            g.step(50)
            worst = max(worst, np.max(np.abs(g.voltage() - s.V)) / np.max(np.abs(s.V)))
    assert np.max(s.V) > 0.0 and worst <= 1e-6, worst
    # the tolerances of the Crank-Nicolson case in test_gpu_tissue.py
    assert np.allclose(g.states()[:, 1:], cells.state[:, 1:], rtol=1e-6, atol=1e-9)
    g.close()
