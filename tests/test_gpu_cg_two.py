"""The two-pass CG kernel, which matrices that stream from DRAM run: its gather forms,
thread counts and predictors against the one-pass kernel on a mesh just large enough
for the shapes named here, a batch whose instances get from one to all but two CTAs,
and a wait that gives up."""
import numpy as np
import pytest

from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Batch, Monodomain

pytestmark = pytest.mark.gpu
D = M.sigma_to_D(1.2, 0.2)
# the kernels take the same iterates; recurrences and sums differ in rounding only
TOL = {capi.FP64: 1e-12, capi.FP32: 1e-6}
ONE_PASS = dict(cg_block=256, cg_per_sm=2, cg_batch=4)


def _slab(*dims):
    return M.slab(*dims, *(0.02 * (k - 1) for k in dims))


@pytest.fixture(scope="module")
def big():
    m = _slab(203, 199, 27)
    rng = np.random.default_rng(0)
    return m, -85.0 + 120.0 * (m.xyz[:, 0] < m.xyz[:, 0].mean()) + rng.normal(0, 1.0, m.n)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
def test_shapes_and_predictors_equal_the_one_pass_kernel(gpu, big, prec):
    m, V = big
    g = Monodomain(m, capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02, D=D, cg_tol=1e-7)
    S = g.states()

    def run(cfg, predict):
        g.set_launch_config(cg_predict=predict, cg_prefetch=cfg.pop("cg_prefetch", 0), **cfg)
        g.set_states(S)
        g.set_voltage(V)
        it = [g.diffusion_half_step()[0]]
        if predict:
            g.step(2)
        return it, g.voltage()

    for predict in (0, 1, 2):
        it, ref = run(dict(ONE_PASS), predict)
        assert it[0] > 3
        for cfg in (dict(cg_block=768, cg_per_sm=2, cg_batch=4), dict(cg_block=768, cg_per_sm=1, cg_batch=4, cg_prefetch=2),
                    dict(cg_block=256, cg_per_sm=4, cg_batch=8), dict(cg_block=128, cg_per_sm=3, cg_batch=8),
                    dict(cg_block=256, cg_per_sm=2, cg_batch=32, cg_prefetch=3), dict(cg_block=256, cg_per_sm=0, cg_batch=16)):
            it2, got = run(dict(cfg), predict)
            assert it2 == it, cfg
            # (a predicted run goes through two whole steps of the cell model)
            assert np.max(np.abs(got - ref)) <= (10 if predict else 1) * TOL[prec] * np.max(np.abs(ref)), (cfg, predict)
    g.close()


@pytest.mark.parametrize("prec,cfg", [(capi.FP64, dict(cg_block=768, cg_per_sm=1)), (capi.FP32, dict(cg_block=768, cg_per_sm=1)),
                                      (capi.FP32, dict(cg_block=256, cg_per_sm=4, cg_batch=8))])
def test_uneven_batch(gpu, big, prec, cfg):
    meshes = [_slab(9, 7, 5), big[0], _slab(3, 3, 3)]
    rng = np.random.default_rng(4)
    V = np.concatenate([-85.0 + 120.0 * (m.xyz[:, 0] < m.xyz[:, 0].mean()) + rng.normal(0, 1.0, m.n) for m in meshes])
    out = []
    for c in (cfg, ONE_PASS):
        b = Batch([dict(mesh=m, D=D) for m in meshes], capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02)
        b.set_launch_config(**c)
        b.set_voltage(V)
        b.diffusion_half_step()
        out.append((list(b.cg_last()[0]), b.voltage()))
        b.close()
    assert out[0][0] == out[1][0]
    assert np.max(np.abs(out[0][1] - out[1][1])) <= TOL[prec] * np.max(np.abs(V))


def test_a_wait_that_gives_up_leaves_the_handle_usable(gpu, big):
    m, V = big
    g = Monodomain(m, capi.TUSSCHER, capi.FP32, dt=0.1, ionic_dt=0.02, D=D)
    g.set_launch_config(cg_block=256, cg_per_sm=2, cg_batch=32)
    g.set_voltage(V)
    g.diffusion_half_step()
    ref = g.voltage()
    g.set_wait_limits(grid_polls=2000)
    g.test_hold_barrier(3)
    g.set_voltage(V)
    with pytest.raises(capi.EPError):
        g.diffusion_half_step()
    g.test_hold_barrier(0)
    g.set_wait_limits()
    g.set_voltage(V)
    g.diffusion_half_step()
    assert np.array_equal(g.voltage(), ref)
    g.close()
