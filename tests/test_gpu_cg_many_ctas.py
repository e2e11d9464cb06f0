"""CG launches of more CTAs than read each other's sums directly (296): a shape the
caller sets, on meshes with more and with fewer slices than CTAs, and a batch whose
instances lie on both sides of that number, against one CTA per SM; a wait that
never ends in the sums of sums."""
import numpy as np
import pytest

from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Batch, Monodomain

pytestmark = pytest.mark.gpu
D = M.sigma_to_D(1.2, 0.2)
# the launches take the same iterates; their sums differ in order only
TOL = {capi.FP64: 1e-12, capi.FP32: 1e-6}


def _slab(*dims):
    return M.slab(*dims, *(0.02 * (k - 1) for k in dims))


def _voltage(m, seed):
    rng = np.random.default_rng(seed)
    return -85.0 + 120.0 * (m.xyz[:, 0] < m.xyz[:, 0].mean()) + rng.normal(0, 1.0, m.n)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("cfg", [dict(cg_block=128, cg_per_sm=8), dict(cg_block=128, cg_per_sm=3),
                                 dict(cg_block=256, cg_per_sm=4), dict(cg_block=256, cg_per_sm=3, cg_batch=8),
                                 dict(cg_block=128, cg_per_sm=5, cg_batch=16)])
@pytest.mark.parametrize("dims", [(5, 4, 3), (41, 31, 9)])
def test_many_ctas_equal_one_per_sm(gpu, prec, cfg, dims):
    m = _slab(*dims)
    out = []
    for c in (cfg, dict(cg_per_sm=1)):
        g = Monodomain(m, capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02, D=D, cg_tol=1e-7)
        g.set_launch_config(**c)
        g.set_voltage(_voltage(m, 5))
        it = [g.diffusion_half_step()[0] for _ in range(3)]
        out.append((it, g.voltage()))
        g.close()
    assert out[0][0] == out[1][0] and out[0][0][0] > 1
    assert np.max(np.abs(out[0][1] - out[1][1])) <= TOL[prec] * np.max(np.abs(out[1][1]))


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
def test_batch_groups_of_few_and_many_ctas(gpu, prec):
    meshes = [_slab(41, 31, 9), _slab(9, 7, 5), _slab(31, 21, 9)]
    V = [_voltage(m, k) for k, m in enumerate(meshes)]
    out = []
    for c in (dict(cg_block=128, cg_per_sm=8), dict(cg_per_sm=1)):
        b = Batch([dict(mesh=m, D=D) for m in meshes], capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02)
        b.set_launch_config(**c)
        b.set_voltage(np.concatenate(V))
        b.diffusion_half_step()
        out.append(b.voltage())
        b.close()
    assert np.max(np.abs(out[0] - out[1])) <= TOL[prec] * np.max(np.abs(out[1]))


def test_a_wait_that_gives_up_leaves_the_handle_usable(gpu):
    m = _slab(21, 17, 5)
    V = _voltage(m, 2)
    g = Monodomain(m, capi.TUSSCHER, capi.FP32, dt=0.1, ionic_dt=0.02, D=D)
    g.set_launch_config(cg_block=128, cg_per_sm=8)
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
