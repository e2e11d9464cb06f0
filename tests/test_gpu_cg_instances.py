"""Batches of more instances than the one-pass CG kernel has CTAs for in a launch shape:
each still runs, on the two-pass kernel's CTAs, and gives every instance the result of the
library's own launch."""
import numpy as np
import pytest

from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Batch

pytestmark = pytest.mark.gpu
D = M.sigma_to_D(1.2, 0.2)
# the kernels take the same iterates; recurrences and sums differ in rounding only
TOL = {capi.FP64: 1e-12, capi.FP32: 1e-6}


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("count,cfg", [(149, dict(cg_block=768, cg_per_sm=2)), (256, dict(cg_block=768, cg_per_sm=2)),
                                       (256, dict(cg_block=768, cg_per_sm=0))])
def test_every_instance_has_a_cta(gpu, prec, count, cfg):
    meshes = [M.slab(*d, *(0.02 * (k - 1) for k in d)) for d in ((3, 3, 3), (7, 5, 4))]
    b = Batch([dict(mesh=meshes[k % 7 == 3], D=D) for k in range(count)], capi.LUORUDY, prec, dt=0.1, ionic_dt=0.1)
    rng = np.random.default_rng(count)
    V = -85.0 + 100.0 * rng.random(b.n)
    out = []
    for c in ({}, cfg):
        b.set_launch_config(**c)
        b.set_voltage(V)
        b.diffusion_half_step()
        out.append((list(b.cg_last()[0]), b.voltage()))
    b.close()
    assert out[0][0] == out[1][0] and max(out[0][0]) > 1
    assert np.max(np.abs(out[0][1] - out[1][1])) <= TOL[prec] * np.max(np.abs(V))
