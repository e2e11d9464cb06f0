"""The trainer's products at the edges of their 64 x 64 tiles, 16-deep slices
and chunks of the batch: gradients against the FP64 numpy network."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from ucla_cmg_b200 import surrogate as SG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 33, 64, 2049])
@pytest.mark.parametrize("dims", [[1, 1], [23, 64, 19], [16, 65, 63, 7], [23, 128, 128, 128, 19]])
def test_gradients_at_tile_edges(gpu, dims, rows):
    import torch
    tr = SG.Trainer(dims, seed=3)
    p = tr.params().astype(np.float64)
    rng = np.random.default_rng(rows)
    X = rng.normal(size=(rows, dims[0])).astype(np.float32)
    Y = rng.normal(size=(rows, dims[-1])).astype(np.float32)
    Xd, Yd = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()
    loss, g = tr.loss_grad(Xd.data_ptr(), Yd.data_ptr(), rows, want_grad=True)
    out = torch.empty_like(Yd)
    tr.forward(Xd.data_ptr(), out.data_ptr(), rows)
    torch.cuda.synchronize()
    tr.close()
    lo, go = MO.loss_grad(p, dims, X.astype(np.float64), Y.astype(np.float64), np.ones(dims[-1]))
    fo, _ = MO.forward(p, dims, X.astype(np.float64))
    # FP32 products of up to 2049 terms: far below 1e-4 of the largest entry
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    assert np.max(np.abs(g - go)) <= 1e-4 * np.max(np.abs(go))
    assert np.max(np.abs(out.cpu().numpy() - fo)) <= 1e-5 * max(1.0, np.abs(fo).max())
