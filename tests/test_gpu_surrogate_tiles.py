"""The learned step's network at the edges of its tilings: one tile of 128 rows
per CTA up to one tile per SM, four tiles at once per CTA beyond, partial last
tiles and slots that have no tile.  A tile goes through the same instructions
wherever it runs, so every row has the bits that it has in a call of its own
tile, which test_gpu_mlp.py compares with the oracle."""
import numpy as np
import pytest
import torch

from ucla_cmg_b200 import surrogate as SG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,extra", [(0, 1), (1, -1), (1, 0), (1.0, 1), ("sms", -1), ("sms", 0), ("sms", 1),
                                         ("sms2", 77), ("sms4", 0), ("sms4", 1), ("sms9", -127)])
def test_rows_do_not_depend_on_the_tiling(gpu, tiles, extra):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = int(sms * int(tiles[3:] or 1) if isinstance(tiles, str) else tiles) * 128 + extra
    sg = SG.Surrogate.load()
    rng = np.random.default_rng(n)
    one = rng.standard_normal((3 * 128, 23)).astype(np.float32)
    X = np.resize(one, (n, 23))
    Y = sg.forward_kernel(X)
    ref = np.concatenate([sg.forward_kernel(one[128 * k:128 * k + 128]) for k in range(3)])
    assert np.array_equal(Y, np.resize(ref, Y.shape))
