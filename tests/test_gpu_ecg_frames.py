"""The offline pseudo-ECG of many frames (ep_ecg_eval) against the oracle's weights times
the frames in NumPy: every form of the kernel (1-4, 5-8 and 9-16 leads: 8, 4 and 2 frames
a CTA), partial last groups, one handle with growing and shrinking calls, uploads below and
above the pieces' sizes, and more frames than one launch takes groups of."""
import numpy as np
import pytest

from oracle import oracle as O
from ucla_cmg_b200 import mesh as M
from ucla_cmg_b200.compute_ecg import Ecg

pytestmark = pytest.mark.gpu
D = (1e-3, 5e-4, 2.5e-4)


def _case(dims, leads):
    m = M.slab(*dims, *(0.02 * (k - 1) for k in dims))
    el = M.fibonacci_sphere(leads, 3.0, m.xyz.mean(0))
    W = O.ecg_weights(m.xyz, m.tets, m.fibers, D, el)
    return m, el, W


def _check(ecg, W, V):
    got, ref = ecg(V), V @ W.T
    # FP64 sums of n products, in another order: n roundings of the absolute sum
    bound = 2.2e-16 * W.shape[1] * (np.abs(V) @ np.abs(W).T)
    assert got.shape == ref.shape and np.all(np.abs(got - ref) <= bound)


@pytest.mark.parametrize("leads", [1, 4, 5, 8, 9, 16])
def test_leads_and_frames(gpu, leads):
    m, el, W = _case((31, 23, 9), leads)
    rng = np.random.default_rng(leads)
    V = rng.normal(-40.0, 30.0, (33, m.n))
    ecg = Ecg(m, el, D=D)
    for frames in (1, 2, 3, 9, 33, 8, 7, 1, 33):
        _check(ecg, W, V[:frames])
    ecg.close()


@pytest.mark.parametrize("leads", [3, 12])
def test_large_uploads(gpu, leads):
    m, el, W = _case((51, 41, 11), leads)
    rng = np.random.default_rng(leads)
    V = rng.normal(-40.0, 30.0, (90, m.n))          # 16.5 MB
    ecg = Ecg(m, el, D=D)
    for frames in (1, 5, 6, 12, 90, 23, 90) + (90,) * 8:
        _check(ecg, W, V[:frames])
    ecg.close()


@pytest.mark.parametrize("leads,frames", [(9, 2 * 65535 + 5), (6, 4 * 65535 + 3), (2, 8 * 65535 + 9)])
def test_more_frames_than_a_launch_has_groups(gpu, leads, frames):
    m, el, W = _case((3, 2, 2), leads)
    rng = np.random.default_rng(leads)
    V = rng.normal(-40.0, 30.0, (frames, m.n))
    ecg = Ecg(m, el, D=D)
    _check(ecg, W, V)
    _check(ecg, W, V[:7])
    ecg.close()
