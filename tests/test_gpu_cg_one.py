"""Small meshes are solved on one CTA (k_cn_one) up to 64 slices of 32 rows: at
the edges of its forms (slices per warp) and of its range, against a set launch
of the general kernel, with and without the predictors; rows too wide for one
SM's shared memory, and just past the range the ring kernel with wide rows."""
import numpy as np
import pytest
import torch

from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Batch, Monodomain

pytestmark = pytest.mark.gpu
D = M.sigma_to_D(1.2, 0.2)
# the launches take the same iterates; their sums differ in order only
TOL = {capi.FP64: 1e-12, capi.FP32: 1e-6}


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("predict", [0, 1, 2])
@pytest.mark.parametrize("dims", [(3, 2, 2), (4, 4, 2), (8, 8, 6), (11, 7, 5), (16, 8, 8), (15, 14, 5), (16, 16, 6),
                                  (17, 13, 7), (32, 16, 4), (19, 18, 6)])
def test_one_cta_equals_a_set_launch(gpu, prec, predict, dims):
    m = M.slab(*dims, *(0.02 * (k - 1) for k in dims))
    rng = np.random.default_rng(m.n)
    V = -85.0 + 120.0 * (m.xyz[:, 0] < m.xyz[:, 0].mean()) + rng.normal(0, 1.0, m.n)
    out = []
    for per_sm in (0, 1):
        g = Monodomain(m, capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02, D=D, cg_tol=1e-7)
        g.set_launch_config(cg_per_sm=per_sm, cg_predict=predict)
        g.set_voltage(V)
        it = [g.diffusion_half_step()[0] for _ in range(3)]
        out.append((it, g.voltage()))
        g.close()
    assert out[0][0] == out[1][0] and out[0][0][0] > 1
    assert np.max(np.abs(out[0][1] - out[1][1])) <= TOL[prec] * np.max(np.abs(V))


@pytest.mark.parametrize("prec,ty", [(capi.FP64, np.float64), (capi.FP32, np.float32)])
@pytest.mark.parametrize("n,wide", [(33, 8), (700, 130), (2117, 24)])
def test_wide_rows(gpu, prec, ty, n, wide):
    """Symmetric systems with scattered neighbours through the allocation-free
    entry, whose launch is chosen before the widths are known: small, wider than
    one SM holds, and past one CTA's range (a ring of wide slices)."""
    S = 32
    rng = np.random.default_rng(n)
    A = np.zeros((n, n))
    for i in range(n):
        j = (i + rng.choice(np.arange(1, n), wide // 2, replace=False)) % n
        A[i, j] = A[j, i] = -rng.uniform(0.0, 1.0, len(j))
    np.fill_diagonal(A, np.abs(A).sum(1) * 1.3 + 0.1)
    B = 2.0 * np.diag(np.diag(A)) - A
    ns = (n + S - 1) // S
    ptr, col, av, bv = [0], [], [], []
    for s in range(ns):
        rows = range(S * s, min(n, S * s + S))
        w = max(np.count_nonzero(A[r]) for r in rows)
        c, a, b = np.zeros((w, S), np.int32), np.zeros((w, S)), np.zeros((w, S))
        for r in rows:
            j = np.flatnonzero(A[r])
            c[:len(j), r - S * s], a[:len(j), r - S * s], b[:len(j), r - S * s] = j, A[r, j], B[r, j]
        ptr.append(ptr[-1] + w * S)
        col.append(c), av.append(a), bv.append(b)
    cat = lambda v, t: np.concatenate([k.ravel() for k in v]).astype(t)  # noqa: E731
    x0 = rng.normal(0, 30.0, n).astype(ty)
    arrays = [torch.from_numpy(v).cuda() for v in (np.array(ptr, np.int32), cat(col, np.int32), cat(av, ty), cat(bv, ty),
                                                   (1 / np.diag(A)).astype(ty), x0)]
    capi.check(capi.lib().ep_cn_half_step_noalloc(prec, n, ns, *(t.data_ptr() for t in arrays), 1e-12, 500, None, None,
                                                  None))
    ref = np.linalg.solve(A.astype(ty).astype(np.float64), B.astype(ty).astype(np.float64) @ x0)
    # relative residual 1e-12 (FP32: the resolution 1.2e-7) times the condition
    # number, below 10 for these three, and FP32's rounding of the same size
    tol = 1e-10 if prec == capi.FP64 else 1e-5
    assert np.linalg.norm(arrays[-1].cpu().numpy() - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("count", [2, 37, 38])
def test_batches_of_few_and_many_instances(gpu, prec, count):
    """Batches at the edge between one and two CTAs per SM (a quarter as many
    instances as 148 SMs), uneven instances: each as on its own."""
    dims = [(5 + k % 7, 4 + k % 5, 4) for k in range(count)]
    dims[0] = (41, 31, 9)
    meshes = [M.slab(*d, *(0.02 * (k - 1) for k in d)) for d in dims]
    rng = np.random.default_rng(count)
    V = [-85.0 + 120.0 * (m.xyz[:, 0] < m.xyz[:, 0].mean()) + rng.normal(0, 1.0, m.n) for m in meshes]
    b = Batch([dict(mesh=m, D=D) for m in meshes], capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02)
    b.set_voltage(np.concatenate(V))
    b.diffusion_half_step()
    got = b.split(b.voltage())
    b.close()
    for k in (0, 1, count - 1):
        g = Monodomain(meshes[k], capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02, D=D)
        g.set_launch_config(cg_per_sm=1)
        g.set_voltage(V[k])
        g.diffusion_half_step()
        assert np.max(np.abs(g.voltage() - got[k])) <= TOL[prec] * np.max(np.abs(V[k]))
        g.close()
