"""The CG launches the library chooses by itself (k_cn_smem, or one CTA of
k_cn_half) at the edges of their ranges: one slice, the last size of one CTA
and the first of two, 256 and 512 threads, a matrix that stays in shared memory
and one that streams through its ring, slices wider than the ring, arrays that
bulk copies cannot read, and batches whose instances share slices."""
import numpy as np
import pytest

from ucla_cmg_b200 import capi, mesh as M
from ucla_cmg_b200.simulation import Batch, Monodomain

pytestmark = pytest.mark.gpu
D = M.sigma_to_D(1.2, 0.2)
# both launches take the same iterates; their sums differ in order only
TOL = {capi.FP64: 1e-12, capi.FP32: 1e-6}


def _voltage(m, seed):
    rng = np.random.default_rng(seed)
    return -85.0 + 120.0 * (m.xyz[:, 0] < m.xyz[:, 0].mean()) + rng.normal(0, 1.0, m.n)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("dims", [(4, 4, 2), (11, 3, 2), (16, 16, 4), (33, 8, 4), (61, 61, 11), (101, 101, 17)])
def test_library_choice_equals_a_set_launch(gpu, prec, dims):
    m = M.slab(*dims, *(0.02 * (k - 1) for k in dims))
    V = _voltage(m, 3)
    out = []
    for cfg in ({}, dict(cg_per_sm=1)):
        g = Monodomain(m, capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02, D=D, cg_tol=1e-7)
        g.set_launch_config(**cfg)
        assert g.launch_config()["cg_per_sm"] == cfg.get("cg_per_sm", 0)
        g.set_voltage(V)
        it = [g.diffusion_half_step()[0] for _ in range(2)]
        out.append((it, g.voltage()))
        g.close()
    assert out[0][0] == out[1][0] and out[0][0][0] > 3
    assert np.max(np.abs(out[0][1] - out[1][1])) <= TOL[prec] * np.max(np.abs(V))


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
def test_batch_instances_share_slices(gpu, prec):
    meshes = [M.slab(nx, ny, 4, 0.02 * (nx - 1), 0.02 * (ny - 1), 0.06) for nx, ny in ((13, 9), (21, 17), (3, 3))]
    V = np.concatenate([_voltage(m, k) for k, m in enumerate(meshes)])
    b = Batch([dict(mesh=m, D=D) for m in meshes], capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02)
    b.set_voltage(V)
    b.diffusion_half_step()
    got = b.split(b.voltage())
    b.close()
    for m, v, x in zip(meshes, np.split(V, np.cumsum([m.n for m in meshes])[:-1]), got):
        g = Monodomain(m, capi.TUSSCHER, prec, dt=0.1, ionic_dt=0.02, D=D)
        g.set_launch_config(cg_per_sm=1)
        g.set_voltage(v)
        g.diffusion_half_step()
        assert np.max(np.abs(g.voltage() - x)) <= TOL[prec] * np.max(np.abs(v))
        g.close()


@pytest.mark.parametrize("prec,ty", [(capi.FP64, np.float64), (capi.FP32, np.float32)])
@pytest.mark.parametrize("shift", [0, 1])
def test_wide_rows_and_unaligned_arrays(gpu, prec, ty, shift):
    """Rows of 32 to 56 columns (a ring of two units takes a slice in several
    rounds), 301 rows; shift 1 moves every array off its 16-byte boundary."""
    import torch
    n, S = 301, 32
    rng = np.random.default_rng(8)
    A = np.zeros((n, n))
    for i in range(n):
        j = (i + rng.choice(np.arange(1, n), 20 + i % 5, replace=False)) % n
        A[i, j] = A[j, i] = -rng.uniform(0.0, 1.0, len(j))
    A[np.arange(n), np.arange(n)] = 1.0 - A.sum(axis=1)
    B = np.diag(rng.uniform(0.5, 1.5, n))
    pat = A != 0
    ns = (n + S - 1) // S
    w = [int(pat[s * S:(s + 1) * S].sum(axis=1).max()) for s in range(ns)]
    sp = np.concatenate([[0], np.cumsum(np.array(w) * S)]).astype(np.int32)
    col, av, bv = np.zeros(sp[-1], np.int32), np.zeros(sp[-1], ty), np.zeros(sp[-1], ty)
    for i in range(n):
        c = np.flatnonzero(pat[i])
        at = sp[i // S] + np.arange(len(c)) * S + i % S
        col[at], av[at], bv[at] = c, A[i, c], B[i, c]
    x = rng.normal(0, 1.0, n)

    def dev(a):
        t = torch.zeros(len(a) + shift, dtype=torch.from_numpy(a).dtype, device="cuda")
        t[shift:] = torch.from_numpy(a).cuda()
        return t[shift:]
    arrays = [dev(a) for a in (sp, col, av, bv, (1.0 / np.diag(A)).astype(ty), x.astype(ty))]
    capi.check(capi.lib().ep_cn_half_step_noalloc(prec, n, ns, *(t.data_ptr() for t in arrays), 1e-10, 1000, None, None,
                                                  None))
    ref = np.linalg.solve(A.astype(ty).astype(np.float64), B.astype(ty).astype(np.float64) @ x.astype(ty))
    # relative residual 1e-10 (FP32: the resolution 1.2e-7) times the condition number, below 50
    tol = 5e-9 if prec == capi.FP64 else 6e-6
    assert np.linalg.norm(arrays[-1].cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
