"""What users of this framework have it do, as calls that can be timed.

Five kinds of work, each through its public entry point:

* ``tissue``  -- a running simulation advanced by a number of global steps and
  its voltage read back (``Monodomain.step`` / ``Batch.step`` + ``voltage``):
  the time loop of every driver run.  The state starts as a travelling wave
  and goes on from pass to pass, as a run does between two output frames.
* ``half``    -- one Crank-Nicolson half diffusion step of a host that owns its
  device memory (``ep_cn_half_step_noalloc``).
* ``cells``   -- the ionic phase of independent cells, the targets that the
  learned step's training data are made of (``ionic_phase_targets``).
* ``ecg``     -- the pseudo-ECG of stored voltage frames (``compute_ecg.Ecg``).
* ``train``   -- one optimiser step of the learned step's network (``Trainer``).

Sizes are those of the repository's workloads, tests and benchmark: slabs of a
few hundred to some 200,000 nodes, the ellipsoid shell at several spacings,
batches of uneven slabs.  Values of FP32 handles come back as FP32: the API
widens them to FP64 without changing them.

The exact values are computed here in 64 bits from the model equations (ten
Tusscher 2006 and Mahajan 2008 as the reference writes them), the linear-tet
matrices and a conjugate-gradient solve taken to rounding; the learned step has
none, since its network is defined by its own arithmetic.
"""
import functools
import math

import numpy as np
import torch

from ucla_cmg_b200 import capi, mesh as M, surrogate as SG
from ucla_cmg_b200.compute_ecg import Ecg
from ucla_cmg_b200.simulation import Batch, Monodomain, assemble_operators

H = 0.02                                  # node spacing of the slabs, cm
D = M.sigma_to_D(1.2, 0.2)                # cm^2/ms
PRECISION = {"fp64": capi.FP64, "fp32": capi.FP32, "learned": capi.SURROGATE}
XI = {"tt": 2000.0, "mahajan": 1.55e-4 / 2.58e-8}
ELECTRODES = 3.0 * np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0],
                             [0, 1, 1], [1, 0, 1], [-1, 1, 1]], dtype=np.float64)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # Solve() called once per step on a test-sized slab: launches and latency
        dict(name="tissue_tt_fp64_tiny", kind="tissue", model="tt", precision="fp64", nx=13, ny=11, nz=5, steps=1),
        # an odd slab in the parity precision up to a checkpoint: the voltage and every cell state come back
        dict(name="tissue_tt_fp64_odd", kind="tissue", model="tt", precision="fp64", nx=37, ny=43, nz=9, steps=20,
             states=True),
        # the 1 x 1 x 0.2 cm slab over one ECG sample interval (1 ms)
        dict(name="tissue_tt_fp32_slab", kind="tissue", model="tt", precision="fp32", nx=51, ny=51, nz=11, steps=50),
        # a quarter of the 4 x 4 x 0.4 cm Mahajan slab
        dict(name="tissue_mahajan_fp32", kind="tissue", model="mahajan", precision="fp32", nx=101, ny=101, nz=21,
             steps=20),
        # the ventricular shell, plain FP32, 0.1 ms steps of five ionic sub-steps
        dict(name="tissue_shell_fp32", kind="tissue", model="tt", precision="fp32", shell=0.073, layers=10, steps=10),
        # the shell with the learned ionic step, the largest tissue here
        dict(name="tissue_shell_learned", kind="tissue", model="tt", precision="learned", shell=0.05, layers=14,
             steps=10),
        # uneven slabs advanced together (parameter studies)
        dict(name="batch_tt_fp32", kind="tissue", model="tt", precision="fp32", batch=24, steps=20),
        # half diffusion steps inside another code's memory: small FP64, large FP32
        dict(name="half_fp64", kind="half", precision="fp64", nx=41, ny=29, nz=11, dt=0.02),
        dict(name="half_fp32_large", kind="half", precision="fp32", nx=127, ny=101, nz=17, dt=0.1),
        # training targets for one snapshot of a slab
        dict(name="cells_tt_fp64", kind="cells", precision="fp64", n=12001),
        # post-processing of a stored run: 100 frames, six leads
        dict(name="ecg_frames", kind="ecg", nx=51, ny=51, nz=11, frames=100, leads=6),
        # one minibatch of the learned step's training
        dict(name="train_step", kind="train", rows=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _slab_dims(rng, lo, hi):
    """Slab shape of about n nodes, n spread over [lo, hi] logarithmically."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nz = rng.randint(4, 21) if n > 4000 else rng.randint(4, 7)
    nx = max(5, int(round(math.sqrt(n / nz) * rng.uniform(0.7, 1.4))))
    ny = max(5, int(round(n / nz / nx)))
    return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choice(["tissue"] * 6 + ["shell"] * 3 + ["batch", "half", "half", "cells", "ecg", "train"])
    if kind == "tissue":
        model = rng.choice(["tt", "tt", "mahajan"])
        d = _slab_dims(rng, 400, 200000)
        small = d["nx"] * d["ny"] * d["nz"] < 40000
        return dict(kind="tissue", model=model, precision=rng.choice(["fp32", "fp64"]), **d,
                    steps=rng.randint(1, 50) if small else rng.randint(1, 10), states=small and rng.random() < 0.5)
    if kind == "shell":
        return dict(kind="tissue", model="tt", precision=rng.choice(["learned", "learned", "fp32", "fp64"]),
                    shell=round(rng.uniform(0.08, 0.2), 4), layers=rng.randint(5, 12), steps=rng.randint(1, 10))
    if kind == "batch":
        return dict(kind="tissue", model="tt", precision=rng.choice(["fp32", "fp64"]), batch=rng.randint(2, 24),
                    steps=rng.randint(2, 20))
    if kind == "half":
        return dict(kind="half", precision=rng.choice(["fp64", "fp32"]), **_slab_dims(rng, 400, 240000),
                    dt=rng.choice([0.01, 0.02, 0.05, 0.1]))
    if kind == "cells":
        return dict(kind="cells", precision=rng.choice(["fp64", "fp64", "fp32"]), n=_log_int(rng, 100, 60000))
    if kind == "ecg":
        return dict(kind="ecg", **_slab_dims(rng, 2000, 100000), frames=rng.randint(1, 64), leads=rng.randint(1, 10))
    return dict(kind="train", rows=_log_int(rng, 512, 65536))


# ------------------------------------------------------------- the geometry
@functools.lru_cache(maxsize=6)
def _slab(nx, ny, nz):
    return M.slab(nx, ny, nz, (nx - 1) * H, (ny - 1) * H, (nz - 1) * H)


@functools.lru_cache(maxsize=2)
def _shell(h, layers):
    return M.shell(h=h, n_rho=layers)


def _mesh(case):
    return _shell(case["shell"], case["layers"]) if "shell" in case else _slab(case["nx"], case["ny"], case["nz"])


def _batch_dims(k):
    """Uneven slab shapes, 21 x 21 x 6 up to 71 x 71 x 11."""
    return [(21 + (7 * i) % 51, 21 + (13 * i + 5) % 51, 6 + (5 * i) % 6) for i in range(k)]


def _steps_of(case):
    """(dt, ionic dt) of a tissue case: the shell's 0.1 / 0.02 ms, the slabs' 0.02 (ten Tusscher) and 0.01 ms."""
    return (0.1, 0.02) if "shell" in case else (0.01, 0.01) if case["model"] == "mahajan" else (0.02, 0.02)


def _cell_maps(case, mesh):
    """Transmural parameter sets and the apicobasal G_Ks scale of the shell; one set elsewhere."""
    if "shell" not in case:
        return None, None, None
    rho = mesh.meta["rho"]
    return (np.where(rho < 0.4, 0, np.where(rho < 0.7, 1, 2)).astype(np.uint8), TT_SETS,
            0.8 + 0.4 * mesh.meta["height"])


# --------------------------------------------- the cell models, in 64 bits
def _exp(x):
    return math.exp(x) if isinstance(x, float) else torch.exp(x)


def _log(x):
    return math.log(x) if isinstance(x, float) else torch.log(x)


def _sqrt(x):
    return math.sqrt(x) if isinstance(x, float) else torch.sqrt(x)


def _sel(c, a, b):
    return (a if c else b) if isinstance(c, bool) else torch.where(c, *(
        v if isinstance(v, torch.Tensor) else torch.full_like(b if isinstance(b, torch.Tensor) else a, v)
        for v in (a, b)))


def _sig(x):
    return 1.0 / (1.0 + _exp(x))


# ten Tusscher 2006, the reference's epicardial set; [15] G_Ks, [20] G_to, [53] the endocardial s gate
TT_EPI = np.array([
    8314.472, 310.0, 96485.3415, 0.185, 0.016404, 10.0, 1000.0, 1.0, 52.0, 0.03, 5.4, 140.0, 2.0, 5.405, 0.153, 0.392,
    14.838, 0.00029, 3.98e-05, 0.000592, 0.294, 2.724, 1.0, 40.0, 1000.0, 0.1, 2.5, 0.35, 1.38, 87.5, 0.1238, 0.0005,
    0.0146, 0.15, 0.045, 0.06, 0.005, 1.5, 2.5, 1.0, 0.102, 0.0038, 0.00025, 0.00036, 0.006375, 0.2, 0.001, 10.0, 0.3,
    0.4, 0.00025, 0.001094, 5.468e-05, 0.0])
TT_ENDO, TT_MID = TT_EPI.copy(), TT_EPI.copy()
TT_ENDO[20], TT_ENDO[53] = 0.073, 1.0
TT_MID[15] = 0.098
TT_SETS = np.stack([TT_ENDO, TT_MID, TT_EPI])
TT_REST = [-85.423, 136.89, 8.604, 0.000126, 0.00621, 0.4712, 0.0095, 0.00172, 0.7444, 0.7045, 0.00036, 3.373e-5, 0.7888,
           0.9755, 0.9953, 0.999998, 2.42e-8, 3.64, 0.9073]
TT_GATES = (4, 5, 6, 7, 8, 9, 11, 12, 13, 14, 15, 16)     # Xr1 Xr2 Xs m h j d f f2 fCass s r
TT_CONC = (1, 2, 3, 10, 17, 18)                           # Ki Nai Cai Cass CaSR R'


def _tt_gates(V, Cass, endo):
    """(steady state, time constant) of the twelve gates."""
    g = [(_sig((-26 - V) / 7), 450 * _sig((-45 - V) / 10) * 6 * _sig((V + 30) / 11.5)),
         (_sig((V + 88) / 24), 3 * _sig((-60 - V) / 20) * 1.12 * _sig((V - 60) / 20)),
         (_sig((-5 - V) / 14), 1400 / _sqrt(1 + _exp((5 - V) / 6)) * _sig((V - 35) / 15) + 80),
         (_sig((-56.86 - V) / 9.03) ** 2,
          _sig((-60 - V) / 5) * (0.1 * _sig((V + 35) / 5) + 0.1 * _sig((V - 50) / 200)))]
    lo = V < -40
    inf = _sig((V + 71.55) / 7.43) ** 2
    ah = _sel(lo, 0.057 * _exp(-(V + 80) / 6.8), 0.0)
    bh = _sel(lo, 2.7 * _exp(0.079 * V) + 3.1e5 * _exp(0.3485 * V), 0.77 / 0.13 * _sig((V + 10.66) / -11.1))
    aj = _sel(lo, (-25428 * _exp(0.2444 * V) - 6.948e-6 * _exp(-0.04391 * V)) * (V + 37.78) * _sig(0.311 * (V + 79.23)),
              0.0)
    bj = _sel(lo, 0.02424 * _exp(-0.01052 * V) * _sig(-0.1378 * (V + 40.14)),
              0.6 * _exp(0.057 * V) * _sig(-0.1 * (V + 32)))
    g += [(inf, 1 / (ah + bh)), (inf, 1 / (aj + bj)),
          (_sig((-8 - V) / 7.5), (1.4 * _sig((-35 - V) / 13) + 0.25) * 1.4 * _sig((V + 5) / 5) + _sig((50 - V) / 20)),
          (_sig((V + 20) / 7), 1102.5 * _exp(-(V + 27) ** 2 / 225) + 200 * _sig((13 - V) / 10)
           + 180 * _sig((V + 30) / 10) + 20),
          (0.67 * _sig((V + 35) / 7) + 0.33, 562 * _exp(-(V + 27) ** 2 / 240) + 31 * _sig((25 - V) / 10)
           + 80 * _sig((V + 30) / 10))]
    q = 1 / (1 + (Cass / 0.05) ** 2)
    g += [(0.6 * q + 0.4, 80 * q + 2),
          (_sel(endo, _sig((V + 28) / 5), _sig((V + 20) / 5)),
           _sel(endo, 1000 * _exp(-(V + 67) ** 2 / 1000) + 8,
                85 * _exp(-(V + 45) ** 2 / 320) + 5 * _sig((V - 20) / 5) + 3)),
          (_sig((20 - V) / 6), 9.5 * _exp(-(V + 40) ** 2 / 1800) + 0.8)]
    return g


def _tt_rates(V, s, x, ist, gks, gto):
    """dV/dt and the rates of (Ki, Nai, Cai, Cass, CaSR, R') = x; s: the 19 reference states (gates are read)."""
    c = [float(v) for v in TT_EPI]
    Ki, Nai, Cai, Cass, Casr, Rp = x
    RT, F = c[0] * c[1], c[2]
    ENa, EK = RT / F * _log(c[11] / Nai), RT / F * _log(c[10] / Ki)
    EKs = RT / F * _log((c[10] + c[9] * c[11]) / (Ki + c[9] * Nai))
    ECa = 0.5 * RT / F * _log(c[12] / Cai)
    vk = V - EK
    a = 0.1 * _sig(0.06 * (vk - 200))
    b = (3 * _exp(0.0002 * (vk + 100)) + _exp(0.1 * (vk - 10))) * _sig(-0.5 * vk)
    sq = math.sqrt(c[10] / 5.4)
    i_k1 = c[13] * a / (a + b) * sq * vk
    i_to = gto * s[16] * s[15] * vk
    i_kr = c[14] * sq * s[4] * s[5] * vk
    i_ks = gks * s[6] ** 2 * (V - EKs)
    i_na = c[16] * s[7] ** 3 * s[8] * s[9] * (V - ENa)
    i_bna = c[17] * (V - ENa)
    i_nak = c[21] * c[10] / (c[10] + c[22]) * Nai / (Nai + c[23]) / (
        1 + 0.1245 * _exp(-0.1 * V * F / RT) + 0.0353 * _exp(-V * F / RT))
    e, e1 = _exp(c[27] * V * F / RT), _exp((c[27] - 1) * V * F / RT)
    i_naca = c[24] * (e * Nai ** 3 * c[12] - e1 * c[11] ** 3 * Cai * c[26]) / (
        (c[29] ** 3 + c[11] ** 3) * (c[28] + c[12]) * (1 + c[25] * e1))
    u = 2 * (V - 15) * F / RT
    ghk = _sel(abs(u) < 1e-6, 1 - 0.5 * u, u / (_exp(u) - 1 + (u == 0) * 1.0))       # u / (e^u - 1)
    i_cal = c[18] * s[11] * s[12] * s[13] * s[14] * 2 * F * ghk * (0.25 * Cass * _exp(u) - c[12])
    i_bca = c[19] * (V - ECa)
    i_pk = c[32] * vk * _sig((25 - V) / 5.98)
    i_pca = c[30] * Cai / (Cai + c[31])
    dV = -(i_k1 + i_to + i_kr + i_ks + i_cal + i_nak + i_na + i_bna + i_naca + i_bca + i_pk + i_pca + ist)
    cap = c[3] / (c[4] * F)
    up = c[44] / (1 + c[42] ** 2 / Cai ** 2)
    leak, xfer = c[43] * (Casr - Cai), c[41] * (Cass - Cai)
    kcasr = c[38] - (c[38] - c[39]) / (1 + (c[37] / Casr) ** 2)
    k1 = c[33] / kcasr * Cass ** 2
    rel = c[40] * k1 * Rp / (c[35] + k1) * (Casr - Cass)
    return dV, [-(i_k1 + i_to + i_kr + i_ks + i_pk + ist - 2 * i_nak) * cap,
                -(i_na + i_bna + 3 * i_nak + 3 * i_naca) * cap,
                ((leak - up) * c[51] / c[4] + xfer - (i_bca + i_pca - 2 * i_naca) * cap / 2)
                / (1 + c[45] * c[46] / (Cai + c[46]) ** 2),
                (-i_cal * c[3] / (2 * c[52] * F) + rel * c[51] / c[52] - xfer * c[4] / c[52])
                / (1 + c[49] * c[50] / (Cass + c[50]) ** 2),
                (up - rel - leak) / (1 + c[47] * c[48] / (Casr + c[48]) ** 2),
                -c[34] * kcasr * Cass * Rp + c[36] * (1 - Rp)]


def _tt_compute(V, s, ist, h, gks, gto, endo):
    """One Compute_Ion call on columns s[1..18] (in place): semi-implicit gates, then the implicit Euler step of the six
    concentrations by Newton to rounding.  Returns dV/dt."""
    for k, (inf, tau) in zip(TT_GATES, _tt_gates(V, s[10], endo)):
        s[k] = (s[k] + h * inf / tau) / (1 + h / tau)
    x0 = torch.stack([s[k] for k in TT_CONC])
    x = x0.clone()
    rates = lambda y: torch.stack(_tt_rates(V, s, list(y), ist, gks, gto)[1])  # noqa: E731
    for _ in range(6):
        cols = []
        for i in range(6):
            d = 1e-4 * x[i]
            up, dn = x.clone(), x.clone()
            up[i] += d
            dn[i] -= d
            cols.append((up - dn - h * (rates(up) - rates(dn))) / (up[i] - dn[i]))
        J = torch.stack(cols, 1).permute(2, 0, 1)                     # [node, equation, unknown]
        x = x - torch.linalg.solve(J, (x - x0 - h * rates(x)).T.unsqueeze(2)).squeeze(2).T
    for i, k in enumerate(TT_CONC):
        s[k] = x[i]
    return _tt_rates(V, s, list(x), ist, gks, gto)[0]


MH_REST = [-81.4359, 0.002789, 0.96679, 0.97859, 0.014994, 0.044487, 0.091992, 2.1933, 0.23277, 0.24868, 101.6418, 95.4278,
           0.009495, 3.7e-005, 0.96094, 0.003718, 6.7e-005, 0.010571, 0.024659, 11.5909, 0.00533, 0.99047, 0.005333,
           0.17488, 21.5955, 20.0206]
_NAO, _KI, _KO, _CAO = 136.0, 140.0, 5.4, 1.8
_FRT = 96.485 / (8.314 * 308.0)


def _mh_rates(s, h, ist):
    """Rates of the 26 Mahajan states, s[0] = V (the reference's first parameter set)."""
    V, r, E = s[0], [None] * 26, _exp
    relax = lambda inf, tau, k: (inf - (inf - s[k]) * E(-h / tau) - s[k]) / h  # noqa: E731
    w = V - _log((100 * _KO + _NAO) / (100 * _KI + s[19])) / _FRT
    ak = 1.02 * _sig(0.2385 * (w - 59.215))
    bk = (0.49124 * E(0.08032 * (w + 5.476)) + E(0.06175 * (w - 594.31))) * _sig(-0.5143 * (w + 4.753))
    xik1 = 0.3 * ak / (ak + bk) * w
    vk = V - math.log(_KO / _KI) / _FRT
    xi, yi = _sig(-(V + 3) / 15), _sig((V + 33.5) / 10)
    xito = 0.04 * s[22] * (s[23] + 0.5 * yi) * vk + 0.11 * s[20] * s[21] * vk
    r[22] = relax(xi, 9 * _sig((V + 3) / 15) + 0.5, 22)
    r[23] = relax(yi, 3000 * _sig((V + 60) / 10) + 30, 23)
    r[20] = relax(xi, 3.5 * E(-(V / 30) ** 2) + 1.5, 20)
    r[21] = relax(yi, 20 * yi + 20, 21)
    sigma = (math.exp(_NAO / 67.3) - 1) / 7
    xinak = 1.5 / (1 + 0.1245 * E(-0.1 * V * _FRT) + 0.0365 * sigma * E(-V * _FRT)) / (1 + 12 / s[19]) * _KO / (_KO + 1.5)
    csm, na3, nao3, ez = s[8] / 1000, s[19] ** 3, _NAO ** 3, E(-0.65 * V * _FRT)
    jnaca = 0.84 / (1 + (0.3 / s[8]) ** 3) * (na3 * _CAO * E(0.35 * V * _FRT) - nao3 * csm * ez) / (1 + 0.2 * ez) / (
        1.3 * na3 + 669921.875 * csm + 1860.867 * _CAO * (1 + csm / 0.0036) + 0.0036 * nao3 * (1 + (s[19] / 12.3) ** 3)
        + na3 * _CAO + nao3 * csm)
    jd = (s[8] - s[9]) / 4
    r[24] = 0.0327 * s[9] * (70 - s[24]) - 0.0196 * s[24]
    r[25] = 0.0327 * s[8] * (70 - s[25]) - 0.0196 * s[25]
    jup = 0.4 * s[9] ** 2 / (s[9] ** 2 + 0.25)
    jleak = 0.00002069 * s[10] ** 2 / (s[10] ** 2 + 2500) * (s[10] * 16.667 - s[9])
    al = _sig(-V / 8)
    be = 1 - al
    fca = 1 / (1 + (3 / s[7]) ** 3)
    s1, s1t, k1, k2, k1t, k2t = 0.0182688 * fca, 0.00195, 0.024168 * fca, 1.03615e-4, 0.00413, 0.00224
    s2, s2t = s1 * 0.1 * k2 / k1, s1t * 0.1 * k2t / k1t
    k3 = (1 - _sig(-(V + 40) / 3)) / 3
    pr, ps = 1 - _sig(-(V + 40) / 4), _sig(-(V + 40) / 11.32)
    rec = 10 + 4954 * E(V / 15.6)
    tca = 78.0329 / (1 + (s[7] / 6.09365) ** 4) + 0.1
    tauca, tauba = (rec - tca) * pr + tca, (rec - 450) * pr + 450
    k6, k5, k6t, k5t = fca * ps / tauca, (1 - ps) / tauca, ps / tauba, (1 - ps) / tauba
    k4, k4t = k3 * (al / be) * (k1 / k2) * (k5 / k6), k3 * (al / be) * (k1t / k2t) * (k5t / k6t)
    po = 1 - s[15] - s[17] - s[16] - s[18] - s[13] - s[14]
    r[14] = be * s[13] + k5 * s[17] + k5t * s[18] - (k6 + k6t + al) * s[14]
    r[13] = al * s[14] + k2 * s[15] + k2t * s[16] + 3 * po - (be + 0.3 + k1t + k1) * s[13]
    r[15] = k1 * s[13] + k4 * s[17] + s1 * po - (k3 + k2 + s2) * s[15]
    r[17] = k3 * s[15] + k6 * s[14] - (k5 + k4) * s[17]
    r[16] = k1t * s[13] + k4t * s[18] + s1t * po - (k3 + k2t + s2t) * s[16]
    r[18] = k3 * s[16] + k6t * s[14] - (k5t + k4t) * s[18]
    za = 2 * V * _FRT
    f1 = 4 * 0.00054 * 96.485 ** 2 / (8.314 * 308.0)
    num = f1 * (csm * E(za) - 0.341 * _CAO)
    rxa = _sel(abs(za) < 0.001, num / (2 * _FRT), V * num / (E(za) - 1 + (za == 0) * 1.0))
    jca = 182 * po * rxa
    buf = lambda c: 1 / (1 + 168 / (7 + c) ** 2 + 28.2 / (0.6 + c) ** 2 + 4.5 / (0.3 + c) ** 2  # noqa: E731
                         + 546 / (13 + c) ** 2)
    r[8] = buf(s[8]) * (50 * (s[12] - jd - jca + jnaca) - r[25])
    r[9] = buf(s[9]) * (jd - jup + jleak - r[24])
    r[10] = -s[12] + jup - jleak
    r[11] = (s[10] - s[11]) / 100
    q = _sel(s[11] >= 90.0, 11.3 * s[11] + 40 - 11.3 * 90, _sel(s[11] > 50.0, s[11] - 50, 0.0 * s[11]))
    Qr = s[10] * _sel(q >= 153.0, 153.0, q) / 90
    ar = abs(rxa)
    r[12] = 2.58079 * po * ar * _sig(0.05 * (V + 30)) * Qr - s[12] * (1 - 30 * r[10] / s[10]) / 30
    r[7] = po * Qr * ar * 26841.8 * _sig(0.3576 * (V + 30)) + po * 9000 * ar - (s[7] - s[8]) / 0.5
    vm = V + 47.13
    am = _sel(abs(vm) > 0.001, 0.32 * vm / (1 - E(-0.1 * vm) + (vm == 0) * 1.0), 3.2)
    bm = 0.08 * E(-V / 11)
    a = 1 - _sig(-(V + 40) / 0.24)
    ah = a * 0.135 * E((80 + V) / -6.8)
    bh = (1 - a) / (0.13 * (1 + E((V + 10.66) / -11.1))) + a * (3.56 * E(0.079 * V) + 3.1e5 * E(0.35 * V))
    aj = a * (-1.2714e5 * E(0.2444 * V) - 3.474e-5 * E(-0.04391 * V)) * (V + 37.78) * _sig(0.311 * (V + 79.23))
    bj = (1 - a) * 0.3 * E(-2.535e-7 * V) * _sig(-0.1 * (V + 32)) + a * 0.1212 * E(-0.01052 * V) * _sig(-0.1378 * (V + 40.14))
    xina = 12 * s[2] * s[3] * s[1] ** 3 * (V - _log(_NAO / s[19]) / _FRT)
    for k, (x, y) in ((1, (am, bm)), (2, (ah, bh)), (3, (aj, bj))):
        r[k] = relax(x / (x + y), 1 / (x + y), k)
    v1 = _sel(abs(V + 7) > 0.001, 0.00138 * (V + 7) / (1 - E(-0.123 * (V + 7)) + (V == -7) * 1.0), 0.00138 / 0.123)
    v2 = _sel(abs(V + 10) > 0.001, 0.00061 * (V + 10) / (E(0.145 * (V + 10)) - 1 + (V == -10) * 1.0), 0.00061 / 0.145)
    xikr = 0.0125 * s[4] * _sig((V + 33) / 22.4) * vk
    r[4] = relax(_sig(-(V + 50) / 7.5), 1 / (v1 + v2), 4)
    v3 = V + 30
    t1 = _sel(abs(v3) < 0.001 / 0.0687, 1 / (0.0000719 / 0.148 + 0.000131 / 0.0687),
              1 / (0.0000719 * v3 / (1 - E(-0.148 * v3) + (v3 == 0) * 1.0)
                   + 0.000131 * v3 / (E(0.0687 * v3) - 1 + (v3 == 0) * 1.0)))
    xs = _sig(-(V - 1.5) / 16.7)
    xiks = 0.608 * (1 + 0.8 / (1 + (0.5 / s[9]) ** 3)) * s[5] * s[6] * (
        V - _log((_KO + 0.01833 * _NAO) / (_KI + 0.01833 * s[19])) / _FRT)
    r[5], r[6] = relax(xs, t1, 5), relax(xs, 4 * t1, 6)
    wca = 8.0313
    r[19] = -(xina + 3 * xinak + 3 * wca * jnaca) / (1000 * wca)
    r[0] = -(xina + xik1 + xikr + xiks + xito + wca * jnaca + 2 * wca * jca + xinak) + ist
    return r


def _mh_compute(V, s, ist, dt):
    """One Compute_Ion call (in place): a step of dt, or ten of dt/10 where dV/dt truncates to over 20."""
    s[0] = V
    r = _mh_rates(s, dt, ist)
    fast = abs(r[0]) >= 21.0
    one = [x + dt * y for x, y in zip(s, r)]
    last = r[0]
    if bool(fast.any()):
        t = list(s)
        for _ in range(10):
            q = _mh_rates(t, dt / 10, ist)
            t = [x + dt / 10 * y for x, y in zip(t, q)]
        one = [_sel(fast, a, b) for a, b in zip(t, one)]
        last = _sel(fast, q[0], last)
    s[:] = one
    return last


@functools.lru_cache(maxsize=2)
def _action_potential(model):
    """States of a single cell every 0.1 ms over an action potential, stimulated at the start."""
    rows = []
    if model == "tt":
        s = [float(v) for v in TT_REST]
        h, every = 0.02, 5
        for k in range(16000):
            if k % every == 0:
                rows.append(list(s))
            V, ist = s[0], -52.0 if k * h < 1.0 else 0.0
            for g, (inf, tau) in zip(TT_GATES, _tt_gates(V, s[10], False)):
                s[g] = (s[g] + h * inf / tau) / (1 + h / tau)
            dV, r = _tt_rates(V, s, [s[j] for j in TT_CONC], ist, 0.392, 0.294)
            for j, d in zip(TT_CONC, r):
                s[j] += h * d
            s[0] = V + h * dV
    else:
        s = [float(v) for v in MH_REST]
        for k in range(25000):
            if k % 10 == 0:
                rows.append(list(s))
            r = _mh_rates(s, 0.01, 50.0 if k < 100 else 0.0)
            s = [x + 0.01 * d for x, d in zip(s, r)]
    return np.array(rows)


def _wave(model, xyz, seed):
    """States (n, nstate) of a plane wave of seeded direction and speed with its front inside the tissue."""
    rng = np.random.default_rng(seed)
    ap = _action_potential(model)
    a, tilt = rng.uniform(0, 2 * np.pi), rng.uniform(-0.3, 0.3)
    u = xyz @ np.array([np.cos(a), np.sin(a), tilt])
    lo, hi = u.min(), u.max()
    t = (lo + rng.uniform(0.3, 0.5) * (hi - lo) - u) / rng.uniform(0.05, 0.07)        # ms since the front passed
    return np.ascontiguousarray(ap[np.clip((t / 0.1).astype(np.int64), 0, len(ap) - 1)])


# ----------------------------------------------------------------- prepare
def _sell(A, B):
    """SELL-32 arrays of two CSR matrices of one pattern: slices of 32 rows, column-major, padded with the row itself."""
    n, rp = A.shape[0], A.indptr.astype(np.int64)
    ns, ln = (n + 31) // 32, np.diff(rp)
    full = np.zeros(ns * 32, np.int64)
    full[:n] = ln
    sp = np.concatenate([[0], np.cumsum(full.reshape(ns, 32).max(axis=1) * 32)])
    pos = np.arange(sp[-1])
    sl = np.searchsorted(sp, pos, side="right") - 1
    col = np.minimum(sl * 32 + (pos - sp[sl]) % 32, n - 1).astype(np.int32)
    av, bv = np.zeros(sp[-1]), np.zeros(sp[-1])
    row = np.repeat(np.arange(n), ln)
    at = sp[row // 32] + (np.arange(rp[-1]) - rp[row]) * 32 + row % 32
    col[at], av[at], bv[at] = A.indices, A.data, B.data
    return ns, sp.astype(np.int32), col, av, bv, 1.0 / A.diagonal()


def _cells_inputs(case, seed):
    """Snapshots along an action potential inside the learned domain, as the training set keeps them."""
    rng = np.random.default_rng(seed)
    ap = _action_potential("tt")
    S = ap[rng.integers(30, len(ap), case["n"])]
    S[:, 1:] *= rng.uniform(0.999, 1.0, (case["n"], 18))
    return (np.ascontiguousarray(S), np.zeros(case["n"]), rng.integers(0, 3, case["n"]).astype(np.uint8), TT_SETS,
            rng.uniform(0.6, 1.4, case["n"]))


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    p = []
    for a, b in zip(SG.DIMS, SG.DIMS[1:]):
        p += [rng.uniform(-1, 1, a * b) * math.sqrt(6.0 / (a + b)), np.zeros(b)]
    X = rng.normal(size=(case["rows"], SG.DIMS[0]))
    Y = np.tanh(X[:, :19] + 0.5 * X[:, 4:23]) + 0.1 * rng.normal(size=(case["rows"], 19))
    w = np.zeros(19)
    w[list(SG.CONC_OUTPUTS)] = 1.0
    return np.concatenate(p).astype(np.float32), X.astype(np.float32), Y.astype(np.float32), w.astype(np.float32)


def _frames(case, seed):
    """Voltage frames 1 ms apart of a wave crossing the slab, host data as read from the files."""
    mesh, rng, ap = _mesh(case), np.random.default_rng(seed), _action_potential("tt")
    a = rng.uniform(0, 2 * np.pi)
    t0 = -(mesh.xyz @ np.array([np.cos(a), np.sin(a), 0.1])) / rng.uniform(0.05, 0.07)
    return np.stack([ap[np.clip(((t0 + f + 5.0) / 0.1).astype(np.int64), 0, len(ap) - 1), 0]
                     for f in range(case["frames"])])


def _batch_instances(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k, d in enumerate(_batch_dims(case["batch"])):
        c = TT_EPI.copy()
        c[15] *= rng.uniform(0.5, 1.5)
        c[20] *= rng.uniform(0.5, 1.5)
        out.append((M.slab(*d, *((v - 1) * H for v in d)), c, seed * 100 + k))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tissue" and "batch" in case:
        inst = _batch_instances(case, seed)
        g = Batch([dict(mesh=m, D=D, type_consts=c[None, :], n_types=1) for m, c, _ in inst], capi.TUSSCHER,
                  PRECISION[case["precision"]], dt=0.02, ionic_dt=0.02, tt_jacobian=capi.TT_JAC_TRUE)
        S = np.concatenate([_wave("tt", m.xyz, s) for m, _, s in inst])
    elif kind == "tissue":
        m = _mesh(case)
        dt, idt = _steps_of(case)
        node_type, sets, gks = _cell_maps(case, m)
        g = Monodomain(m, capi.TUSSCHER if case["model"] == "tt" else capi.MAHAJAN, PRECISION[case["precision"]], dt=dt,
                       ionic_dt=idt, D=D, node_type=node_type, type_consts=sets, gks_scale=gks,
                       tt_jacobian=capi.TT_JAC_TRUE, ecg_every=max(1, int(round(1.0 / dt))))
        if case["precision"] == "learned":
            SG.Surrogate.load().deploy(g)
        g.set_electrodes(ELECTRODES[:2] + m.xyz.mean(axis=0))
        ids, on, amp = _stimulus(case, m)
        g.set_stimulus(ids, on, on + 1.0, amp)
        S = _wave(case["model"], m.xyz, seed)
    elif kind == "half":
        m = _mesh(case)
        A, B, _ = assemble_operators(m, D, case["dt"])
        ns, sp, col, a, b, dinv = _sell(A, B)
        t = torch.float64 if case["precision"] == "fp64" else torch.float32
        dev = lambda v, ty: torch.from_numpy(v).to("cuda", ty)  # noqa: E731
        V = _wave("tt", m.xyz, seed)[:, 0]
        return dict(case, n=m.n, ns=ns, sp=dev(sp, torch.int32), col=dev(col, torch.int32), A=dev(a, t), B=dev(b, t),
                    dinv=dev(dinv, t), V=dev(np.ascontiguousarray(V), t), x=dev(np.zeros(m.n), t))
    elif kind == "cells":
        return dict(case, args=_cells_inputs(case, seed))
    elif kind == "ecg":
        m = _mesh(case)
        return dict(case, ecg=Ecg(m, ELECTRODES[:case["leads"]] + m.xyz.mean(axis=0)), frames=_frames(case, seed))
    else:
        p, X, Y, w = _train_inputs(case, seed)
        tr = SG.Trainer()
        tr.set_params(p)
        return dict(case, tr=tr, X=torch.from_numpy(X).cuda(), Y=torch.from_numpy(Y).cuda(), w=w)
    g.set_states(S)
    g.set_voltage(S[:, 0])
    return dict(case, g=g)


def _stimulus(case, m):
    """A corner of the tissue stimulated over the first millisecond (50 uA/cm^2)."""
    ids = np.where(np.linalg.norm(m.xyz - m.xyz[0], axis=1) <= 0.1)[0].astype(np.int32)
    return ids, np.zeros(len(ids)), np.full(len(ids), 50.0 * XI[case["model"]])


# --------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "tissue":
        g = state["g"]
        g.step(state["steps"])
        real = np.float64 if state["precision"] == "fp64" else np.float32
        v = g.voltage().astype(real, copy=False)
        return dict(V=v, states=g.states().astype(real, copy=False)) if state.get("states") else v
    if kind == "half":
        x = state["x"]
        x.copy_(state["V"])
        p = lambda k: state[k].data_ptr()  # noqa: E731
        capi.check(capi.lib().ep_cn_half_step_noalloc(
            PRECISION[state["precision"]], state["n"], state["ns"], p("sp"), p("col"), p("A"), p("B"), p("dinv"), p("x"),
            1e-7, 1000, torch.cuda.current_stream().cuda_stream, None, None))
        return x
    if kind == "cells":
        return SG.ionic_phase_targets(*state["args"], precision=PRECISION[state["precision"]],
                                      newton_tol=1e-12 if state["precision"] == "fp64" else 1e-6)
    if kind == "ecg":
        return state["ecg"](state["frames"])
    tr = state["tr"]
    loss, g = tr.loss_grad(state["X"].data_ptr(), state["Y"].data_ptr(), state["rows"], state["w"], want_grad=True)
    tr.adam(2e-5)                         # late on the cosine schedule
    return dict(loss=np.float32(loss), grad=g, params=tr.params())


# -------------------------------------------------------------------- work
def _tissue_counts(case):
    """(nodes, matrix entries, states, FLOPs of a node's ionic phase per global step)"""
    if "batch" in case:
        dims = _batch_dims(case["batch"])
        n = sum(a * b * c for a, b, c in dims)
    else:
        n = _mesh(case).n
    sub = 5 if "shell" in case else 1
    flops = 82000 if case["precision"] == "learned" else (2000 * sub if case["model"] == "tt" else 900)
    return n, 14 * n, (19 if case["model"] == "tt" else 26), flops


def work(case):
    kind = case["kind"]
    R = 8 if case.get("precision") == "fp64" else 4
    if kind == "tissue":
        n, nnz, ns, fl = _tissue_counts(case)
        # each step: both half steps read A, B and the columns and V once and write V; the states in and out
        by = 2 * (nnz * (2 * R + 4) + 2 * n * R) + 2 * n * ns * R
        return dict(bytes=case["steps"] * by, flops=case["steps"] * (n * fl + 2 * 6 * 2 * nnz))
    if kind == "half":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=14 * n * (2 * R + 4) + 3 * n * R, flops=6 * 2 * 14 * n)
    if kind == "cells":
        return dict(bytes=2 * case["n"] * 20 * 8, flops=case["n"] * 5 * 3000)
    if kind == "ecg":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=8 * n * (case["frames"] + case["leads"]), flops=2 * n * case["frames"] * case["leads"])
    wts = sum(a * b for a, b in zip(SG.DIMS, SG.DIMS[1:]))
    return dict(bytes=4 * (case["rows"] * 42 + 6 * wts), flops=6 * case["rows"] * wts)


# ------------------------------------------------- exact values, in 64 bits
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev())


_QA, _QB = 0.58541020, 0.13819660         # the reference's four-point rule


def _shape(q, a):
    """Shape function a at quadrature point q."""
    p = [_QB, _QB, _QB]
    if q < 3:
        p[q] = _QA
    return p[a - 1] if a else 1 - sum(p)


def _elements(m, De3):
    """Volumes, shape gradients (m, 4, 3) and diffusion tensors (m, 3, 3) of the tets."""
    x = _t(m.xyz)[_t(m.tets, torch.long)]
    T = (x[:, 1:] - x[:, :1]).transpose(1, 2)
    inv = torch.linalg.inv(T)
    dN = torch.cat([-inv.sum(1, keepdim=True), inv], 1)
    f = _t(m.fibers).reshape(-1, 3, 3)
    return x, torch.linalg.det(T) / 6, dN, torch.einsum("p,epa,epb->eab", _t(De3), f, f)


def _operators(m, dt):
    """A = M + dt/4 K, B = M - dt/4 K (sparse) and 1 / diag A."""
    _, vol, dN, De = _elements(m, D)
    K = torch.einsum("e,eai,eij,ebj->eab", vol, dN, De, dN)
    N = _t([[_shape(q, a) for a in range(4)] for q in range(4)])
    Mm = torch.einsum("e,ab->eab", vol / 4, N.T @ N)
    tets = _t(m.tets, torch.long)
    ij = torch.stack([tets[:, :, None].expand(-1, 4, 4).reshape(-1), tets[:, None, :].expand(-1, 4, 4).reshape(-1)])
    mk = lambda v: torch.sparse_coo_tensor(ij, v.reshape(-1), (m.n, m.n)).coalesce().to_sparse_csr()  # noqa: E731
    diag = torch.zeros(m.n, dtype=torch.float64, device=_dev())
    diag.index_add_(0, tets.reshape(-1), torch.diagonal(Mm + dt / 4 * K, dim1=1, dim2=2).reshape(-1))
    return mk(Mm + dt / 4 * K), mk(Mm - dt / 4 * K), 1 / diag


def _half(op, V):
    A, B, dinv = op
    b, x = B @ V, V.clone()
    r = b - A @ x
    stop = 1e-14 * float(r.norm()) + 1e-17 * float(b.norm())
    z = dinv * r
    p, rz = z.clone(), float(r @ z)
    for _ in range(400):
        if float(r.norm()) <= stop:
            break
        q = A @ p
        a = rz / float(p @ q)
        x, r = x + a * p, r - a * q
        z = dinv * r
        new = float(r @ z)
        p, rz = z + new / rz * p, new
    return x


def _exact_tissue(m, case, S, consts, stim, steps, dt, idt):
    gks, gto, endo = consts
    op, s, V = _operators(m, dt), [_t(S[:, k]) for k in range(S.shape[1])], _t(S[:, 0])
    sub = int(round(dt / idt))
    for k in range(steps):
        V = _half(op, V)
        ist = torch.zeros_like(V)
        if stim is not None and k < int(1.0 / dt):
            ist[_t(stim[0], torch.long)] = float(stim[2][0]) / XI[case["model"]]
        for _ in range(sub):
            V = V + dt / sub * (_tt_compute(V, s, -ist, dt / sub, gks, gto, endo) if case["model"] == "tt"
                                else _mh_compute(V, s, ist, dt / sub))
        V = _half(op, V)
    V = V.cpu().numpy()
    if not case.get("states"):
        return V
    return dict(V=V, states=np.stack([V] + [s[k].cpu().numpy() for k in range(1, S.shape[1])], 1))


def _tt_maps(n, node_type, sets, gks):
    c = _t(sets)[_t(node_type, torch.long)] if node_type is not None else _t(sets[0]).expand(n, -1)
    return c[:, 15] * (_t(gks) if gks is not None else 1.0), c[:, 20], c[:, 53] != 0


def exact(case, seed):
    kind = case["kind"]
    if kind == "tissue":
        if case["precision"] == "learned":
            return None
        if "batch" in case:
            # the slabs as one mesh of unconnected parts
            inst = _batch_instances(case, seed)
            off = np.cumsum([0] + [m.n for m, _, _ in inst])
            part = np.repeat(np.arange(len(inst)), np.diff(off)).astype(np.uint8)
            whole = M.TetMesh(np.concatenate([m.xyz for m, _, _ in inst]),
                              np.concatenate([m.tets + o for (m, _, _), o in zip(inst, off)]),
                              np.concatenate([m.fibers for m, _, _ in inst]))
            maps = _tt_maps(whole.n, part, np.stack([c for _, c, _ in inst]), None)
            S = np.concatenate([_wave("tt", m.xyz, k) for m, _, k in inst])
            return _exact_tissue(whole, case, S, maps, None, case["steps"], 0.02, 0.02)
        m = _mesh(case)
        if m.n * case["steps"] * (5 if "shell" in case else 1) > 2e7:
            return None
        dt, idt = _steps_of(case)
        node_type, sets, gks = _cell_maps(case, m)
        maps = _tt_maps(m.n, node_type, TT_EPI[None, :] if sets is None else sets, gks)
        return _exact_tissue(m, case, _wave(case["model"], m.xyz, seed), maps, _stimulus(case, m), case["steps"], dt, idt)
    if kind == "half":
        m = _mesh(case)
        V = _wave("tt", m.xyz, seed)[:, 0]
        V = _t(V if case["precision"] == "fp64" else V.astype(np.float32))
        return _half(_operators(m, case["dt"]), V).cpu().numpy()
    if kind == "cells":
        S, _, node_type, sets, gks = _cells_inputs(case, seed)
        s, V = [_t(S[:, k]) for k in range(19)], _t(S[:, 0])
        maps, zero = _tt_maps(len(S), node_type, sets, gks), torch.zeros(len(S), dtype=torch.float64, device=_dev())
        for _ in range(5):
            V = V + 0.02 * _tt_compute(V, s, zero, 0.02, *maps)
        return torch.stack([V] + s[1:], 1).cpu().numpy() - S
    if kind == "ecg":
        m = _mesh(case)
        x, vol, dN, De = _elements(m, [1e-3, 5e-4, 2.5e-4])
        W = []
        for el in ELECTRODES[:case["leads"]] + m.xyz.mean(axis=0):
            G = 0.0
            for q in range(4):
                d = sum(_shape(q, a) * x[:, a] for a in range(4)) - _t(el)
                G = G - d / (d.norm(dim=1, keepdim=True) ** 3) * (vol / 4)[:, None]
            w = torch.zeros(m.n, dtype=torch.float64, device=_dev())
            W.append(w.index_add_(0, _t(m.tets, torch.long).reshape(-1),
                                  torch.einsum("eai,eij,ej->ea", dN, De, G).reshape(-1)))
        return (_t(_frames(case, seed)) @ torch.stack(W, 1)).cpu().numpy()
    p, X, Y, w = (_t(v) for v in _train_inputs(case, seed))
    p.requires_grad_(True)
    h, at = X, 0
    for k, (a, b) in enumerate(zip(SG.DIMS, SG.DIMS[1:])):
        h = h @ p[at:at + a * b].reshape(b, a).T + p[at + a * b:at + a * b + b]
        h = torch.tanh(h) if k < 3 else h
        at += a * b + b
    loss = (w * (h - Y) ** 2).sum(1).mean()
    g, = torch.autograd.grad(loss, p)
    # Adam's first step: m / c1 = g, v / c2 = g^2
    new = p.detach() - 2e-5 * g / (g.abs() + 1e-8)
    return dict(loss=float(loss), grad=g.cpu().numpy(), params=new.cpu().numpy())
