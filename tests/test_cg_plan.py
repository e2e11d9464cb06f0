"""Which CG kernel a launch of the library's choice runs (csrc/cg_plan.cuh), on the
host: every size gets one, also where a CTA's slice bounds leave no ring."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "native", "cg_plan_host.cu")
OUT = os.path.join(HERE, "native", "_build", "libcg_plan_host.so")
DEPS = [SRC] + [os.path.join(ROOT, "ucla_cmg_b200", "csrc", f) for f in ("cg_plan.cuh", "common.cuh")]
SMS = 148
# (FP32, threads, CTAs per SM) of the launches left to the library
SHAPES = [(1, 256, 1), (1, 512, 1), (1, 256, 2), (0, 256, 1), (0, 384, 1), (0, 256, 2)]


@pytest.fixture(scope="module")
def plan():
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    nvcc = nvcc if os.path.exists(nvcc) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("nvcc not available to build the host harness")
    if not os.path.exists(OUT) or os.path.getmtime(OUT) < max(os.path.getmtime(d) for d in DEPS):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-Xcompiler", "-fPIC",
                        "-shared", "-I", os.path.join(ROOT, "include"), "-o", OUT, SRC], check=True, capture_output=True)
    lib = C.CDLL(OUT)

    def f(fp32, block, per_sm, ns, cols, nslices, grid=None, ninst=1, largest=None):
        o = [C.c_int(0), C.c_int(0), C.c_int(0), C.c_double(0), C.c_int(0), C.c_int(0)]
        k = lib.cg_plan(fp32, ns, C.c_longlong(cols), nslices, ninst, largest or nslices, block, grid or SMS * per_sm,
                        per_sm, *map(C.byref, o))
        return (k,) + tuple(v.value for v in o)
    f.named = lambda *a: lib.cg_named(*a[:-1], C.c_double(a[-1]))
    return f


@pytest.mark.parametrize("fp32,block,per_sm", SHAPES)
def test_every_size_gets_a_launch(plan, fp32, block, per_sm):
    seen = set()
    for wide in (1, 8, 9, 15, 16, 17, 40, 300):
        for ns in (1, 2, 7, 31, 64, 500, 1023, 1024, 1563, 5631, 5632, 9215, 9216, 11263, 11264, 20000, 60000):
            nslices = min(ns * SMS * per_sm, (1 << 31) // (32 * wide))
            k, threads, ring, smem, keep, grid, per = plan(fp32, block, per_sm, ns, nslices * wide, nslices)
            seen.add(k)
            if k == 1:
                # two units of nine columns, 227 KB of shared memory an SM (6 KB of it a CTA's own)
                assert threads == block and ring >= 18 and per_sm * (smem + 6144) <= 227 * 1024
                assert 0 < keep <= 1 and grid == SMS * per_sm
            elif k == 0:
                assert threads == 1024 // per_sm and grid == SMS * per_sm
            else:
                assert k == 2 and threads * per == 1536 and grid == 0
    assert seen == {0, 1, 2}


@pytest.mark.parametrize("fp32,block,per_sm,ns,wide,choice", [
    (1, 512, 1, 11264, 1, 0), (0, 384, 1, 9216, 1, 0), (0, 256, 2, 1024, 1, 0), (0, 256, 2, 1563, 15, 2),
    (1, 256, 2, 5632, 15, 2)])
def test_shares_whose_bounds_leave_no_ring_run_without(plan, fp32, block, per_sm, ns, wide, choice):
    nslices = ns * SMS * per_sm if wide > 1 else 100000
    assert plan(fp32, block, per_sm, ns, wide * nslices, nslices)[0] in (choice, 2)


@pytest.mark.parametrize("fp32,per_sm,ns,mb,choice", [
    (1, 2, 70, 27.0, 0),      # one large instance among small ones: its CTAs' shares are several times the average,
    (1, 2, 160, 50.0, 0),     # the whole matrix is what L2 holds or does not
    (1, 2, 160, 70.0, 1),
    (0, 1, 200, 20.0, 0),
    (0, 1, 200, 40.0, 1)])
def test_uneven_shares_are_judged_by_the_whole_matrix(plan, fp32, per_sm, ns, mb, choice):
    cols = int(mb * 1e6 / (32 * (8 if fp32 else 12)))
    k, threads, ring, smem, keep, grid, per = plan(fp32, 256, per_sm, ns, cols, cols // 15)
    assert k == choice
    if k:
        assert keep == pytest.approx(36.0 / mb if mb > 60 else 1.0, rel=1e-3)


def test_large_matrices_take_two_passes(plan):
    size = lambda mb, fp32: int(mb * 1e6 / (32 * (8 if fp32 else 12)))  # noqa: E731
    for fp32, block, per_sm, ninst, edge in ((1, 512, 1, 1, 390), (0, 384, 1, 1, 350), (0, 384, 1, 10, 250),
                                             (1, 256, 2, 64, 260), (0, 256, 2, 64, 150)):
        for mb, two in ((0.97 * edge, False), (1.03 * edge, True)):
            cols = size(mb, fp32)
            ns = -(-cols // 15 // (SMS * per_sm))
            k, threads, _, _, _, grid, per = plan(fp32, block, per_sm, ns, cols, cols // 15, ninst=ninst,
                                                  largest=cols // 15 // ninst + 1)
            assert (k == 2) == two
            if two:
                assert (threads, per, grid) == ((768, 2, 0) if ninst <= 36 else (256, 6, 0))
    # shares twice as uneven count twice
    cols = size(140, 1)
    assert plan(1, 256, 2, -(-2 * cols // 15 // (2 * SMS)), cols, cols // 15, ninst=64, largest=cols // 600)[0] == 2


def test_one_large_among_many_small_instances_gets_more_ctas(plan):
    nslices = 250 * 16 + 600
    k, threads, _, _, _, grid, per = plan(1, 256, 2, 16, 15 * nslices, nslices, ninst=251, largest=600)
    assert (k, threads, grid, per) == (0, 256, 0, 4)
    assert plan(1, 256, 2, 16, 15 * 4000, 4000, ninst=250, largest=16)[5] != 0


def test_named_shapes_of_large_matrices(plan):
    assert not plan.named(1, 8, 256, 32, 1, 60.0) and plan.named(1, 8, 256, 32, 1, 200.0)
    assert not plan.named(1, 4, 256, 32, 1, 5000.0) and plan.named(1, 4, 768, 48, 1, 200.0)
    assert not plan.named(0, 4, 512, 32, 1, 400.0) and plan.named(0, 4, 512, 32, 100, 400.0)
    assert not plan.named(0, 16, 256, 32, 1, 400.0) and plan.named(0, 32, 256, 24, 1, 400.0)
