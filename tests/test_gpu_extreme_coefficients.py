"""GPU: constant operators and SOR coefficients at the ends of the ranges in which the
kernels choose their arithmetic: Ap at 2^-60 and 2^60 and one ulp to either side,
beyond them, subnormal and zero dividends, neighbour coefficients of zero, and SOR
coefficients of 2^k for k up to and past 60.  The oracle's bits for what a pass makes
of given values; runs of several agree bit for bit between the fused and the separate
launches.  A coefficient that is not finite ends a solve as diverged."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from bcmtools_gb300 import capi
from oracle import pyoracle as po
from tests.helpers import assert_bitexact, outer_dirichlet, small_octree
from tests.test_gpu_field_sweeps import same_bits
from tests.test_gpu_sor_shapes import brick_mask

pytestmark = pytest.mark.gpu

SHAPES = [((8, 8, 8), 1), ((16, 16, 16), 1), ((16, 16, 16), 2), ((32, 32, 32), 1), ((12, 10, 6), 2)]


def setup(n, vc, dt):
    tree = small_octree(periodic=(False, True, False), level=2 if max(n) < 16 else 1, radius=0.3)
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    ld, nid, sf, _ = tree.neighbors()
    bct, bcv = outer_dirichlet(tree, 0.25, periodic=(False, True, False))
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    return tree, bm, po.OracleMesh(ld, nid, sf, n, vc), bct, bcv


def operators(nb, dt, rng):
    """Per block: Ap from the ends of the range of the stored reciprocals, and
    neighbour coefficients zero, small, equal or as large as Ap."""
    eps = np.finfo(np.float64 if dt == "f64" else np.float32).eps
    pool = []
    for e in (-60, 60):
        pool += [2.0 ** e, 2.0 ** e * (1 - eps / 2), 2.0 ** e * (1 + eps), 2.0 ** (e + 1), 2.0 ** (e - 1)]
    pool += [1.0, 3.0, 1.0 / 3.0, 2.0 ** 59 * 1.7, 2.0 ** -59 / 1.7]
    ap = rng.choice(pool, size=nb) * rng.choice([-1.0, 1.0], size=nb)
    cc = np.zeros((nb, 7))
    cc[:, 0] = ap
    kind = rng.integers(0, 4, size=nb)
    same = rng.uniform(0.1, 0.3, size=nb)
    cc[:, 1:] = np.where((kind == 0)[:, None], 0.0,
                         np.where((kind == 1)[:, None], same[:, None],
                                  np.where((kind == 2)[:, None], rng.uniform(0.1, 0.3, (nb, 6)),
                                           (same * np.abs(ap))[:, None])))
    return cc


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("push", [True, False])
def test_jacobi(gpu_ok, n, vc, dt, push):
    tree, bm, m, bct, bcv = setup(n, vc, dt)
    bm.set_ghost_form(push=push)
    rng = np.random.default_rng(15)
    x, b, y = (bm.setDataClass(dt, vc) for _ in range(3))
    T = x.dtype
    cc = operators(x.shape[0], dt, rng)
    op = bm.op_const(cc)
    ax = rng.uniform(-1, 1, size=x.shape).astype(T)
    ab = rng.uniform(-1, 1, size=x.shape)
    big = rng.random(x.shape) < 0.5  # quotients of order one, and at the ends of their range
    ab = np.where(big, ab * np.abs(cc[:, 0])[:, None, None, None], ab).astype(T)
    ab[rng.random(x.shape) < 0.05] = 0.0
    ab[rng.random(x.shape) < 0.02] = -0.0
    ab[rng.random(x.shape) < 0.05] *= np.dtype(T).type(2.0 ** (-1040 if dt == "f64" else -130))
    inner = (slice(None),) + (slice(vc, -vc),) * 3
    flat = lambda a: a[inner].reshape(len(a), -1)  # noqa: E731
    x.upload(ax)
    b.upload(ab)
    ref = np.zeros_like(ax)
    with np.errstate(all="ignore"):
        m.jacobi(ref, ax, ab, 0.8, cc=cc)
        bm.jacobi_sweep(op, y, x, b, 0.8)
        same_bits(flat(y.download()), flat(ref), slice(None), f"sweep {n}")
        bm.jacobi_run(op, x, b, 0.8, 1)
        same_bits(flat(x.download()), flat(ref), slice(None), f"run {n}")
        m.calc_r(ref, ax, ab, cc=cc)
        x.upload(ax)
        bm.calc_r(op, y, x, b)
        same_bits(flat(y.download()), flat(ref), slice(None), f"residual {n}")
        out = []
        for fused in (True, False):
            bm.set_fusion(fused)
            x.upload(ax)
            bm.jacobi_run(op, x, b, 0.8, 4)
            out.append(x.download())
        same_bits(out[0], out[1], brick_mask(n, vc), f"fused and separate {n}")


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("iters", [1, 3, 9])
def test_sor_f64(gpu_ok, n, vc, iters):
    tree, bm, m, bct, bcv = setup(n, vc, "f64")
    rng = np.random.default_rng(16)
    f, s = bm.setDataClass("f64", vc), bm.setDataClass("f64", vc)
    cx = 2.0 ** rng.choice([-2, -1, 0, 1, 30, 59, 60, 61, 62], size=f.shape[0])
    cx = np.where(rng.random(len(cx)) < 0.15, -cx, cx) * rng.choice([1.0, 1.0, 1.5], size=len(cx))
    coef = np.stack([1.0 / (6.0 * cx), cx, cx, cx], 1)
    a, src = rng.uniform(-1, 1, size=f.shape), rng.uniform(-1, 1, size=f.shape)
    a[rng.random(f.shape) < 0.05] = -0.0
    f.upload(a)
    s.upload(src)
    bm.sor_run(f, coef, 1.7, form=2, n_inner=1, n_outer=iters, s=s)
    ref = a.copy()
    m.sor_run(ref, coef, 1.7, 2, 1, iters, bct, bcv, 0, s=src)
    assert_bitexact(f.download(), ref, brick_mask(n, vc), f"sor {n}")


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("which", [0, 3])
def test_not_finite(gpu_ok, n, vc, dt, which):
    """The preconditioner's pass from zero does not multiply by the neighbours'
    coefficients; a solve still sees the one that is not finite."""
    tree, bm, m, bct, bcv = setup(n, vc, dt)
    x, b = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
    b.fill_random(3)
    cc = bg.laplace_coef(np.stack([tree.block_sizes / k for k in n], 1))
    bad = cc.copy()
    bad[1, which] = np.nan
    bad[2, which] = np.inf
    for n_pre in (1, 2):
        x.fill(0.0)
        assert bm.bicgstab(bm.op_const(bad), x, b, omega=0.8, n_pre=n_pre, max_iter=20, eps=1e-8).status == capi.DIVERGED
    x.fill(0.0)
    info = bm.bicgstab(bm.op_const(cc), x, b, omega=0.8, n_pre=2, max_iter=5, eps=1e-30)
    assert info.iterations == 5 and np.isfinite(x.download()).all()
