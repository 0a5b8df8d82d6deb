"""GPU: BiCGSTAB where its passes and sums take other routes than on a few cubic blocks
with a constant operator: coefficient fields (boundary folded in), blocks of other
shapes whose planes are summed in uneven parts, and FP32 meshes on both sides of the
lines between dependent and plain launches."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from oracle import pyoracle as po
from tests.helpers import outer_dirichlet, small_octree

pytestmark = pytest.mark.gpu


def problem(n, vc, dt, fields, roots=0):
    if roots:
        rg = bg.RootGrid(roots, roots, roots, root_length=1.0 / roots)
        tree = bg.Octree.build(rg, bg.Divider.sphere_surface((0.5, 0.5, 0.5), 0.3, 1), "Z")
    else:
        tree = small_octree(periodic=(False, False, False), level=2 if max(n) <= 12 else 1, radius=0.3)
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    ld, nid, sf, _ = tree.neighbors()
    m = po.OracleMesh(ld, nid, sf, n, vc)
    bct, bcv = outer_dirichlet(tree, 0.0)
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    x, b = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
    rng = np.random.default_rng(7)
    inner = (slice(None),) + (slice(vc, -vc),) * 3
    ab = np.zeros(x.shape, x.dtype)
    ab[inner] = rng.uniform(-1, 1, size=ab[inner].shape)
    h = np.stack([tree.block_sizes / k for k in n], 1)
    cc = bg.laplace_coef(h) * h.max() ** 2
    if not fields:
        return bm, m, x, b, ab, bct, bcv, inner, bm.op_const(cc), dict(cc=cc)
    A = [(cc[:, k, None, None, None] * (1 + 0.3 * rng.uniform(0, 1, x.shape))).astype(x.dtype) for k in range(1, 7)]
    A = [-sum(A[1:], A[0]).astype(x.dtype)] + A
    fs = [bm.setDataClass(dt, vc) for _ in range(7)]
    for f, a in zip(fs, A):
        f.upload(a)
    op = bm.op_fields(fs)
    b.upload(ab)
    bm.fold_boundary(op, b)
    m.fold(A, ab, bct, bcv)
    return bm, m, x, b, ab, bct, bcv, inner, op, dict(fields=A)


SHAPES = [((8, 8, 8), 1), ((16, 16, 16), 2), ((24, 20, 12), 1), ((16, 16, 18), 1), ((20, 18, 14), 2), ((4, 6, 8), 1),
          ((32, 32, 32), 1), ((24, 24, 22), 3)]


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("fields", [False, True])
@pytest.mark.parametrize("n_pre", [1, 2])
def test_f64_iterations(gpu_ok, n, vc, fields, n_pre):
    """Five iterations: the oracle forms its inner products in another order (relative
    1e-16 each), which five iterations amplify by far less than 1e4."""
    bm, m, x, b, ab, bct, bcv, inner, op, kw = problem(n, vc, "f64", fields)
    b.upload(ab)
    ref = np.zeros_like(ab)
    m.bicgstab(ref, ab, 0.8, n_pre, 5, 1e-30, bct, bcv, 0, **kw)
    for _ in range(2):  # a second solve finds the work fields as the first left them
        x.fill(0.0)
        info = bm.bicgstab(op, x, b, omega=0.8, n_pre=n_pre, max_iter=5, eps=1e-30)
        assert info.iterations == 5
        g, r = x.download()[inner], ref[inner]
        assert np.linalg.norm(g - r) <= 1e-12 * np.linalg.norm(r)


def check_f32(bm, m, x, b, ab, bct, bcv, inner, op, kw, n_pre):
    """A solve to 1e-5 and the true residual, formed in FP64, of what it gives."""
    info = bm.bicgstab(op, x, b, omega=0.8, n_pre=n_pre, max_iter=400, eps=1e-5)
    assert info.status == 0 and info.residual <= 1e-10
    xs = x.download().astype(np.float64)
    m64 = po.OracleMesh(m.ld, m.id, m.sf, m.n, m.vc)
    m64.vc_update(xs)
    m64.dirichlet(xs, bct, np.zeros_like(bcv), 0)
    r = np.zeros_like(xs)
    if "fields" in kw:
        kw = dict(fields=[a.astype(np.float64) for a in kw["fields"]])
    m64.calc_r(r, xs, ab.astype(np.float64), **kw)
    assert np.linalg.norm(r[inner]) <= 2e-5 * np.linalg.norm(ab[inner].astype(np.float64))


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("fields", [False, True])
def test_f32_solution(gpu_ok, n, vc, fields):
    """To 1e-5: the residual of what comes back, formed in FP64 from the same FP32
    coefficients, is within twice that (the recursive residual's drift from the true
    one over the few dozen iterations is of the order of their number times 2^-24)."""
    bm, m, x, b, ab, bct, bcv, inner, op, kw = problem(n, vc, "f32", fields)
    b.upload(ab)
    x.fill(0.0)
    check_f32(bm, m, x, b, ab, bct, bcv, inner, op, kw, 2)


@pytest.mark.parametrize("n,roots", [((16, 16, 16), 3), ((16, 16, 16), 4), ((16, 16, 16), 6), ((8, 8, 8), 8),
                                     ((4, 4, 4), 14), ((12, 12, 12), 8)])
@pytest.mark.parametrize("n_pre", [1, 2])
def test_f32_repeats_itself(gpu_ok, n, roots, n_pre):
    """Launched as dependents or not, kernels of one solve see what the one before left:
    the same solve twice, and once more after another of the same context."""
    bm, m, x, b, ab, bct, bcv, inner, op, kw = problem(n, 1, "f32", False, roots)
    b.upload(ab)
    out = []
    for k in range(3):
        x.fill(0.0)
        bm.bicgstab(op, x, b, omega=0.8, n_pre=n_pre, max_iter=30, eps=1e-30)
        out.append(x.download()[inner])
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
