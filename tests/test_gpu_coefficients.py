"""GPU: FP64 sweeps choose their arithmetic by the block's coefficients -- one
coefficient for all six neighbours (each product formed once), a power of two
(SOR sums first, scales once), or any others -- and every choice gives the
oracle's bits.  The meshes of the other tests are dyadic cubes; here the cell
sizes are not powers of two, or differ by axis, and zeros of both signs and
blocks at rest are among the values."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from oracle import pyoracle as po
from tests.helpers import assert_bitexact, face_mask, outer_dirichlet, small_octree

pytestmark = pytest.mark.gpu


def sizes(tree, n, cells):
    h = tree.cell_sizes(n).copy()
    if cells == "odd":
        h /= 3.0
    elif cells == "mixed":  # blocks of both kinds in one launch
        h[::2] /= 3.0
    elif cells == "stretched":
        h *= np.array([1.0, 0.75, 1.5])
    return h


def problem(n, vc, seed):
    tree = small_octree(periodic=(False, True, False), level=2 if n < 32 else 1, radius=0.3)
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    ld, nid, sf, _ = tree.neighbors()
    m = po.OracleMesh(ld, nid, sf, n, vc)
    bct, bcv = outer_dirichlet(tree, 0.25, periodic=(False, True, False))
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    rng = np.random.default_rng(seed)
    shape = (tree.num_leaves,) + (n + 2 * vc,) * 3
    x, b = rng.uniform(-1, 1, size=shape), np.zeros(shape)
    b[:, vc:-vc, vc:-vc, vc:-vc] = rng.uniform(-1, 1, size=(shape[0], n, n, n))
    x[0], b[0] = 0.0, 0.0
    x[1, ::2] = -0.0
    b[1, :, ::2] = -0.0
    return tree, bm, m, bct, bcv, x, b


@pytest.mark.parametrize("cells", ["dyadic", "odd", "mixed", "stretched"])
@pytest.mark.parametrize("n,vc,push", [(8, 1, True), (8, 2, False), (16, 1, True), (16, 1, False),
                                       (16, 2, False), (32, 1, True), (32, 2, True)])
def test_jacobi_f64_bits(gpu_ok, n, vc, push, cells):
    tree, bm, m, bct, bcv, ax, ab = problem(n, vc, 3)
    bm.set_ghost_form(push=push)
    X, B, Y = (bm.setDataClass("f64", vc) for _ in range(3))
    X.upload(ax)
    B.upload(ab)
    cc = bg.laplace_coef(sizes(tree, n, cells))
    op = bm.op_const(cc)
    ref, ref1 = ax.copy(), np.zeros_like(ax)
    for _ in range(3):
        m.jacobi(ref1, ref, ab, 0.8, cc=cc)
        ref[:, vc:-vc, vc:-vc, vc:-vc] = ref1[:, vc:-vc, vc:-vc, vc:-vc]
        m.vc_update(ref)
        m.dirichlet(ref, bct, bcv, 0)
    bm.jacobi_run(op, X, B, 0.8, 3)
    assert_bitexact(X.download(), ref, face_mask(n, vc), f"jacobi {cells}")
    inner = (slice(None),) + (slice(vc, -vc),) * 3
    bm.calc_r(op, Y, X, B)
    m.calc_r(ref1, ref, ab, cc=cc)
    assert_bitexact(Y.download()[inner], ref1[inner], what=f"residual {cells}")
    bm.calc_ax(op, Y, X)
    m.calc_ax(ref1, ref, cc=cc)
    assert_bitexact(Y.download()[inner], ref1[inner], what=f"A x {cells}")


@pytest.mark.parametrize("cells", ["dyadic", "odd", "mixed", "stretched"])
@pytest.mark.parametrize("n,vc", [(8, 1), (16, 1), (16, 2)])
@pytest.mark.parametrize("n_inner,n_outer", [(1, 3), (2, 9)])
def test_sor_f64_bits(gpu_ok, n, vc, n_inner, n_outer, cells):
    tree, bm, m, bct, bcv, ax, ab = problem(n, vc, 4)
    X, S = bm.setDataClass("f64", vc), bm.setDataClass("f64", vc)
    X.upload(ax)
    S.upload(ab)
    coef = bg.sor2_coef(sizes(tree, n, cells))
    bm.sor_run(X, coef, 1.8, form=2, n_inner=n_inner, n_outer=n_outer, s=S)
    ref = ax.copy()
    m.sor_run(ref, coef, 1.8, 2, n_inner, n_outer, bct, bcv, 0, s=ab)
    assert_bitexact(X.download(), ref, face_mask(n, vc), f"sor {cells}")


@pytest.mark.parametrize("cells", ["dyadic", "odd", "stretched"])
@pytest.mark.parametrize("n,vc", [(16, 1), (32, 1), (32, 2)])
def test_bicgstab_f64_agrees(gpu_ok, n, vc, cells):
    """Six iterations with two preconditioner passes: the oracle forms its
    inner products in another order (relative 1e-16 each), which six
    iterations amplify by far less than 1e4."""
    tree, bm, m, bct, bcv, _, ab = problem(n, vc, 5)
    X, B = bm.setDataClass("f64", vc), bm.setDataClass("f64", vc)
    B.upload(ab)
    h = sizes(tree, n, cells)
    cc = bg.laplace_coef(h) * h.max() ** 2
    bct0, bcv0 = bct, np.zeros_like(bcv)
    bm.set_boundary(bct0, bcv0, bg.DIRICHLET_SOR)
    op = bm.op_const(cc)
    bm.bicgstab(op, X, B, omega=0.8, n_pre=2, max_iter=6, eps=1e-14)
    ref = np.zeros_like(ab)
    m.bicgstab(ref, ab, 0.8, 2, 6, 1e-14, bct0, bcv0, 0, cc=cc)
    inner = (slice(None),) + (slice(vc, -vc),) * 3
    g, r = X.download()[inner], ref[inner]
    assert np.linalg.norm(g - r) <= 1e-12 * np.linalg.norm(r), cells


def with_a_hole():
    """Two levels with one fine leaf left out: a coarse face fed by three of
    its four quarters, whose other ghosts no launch writes."""
    full = small_octree(periodic=(False, False, False), level=2, radius=0.3)
    ld, nid, _, _ = full.neighbors()
    b, f = np.argwhere(ld == 1)[0]
    peds = np.delete(full.pedigrees, nid[b, f, 2])
    return bg.Octree.from_pedigrees(full.rootgrid, peds)


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("n,vc", [(8, 2), (16, 1), (32, 1)])
@pytest.mark.parametrize("iters", [1, 2, 5])
@pytest.mark.parametrize("push", [True, False])
def test_jacobi_run_with_a_face_fed_in_part(gpu_ok, dt, n, vc, iters, push):
    tree = with_a_hole()
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    ld, nid, sf, outer = tree.neighbors()
    assert ((nid[ld == 1] < 0).any(axis=1) & (nid[ld == 1] >= 0).any(axis=1)).any()
    m = po.OracleMesh(ld, nid, sf, n, vc)
    bct, bcv = outer_dirichlet(tree, 0.25)
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    bm.set_ghost_form(push=push)
    x, b = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
    rng = np.random.default_rng(8)
    a0 = rng.uniform(-1, 1, size=x.shape).astype(x.dtype)
    ab = np.zeros_like(a0)
    inner = (slice(None),) + (slice(vc, -vc),) * 3
    ab[inner] = rng.uniform(-1, 1, size=ab[inner].shape)
    x.upload(a0)
    b.upload(ab)
    cc = bg.laplace_coef(tree.cell_sizes(n))
    bm.jacobi_run(bm.op_const(cc), x, b, 0.9, iters)
    ref, x1 = a0.copy(), np.zeros_like(a0)
    for _ in range(iters):
        m.jacobi(x1, ref, ab, 0.9, cc=cc)
        ref[inner] = x1[inner]
        m.vc_update(ref)
        m.dirichlet(ref, bct, bcv, 0)
    assert_bitexact(x.download(), ref, face_mask(n, vc), f"partly fed {dt} {n} {iters}")


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("vc", [1, 2])
@pytest.mark.parametrize("copies", [1, 3, 6, 12, 50])
def test_blocks_of_32_alone_and_among_others(gpu_ok, dt, vc, copies):
    """The streamed 32^3 sweep splits a block over 8, 4, 2 or 1 CTAs by the number
    of blocks (15 a copy here): every copy of a mesh in one block set gets the
    field it gets alone, bit for bit, and the oracle's; so does its BiCGSTAB."""
    from bcmtools_gb300.batch import Batch
    from bcmtools_gb300.workloads import Workload
    n = 32
    rg = bg.RootGrid(1, 1, 1, root_length=1.0)
    tree = bg.Octree.build(rg, bg.Divider.sphere_surface((0.3, 0.3, 0.3), 0.1, 2), "Z")
    batch = Batch([Workload("copy", tree, n, vc)] * copies)
    bm = batch.bm
    bct, bcv = batch.set_dirichlet(0.25)
    op = batch.laplace_op()
    x, b = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
    rng = np.random.default_rng(9)
    shape = (15,) + x.shape[1:]
    a0, ab = rng.uniform(-1, 1, size=shape).astype(x.dtype), np.zeros(shape, x.dtype)
    inner = (slice(None),) + (slice(vc, -vc),) * 3
    ab[inner] = rng.uniform(-1, 1, size=ab[inner].shape)
    x.upload(np.tile(a0, (copies, 1, 1, 1)))
    b.upload(np.tile(ab, (copies, 1, 1, 1)))
    bm.jacobi_run(op, x, b, 0.9, 3)
    got = x.download()
    for k in range(1, copies):
        assert_bitexact(batch.instance(got, k), batch.instance(got, 0), what=f"copy {k}")
    ld, nid, sf, _ = tree.neighbors()
    m = po.OracleMesh(ld, nid, sf, n, vc)
    cc = bg.laplace_coef(tree.cell_sizes(n))
    ref, x1 = a0.copy(), np.zeros_like(a0)
    for _ in range(3):
        m.jacobi(x1, ref, ab, 0.9, cc=cc)
        ref[inner] = x1[inner]
        m.vc_update(ref)
        m.dirichlet(ref, bct[:15], bcv[:15], 0)
    mask = face_mask(n, vc)
    if dt == "f64":
        assert_bitexact(got[:15], ref, mask, "oracle")
    else:  # C2F ghosts of FP32 fields: one ulp
        d = np.abs(got[:15][:, mask].astype(np.float64) - ref[:, mask])
        assert d.max() <= 1e-6 * np.abs(ref).max()
    batch.set_segments()
    bm.set_boundary(bct, np.zeros_like(bcv))
    x.fill(0.0)
    infos = bm.bicgstab(op, x, b, omega=0.8, n_pre=2, max_iter=5, eps=1e-12)
    infos = infos if isinstance(infos, list) else [infos]
    sol = x.download()
    for k in range(1, copies):
        assert_bitexact(batch.instance(sol, k)[inner], batch.instance(sol, 0)[inner], what=f"solve {k}")
        assert infos[k].iterations == infos[0].iterations
    one = bg.BlockManager(0)
    one.register_octree(tree, n)
    one.set_boundary(bct[:15], np.zeros((15, 6)))
    y, c = one.setDataClass(dt, vc), one.setDataClass(dt, vc)
    c.upload(ab)
    one.bicgstab(one.op_const(cc), y, c, omega=0.8, n_pre=2, max_iter=5, eps=1e-12)
    assert_bitexact(y.download()[inner], sol[:15][inner], what="solve alone")
