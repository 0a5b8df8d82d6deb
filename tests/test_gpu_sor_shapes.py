"""GPU: red-black SOR with one inner pass on blocks of any even shape and on
32^3 blocks (planes streamed through shared memory): the oracle's bits in FP64,
the separate launches' bits in FP32, and the in-place sweep's bits when a memory
budget leaves no room for a second buffer."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from oracle import pyoracle as po
from tests.helpers import assert_bitexact, outer_dirichlet, small_octree

pytestmark = pytest.mark.gpu

SHAPES = [((2, 2, 2), 1), ((4, 4, 4), 2), ((6, 8, 4), 1), ((12, 10, 6), 2), ((24, 24, 24), 1),
          ((20, 12, 32), 3), ((32, 32, 32), 1), ((32, 32, 32), 2), ((8, 16, 40), 1)]


def brick_mask(n, vc):
    """Cells in at most one ghost slab."""
    out = [((np.arange(k + 2 * vc) < vc) | (np.arange(k + 2 * vc) >= k + vc)).astype(int) for k in n]
    return (out[2][:, None, None] + out[1][None, :, None] + out[0][None, None, :]) <= 1


def run(dt, n, vc, form, bcform, fused, iters=3, budget=0):
    tree = small_octree(periodic=(False, True, False), level=2 if max(n) < 24 else 1, radius=0.3)
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    bct, bcv = outer_dirichlet(tree, 0.25, periodic=(False, True, False))
    bm.set_boundary(bct, bcv, bcform)
    bm.set_fusion(fused)
    f, s = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
    rng = np.random.default_rng(11)
    a = rng.uniform(-1, 1, size=f.shape).astype(f.dtype)
    src = rng.uniform(-1, 1, size=f.shape).astype(f.dtype)
    f.upload(a)
    s.upload(src)
    h = np.stack([tree.block_sizes / k for k in n], 1)
    coef, om = (bg.sor1_coef(h, 1.3), 1.3) if form == 1 else (bg.sor2_coef(h), 1.7)
    if budget:
        bm.set_memory_budget(bm.memory_in_use() + budget)
    bm.sor_run(f, coef, om, form=form, n_inner=1, n_outer=iters, s=s if form == 2 else None)
    bm.sync()
    ld, nid, sf, _ = tree.neighbors()
    m = po.OracleMesh(ld, nid, sf, n, vc)
    ref = a.copy()
    m.sor_run(ref, coef, om, form, 1, iters, bct, bcv, bcform, s=src if form == 2 else None)
    return f.download(), ref, a


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("form", [1, 2])
@pytest.mark.parametrize("bcform", [bg.DIRICHLET_SOR, bg.DIRICHLET_BCX])
def test_sor_f64_bits(gpu_ok, n, vc, form, bcform):
    got, ref, a = run("f64", n, vc, form, bcform, True)
    assert_bitexact(got, ref, brick_mask(n, vc), f"sor {form} {n}")
    edges = ~brick_mask(n, vc)
    assert_bitexact(got[:, edges], a[:, edges], what="edges keep their values")


@pytest.mark.parametrize("n,vc", SHAPES)
@pytest.mark.parametrize("form", [1, 2])
def test_sor_f32_equals_separate_launches(gpu_ok, n, vc, form):
    got, _, _ = run("f32", n, vc, form, bg.DIRICHLET_SOR, True)
    ref, _, _ = run("f32", n, vc, form, bg.DIRICHLET_SOR, False)
    mask = brick_mask(n, vc)
    # C2F ghosts: one arithmetic in both; everything else is shared too
    assert_bitexact(got, ref, mask, f"sor {form} {n}")


def test_no_room_for_a_second_buffer(gpu_ok):
    """32^3 FP64 bricks do not fit shared memory: without room for the second
    buffer of the streamed pass the blocks are swept in place."""
    got, ref, _ = run("f64", (32, 32, 32), 1, 2, bg.DIRICHLET_SOR, True, budget=1)
    assert_bitexact(got, ref, brick_mask((32, 32, 32), 1), "in place")


def test_spare_work_fields_are_given_back(gpu_ok):
    """The reciprocals a run with coefficient fields keeps, and the second buffer
    of the streamed SOR pass, do not stand in the way of a later field."""
    tree = small_octree(periodic=(False, False, False), level=1, radius=0.3)
    n, vc = 8, 1
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    bct, bcv = outer_dirichlet(tree, 0.25)
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    x, b = bm.setDataClass("f64", vc), bm.setDataClass("f64", vc)
    one = bm.memory_in_use() // 2
    fs = [bm.setDataClass("f64", vc) for _ in range(7)]
    rng = np.random.default_rng(2)
    for k, f in enumerate(fs):
        f.upload(rng.uniform(0.5, 1.0, size=f.shape) - (7.0 if k == 0 else 0.0))
    x.upload(rng.uniform(-1, 1, size=x.shape))
    b.upload(rng.uniform(-1, 1, size=x.shape))
    op = bm.op_fields(fs)
    a0 = x.download()
    bm.set_memory_budget(bm.memory_in_use() + 2 * one)  # the work copy and one more
    bm.jacobi_run(op, x, b, 0.8, 5)
    with_recip = x.download()
    extra = bm.setDataClass("f64", vc)  # takes the reciprocals' place
    with pytest.raises(bg.BcmgError):
        bm.setDataClass("f64", vc)
    x.upload(a0)
    bm.jacobi_run(op, x, b, 0.8, 5)  # no room for them: divides
    assert_bitexact(x.download(), with_recip, what="with and without the reciprocals")
    bm.destroy(extra)

    bm = bg.BlockManager(0)
    bm.register_octree(tree, 32)
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    f = bm.setDataClass("f64", vc)
    bm.set_memory_budget(2 * bm.memory_in_use())
    coef = bg.sor1_coef(tree.cell_sizes(32), 1.3)
    bm.sor_run(f, coef, 1.3, form=1, n_inner=1, n_outer=2)
    bm.setDataClass("f64", vc)
    bm.sor_run(f, coef, 1.3, form=1, n_inner=1, n_outer=2)
    bm.sync()
