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
