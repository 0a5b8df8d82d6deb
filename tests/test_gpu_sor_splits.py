"""GPU: the streamed red-black SOR pass with a block's planes shared by one, two, four
or eight CTAs -- evenly or with a smaller last share -- and the 32^3 blocks that stay
staged or are swept in place at some block counts: the oracle's bits in FP64, the
separate launches' bits in FP32."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from oracle import pyoracle as po
from tests.helpers import assert_bitexact, outer_dirichlet
from tests.test_gpu_sor_shapes import brick_mask

pytestmark = pytest.mark.gpu


def tree_of(roots, radius):
    rg = bg.RootGrid(*roots, periodic=(False, True, False), root_length=1.0 / max(roots))
    if not radius:
        return bg.Octree.build(rg, bg.Divider.flat(0), "Z")
    return bg.Octree.build(rg, bg.Divider.sphere_surface((0.5, 0.5, 0.5), radius, 1), "Z")


def compare(tree, n, vc, dt, form, iters=3):
    ld, nid, sf, _ = tree.neighbors()
    bct, bcv = outer_dirichlet(tree, 0.25, periodic=(False, True, False))
    rng = np.random.default_rng(14)
    h = np.stack([tree.block_sizes / k for k in n], 1)
    coef, om = (bg.sor1_coef(h, 1.3), 1.3) if form == 1 else (bg.sor2_coef(h), 1.7)
    out = []
    for fused in ([True] if dt == "f64" else [True, False]):
        bm = bg.BlockManager(0)
        bm.register_octree(tree, n)
        bm.set_boundary(bct, bcv, bg.DIRICHLET_BCX)
        bm.set_fusion(fused)
        f, s = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
        if not out:
            a, src = (rng.uniform(-1, 1, size=f.shape).astype(f.dtype) for _ in range(2))
        f.upload(a)
        s.upload(src)
        bm.sor_run(f, coef, om, form=form, n_inner=1, n_outer=iters, s=s if form == 2 else None)
        out.append(f.download())
    if dt == "f64":
        ref = a.copy()
        po.OracleMesh(ld, nid, sf, n, vc).sor_run(ref, coef, om, form, 1, iters, bct, bcv, bg.DIRICHLET_BCX,
                                                  s=src if form == 2 else None)
        out.append(ref)
    mask = brick_mask(n, vc)
    assert_bitexact(out[0], out[1], mask, f"{dt} {n} vc={vc} form {form}, {tree.num_leaves} blocks, {iters}")
    assert_bitexact(out[0][:, ~mask], a[:, ~mask], what="edges keep their values")


@pytest.mark.parametrize("n", [(8, 8, 22), (8, 8, 24), (8, 8, 26), (8, 8, 30), (8, 8, 48), (8, 8, 50), (24, 20, 26)])
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("form", [1, 2])
def test_shares_of_a_block(gpu_ok, n, dt, form):
    compare(tree_of((2, 2, 2), 0.3), n, 1, dt, form)     # few blocks: the most shares
    compare(tree_of((4, 4, 4), 0.25), n, 2, dt, form)


@pytest.mark.parametrize("roots,radius", [((5, 4, 4), 0), ((5, 5, 4), 0), ((4, 4, 4), 0.15), ((6, 6, 6), 0),
                                          ((7, 6, 6), 0), ((4, 4, 4), 0.3), ((7, 7, 7), 0)])
@pytest.mark.parametrize("n,vc", [((32, 32, 32), 1), ((32, 32, 32), 2), ((24, 24, 24), 1)])
@pytest.mark.parametrize("form", [1, 2])
def test_by_number_of_blocks(gpu_ok, roots, radius, n, vc, form):
    tree = tree_of(roots, radius)
    for dt in ("f32", "f64"):
        compare(tree, n, vc, dt, form, iters=2)


def test_shares_of_456_blocks(gpu_ok):
    tree = tree_of((8, 8, 8), 0)
    for dt in ("f32", "f64"):
        compare(tree, (32, 32, 32), 1, dt, 2, iters=1)


@pytest.mark.parametrize("n,vc", [((32, 32, 32), 1), ((32, 32, 32), 2), ((40, 40, 40), 1), ((32, 40, 34), 2)])
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("iters", [1, 2, 3, 4])
def test_bricks_too_large_to_stage(gpu_ok, n, vc, dt, iters):
    compare(tree_of((2, 2, 2), 0.15), n, vc, dt, 2, iters)


@pytest.mark.parametrize("iters", [1, 2, 3])
def test_first_pass_in_place(gpu_ok, iters):
    """More blocks than SMs, no source, an odd number of passes."""
    compare(tree_of((3, 3, 3), 0.3), (32, 32, 32), 1, "f64", 1, iters)
