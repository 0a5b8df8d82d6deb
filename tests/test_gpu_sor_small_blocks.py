"""GPU: red-black SOR on blocks of a few cells: staged whole, a warp or a part of one
per ghost entry by the block's number of them, or streamed from a number of blocks
on.  The oracle's bits in FP64; in FP32 the separate launches' bits."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from oracle import pyoracle as po
from tests.helpers import assert_bitexact, outer_dirichlet
from tests.test_gpu_sor_shapes import brick_mask

pytestmark = pytest.mark.gpu


def mesh(roots, level):
    """Flat meshes have six ghost entries a block at most, two-level ones up to 24."""
    rg = bg.RootGrid(roots, roots, roots, periodic=(False, True, False), root_length=1.0 / roots)
    if not level:
        return bg.Octree.build(rg, bg.Divider.flat(0), "Z")
    return bg.Octree.build(rg, bg.Divider.sphere_surface((0.5, 0.5, 0.5), 0.3, level), "Z")


@pytest.mark.parametrize("n,vc", [((2, 2, 2), 1), ((4, 4, 4), 1), ((4, 4, 4), 2), ((6, 6, 6), 2), ((10, 2, 2), 1),
                                  ((2, 4, 8), 1)])
@pytest.mark.parametrize("roots,level", [(4, 0), (4, 1), (8, 1)])
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("n_inner", [1, 2])
@pytest.mark.parametrize("bcform", [bg.DIRICHLET_SOR, bg.DIRICHLET_BCX])
def test_small_blocks(gpu_ok, n, vc, roots, level, dt, n_inner, bcform):
    tree = mesh(roots, level)
    ld, nid, sf, _ = tree.neighbors()
    bct, bcv = outer_dirichlet(tree, 0.25, periodic=(False, True, False))
    rng = np.random.default_rng(13)
    out = []
    for fused in ([True] if dt == "f64" else [True, False]):
        bm = bg.BlockManager(0)
        bm.register_octree(tree, n)
        bm.set_boundary(bct, bcv, bcform)
        bm.set_fusion(fused)
        f, s = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
        if not out:
            a, src = (rng.uniform(-1, 1, size=f.shape).astype(f.dtype) for _ in range(2))
        f.upload(a)
        s.upload(src)
        coef = bg.sor2_coef(np.stack([tree.block_sizes / k for k in n], 1))
        bm.sor_run(f, coef, 1.7, form=2, n_inner=n_inner, n_outer=3, s=s)
        out.append(f.download())
    if dt == "f64":
        ref = a.copy()
        po.OracleMesh(ld, nid, sf, n, vc).sor_run(ref, coef, 1.7, 2, n_inner, 3, bct, bcv, bcform, s=src)
        out.append(ref)
    assert_bitexact(out[0], out[1], brick_mask(n, vc), f"{dt} {n} {tree.num_leaves} blocks")
    edges = ~brick_mask(n, vc)
    assert_bitexact(out[0][:, edges], a[:, edges], what="edges keep their values")
