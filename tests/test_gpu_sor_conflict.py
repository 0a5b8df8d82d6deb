"""GPU: red-black SOR where a face has a neighbour and a Dirichlet condition: the
ghost update writes its ghosts first and the boundary condition last, on every
block shape, bit for bit as the oracle has it."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from oracle import pyoracle as po
from tests.helpers import assert_bitexact, outer_dirichlet, small_octree
from tests.test_gpu_sor_shapes import brick_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,vc", [((8, 8, 8), 1), ((16, 16, 16), 2), ((32, 32, 32), 1), ((4, 4, 4), 2),
                                  ((6, 8, 4), 1), ((24, 20, 12), 3)])
@pytest.mark.parametrize("bcform", [bg.DIRICHLET_SOR, bg.DIRICHLET_BCX])
@pytest.mark.parametrize("n_inner", [0, 1, 2])
def test_boundary_faces_with_neighbours(gpu_ok, n, vc, bcform, n_inner):
    tree = small_octree(periodic=(False, True, False), level=2 if max(n) < 24 else 1, radius=0.3)
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    bct, bcv = outer_dirichlet(tree, 0.25, periodic=(False, True, False))
    rng = np.random.default_rng(12)
    bct[rng.random(bct.shape) < 0.1] = bg.BC_DIRICHLET
    bcv = np.where(bct != 0, rng.uniform(-1, 1, bct.shape), 0.0)
    bm.set_boundary(bct, bcv, bcform)
    f, s = bm.setDataClass("f64", vc), bm.setDataClass("f64", vc)
    a, src = rng.uniform(-1, 1, size=f.shape), rng.uniform(-1, 1, size=f.shape)
    f.upload(a)
    s.upload(src)
    coef = bg.sor2_coef(np.stack([tree.block_sizes / k for k in n], 1))
    bm.sor_run(f, coef, 1.7, form=2, n_inner=n_inner, n_outer=3, s=s)
    ld, nid, sf, _ = tree.neighbors()
    assert ((bct == bg.BC_DIRICHLET) & (nid >= 0).any(axis=2)).any()
    ref = a.copy()
    po.OracleMesh(ld, nid, sf, n, vc).sor_run(ref, coef, 1.7, 2, n_inner, 3, bct, bcv, bcform, s=src)
    assert_bitexact(f.download(), ref, brick_mask(n, vc), f"sor {n} {n_inner}")
