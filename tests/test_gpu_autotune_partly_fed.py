"""GPU: on a mesh with a face fed in part the fused sweeps have the push form alone,
so the tuners time and name no other."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from tests.helpers import outer_dirichlet
from tests.test_gpu_coefficients import with_a_hole

pytestmark = pytest.mark.gpu

PUSH, PULL_SHAPES = 1, (6, 7)  # bcmg_autotune_jacobi's push form; the SOR pull shapes


@pytest.mark.parametrize("push", [None, False, True])
@pytest.mark.parametrize("n,vc", [(8, 1), (16, 2)])
def test_no_pull_shape_is_named(gpu_ok, push, n, vc):
    tree = with_a_hole()
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    bct, bcv = outer_dirichlet(tree, 0.25)
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    bm.set_ghost_form(push=push)
    x, b = bm.setDataClass("f32", vc), bm.setDataClass("f32", vc)
    x.fill_random(1)
    b.fill_random(2)
    launches = []
    for iters in (2, 4):
        before = bm.launch_count()
        best, us = bm.autotune_jacobi(bm.op_const(bg.laplace_coef(tree.cell_sizes(n))), x, b, 0.8, iters=iters)
        launches.append(bm.launch_count() - before)
        assert best == PUSH and us > 0
    # a warm-up of two sweeps, then iters and 2 iters of them: of the one form
    assert launches[1] - launches[0] == 3 * 2
    best, us = bm.autotune_sor(x, bg.sor2_coef(tree.cell_sizes(n)), 1.7, form=2, s=b, iters=3)
    assert best not in PULL_SHAPES and us > 0
    assert np.isfinite(x.download()).all()
