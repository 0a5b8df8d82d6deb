"""GPU: the first call of a kind makes its work fields; on a stream other than the
context's, whose own stream is still busy, the zeros they start with must not land
on what the call has written.  Every result equals the one on an idle context."""
import numpy as np
import pytest

import bcmtools_gb300 as bg
from tests.helpers import assert_bitexact, outer_dirichlet, small_octree

pytestmark = pytest.mark.gpu

CALLS = ["jacobi_const", "jacobi_fields", "jacobi_solve", "sor_staged", "sor_streamed", "bicgstab"]


def result(call, busy):
    torch = pytest.importorskip("torch")
    n = 32 if call == "sor_streamed" else 16
    tree = small_octree(periodic=(False, False, False), level=1, radius=0.3)
    bm = bg.BlockManager(0)
    bm.register_octree(tree, n)
    bct, bcv = outer_dirichlet(tree, 0.25)
    bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
    x, b = bm.setDataClass("f64", 1), bm.setDataClass("f64", 1)
    rng = np.random.default_rng(4)
    x.upload(rng.uniform(-1, 1, size=x.shape))
    b.upload(rng.uniform(-1, 1, size=x.shape))
    cc = bg.laplace_coef(tree.cell_sizes(n))
    if call == "jacobi_fields":
        fs = [bm.setDataClass("f64", 1) for _ in range(7)]
        for k, f in enumerate(fs):
            f.fill(-6.5 if k == 0 else 1.0)
        op = bm.op_fields(fs)
    else:
        op = bm.op_const(cc)
    bm.sync()
    side = torch.cuda.Stream()
    stream = None
    if busy:
        stream = side.cuda_stream
        other = bm.setDataClass("f64", 1)
        for k in range(400):  # some milliseconds of work on the context's stream
            bm.axpbypz(other, b, b, 1e-3, 1e-3)
    if call.startswith("jacobi_s"):
        bm.jacobi_solve(op, x, b, 0.8, 5, 1e-30, stream=stream)
    elif call.startswith("jacobi"):
        bm.jacobi_run(op, x, b, 0.8, 5, stream=stream)
    elif call.startswith("sor"):
        bm.sor_run(x, bg.sor2_coef(tree.cell_sizes(n)), 1.7, form=2, n_inner=1, n_outer=9, s=b,
                   stream=stream)
    else:
        bm.bicgstab(op, x, b, omega=0.8, n_pre=2, max_iter=3, eps=1e-30, stream=stream)
    side.synchronize()
    bm.sync()
    return x.download()


@pytest.mark.parametrize("call", CALLS)
def test_first_call_on_a_stream_of_its_own(gpu_ok, call):
    assert_bitexact(result(call, True), result(call, False), what=call)
