"""GPU: the work fields a context keeps although it could do without them (the
reciprocals of a coefficient operator, the second buffer of the streamed SOR pass)
are given back when any other allocation of the context finds no room.  The want of
room is made on the host: a stand-in for the runtime's allocation calls refuses
them until something has been freed."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SHIM = r"""
#include <dlfcn.h>
#include <stddef.h>
static int full = 0, refused = 0, given_back = 0;
// the runtime is a dependency of a library opened later: not in this one's scope
static void* real(const char* name) {
  void* h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
  return h ? dlsym(h, name) : NULL;
}
typedef int (*alloc_t)(void**, size_t);
typedef int (*alloc_async_t)(void**, size_t, void*);
typedef int (*free_t)(void*);
void shim_fill(void) { full = 1; refused = given_back = 0; }
int shim_refused(void) { return refused; }
int shim_given_back(void) { return given_back; }
void shim_empty(void) { full = 0; }
int cudaMalloc(void** p, size_t n) {
  static alloc_t f;
  if (full && !given_back) { refused++; return 2; }
  if (!f) f = (alloc_t)real("cudaMalloc");
  return f(p, n);
}
int cudaMallocAsync(void** p, size_t n, void* st) {
  static alloc_async_t f;
  if (full && !given_back) { refused++; return 2; }
  if (!f) f = (alloc_async_t)real("cudaMallocAsync");
  return f(p, n, st);
}
int cudaFree(void* p) {
  static free_t f;
  if (p) given_back++;
  if (!f) f = (free_t)real("cudaFree");
  return f(p);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
import bcmtools_gb300 as bg
from tests.helpers import outer_dirichlet, small_octree
what = sys.argv[1]
shim = ctypes.CDLL(sys.argv[2])
n, vc = 16, 1
tree = small_octree(periodic=(False, False, False), level=1, radius=0.3)
bm = bg.BlockManager(0)
bm.register_octree(tree, n)
bct, bcv = outer_dirichlet(tree, 0.25)
bm.set_boundary(bct, bcv, bg.DIRICHLET_SOR)
x, b = bm.setDataClass("f64", vc), bm.setDataClass("f64", vc)
fs = [bm.setDataClass("f64", vc) for _ in range(7)]
for k, f in enumerate(fs):
    f.fill(-6.5 if k == 0 else 1.0)
b.fill_random(3)
fields = bm.op_fields(fs)
cc = bg.laplace_coef(tree.cell_sizes(n))
const = bm.op_const(cc)
coef = bg.sor2_coef(tree.cell_sizes(n))
calls = {
    "operator": lambda: bm.op_const(cc),
    "sor": lambda: bm.sor_run(x, coef, 1.7, form=2, n_inner=1, n_outer=3, s=b),
    "pull": lambda: (bm.set_ghost_form(push=False), bm.jacobi_run(const, x, b, 0.8, 3)),
    "fold": lambda: bm.fold_boundary(fields, b),
    "boundary": lambda: bm.set_boundary(bct, bcv, bg.DIRICHLET_BCX),
}
bm.set_ghost_form(push=True)
if what == "sor":  # leaves the second buffer too
    calls["sor"]()
if what == "pull":  # its work copy, but no side buffers
    bm.jacobi_run(const, x, b, 0.8, 2)
bm.jacobi_run(fields, x, b, 0.8, 5)  # leaves the reciprocals
bm.sync()
shim.shim_fill()
calls[what]()
bm.sync()
print("refused", shim.shim_refused(), "given back", shim.shim_given_back())
assert shim.shim_refused() > 0 and shim.shim_given_back() > 0
shim.shim_empty()
"""


@pytest.mark.parametrize("what", ["operator", "sor", "pull", "fold", "boundary"])
def test_given_back_to_any_allocation(gpu_ok, tmp_path, what):
    if not shutil.which("gcc"):
        pytest.skip("needs gcc")
    (tmp_path / "shim.c").write_text(SHIM)
    (tmp_path / "child.py").write_text(CHILD)
    so = tmp_path / "shim.so"
    subprocess.run(["gcc", "-D_GNU_SOURCE", "-shared", "-fPIC", str(tmp_path / "shim.c"), "-o", str(so),
                    "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=str(ROOT))
    out = subprocess.run([sys.executable, str(tmp_path / "child.py"), what, str(so)], cwd=ROOT, env=env,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
