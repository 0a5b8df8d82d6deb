"""Performance cases: what programs have this framework do, through its public
entry points, on the GPU.

Every case is one call (or one short sequence of calls) that such a program
repeats: a ghost update, a run of red-black SOR or Jacobi sweeps, the pieces of
a hand-written Krylov loop, or a BiCGSTAB solve.  The meshes are octrees of
equal blocks given as leaf lists; `exact` computes the same results in 64 bits
with torch from those lists alone.

Sizes: blocks of 2^3 to 32^3 cells (8, 16 and 32 the usual ones, others and
non-cubic ones too), 27 to 32768 blocks, one or two ghost layers, single and
double precision, meshes of one level and of several, constant operators and
operators given as seven coefficient fields.
"""
import ctypes

import numpy as np
import torch

import bcmtools_gb300 as bg
from bcmtools_gb300.batch import Batch
from bcmtools_gb300.workloads import Workload

# ---------------------------------------------------------------- the meshes


class Mesh:
    """Leaves of a 2:1 balanced octree over nx*ny*nz root blocks, in Z order:
    level, position at the own level, neighbours -- made here with numpy."""

    def __init__(self, root, level, marks, seed=0, radius=0.0):
        self.root, self.top = tuple(root), level
        n = np.array(root) << level                       # finest lattice
        lev = np.zeros(tuple(n), np.int64)
        rng = np.random.default_rng(seed)
        edge = 1.0 / max(root)                            # root block's edge: the longest side is 1
        box = np.array(root) * edge
        if marks == "flat":
            lev[:] = level
        else:
            if marks == "sphere":
                pts, r = [box / 2], radius
            else:                                         # balls around seeded points
                pts, r = rng.uniform(0, 1, (int(marks[5:]), 3)) * box, radius
            for l in range(level):
                s = 1 << (level - l)
                h = edge / (1 << l)
                m = np.array(root) << l
                lo = [np.arange(m[a]) * h for a in range(3)]
                meets = np.zeros(tuple(m), bool)
                for p in pts:
                    near = [np.maximum(np.maximum(lo[a] - p[a], p[a] - lo[a] - h), 0) for a in range(3)]
                    far = [np.maximum(np.abs(lo[a] - p[a]), np.abs(lo[a] + h - p[a])) for a in range(3)]
                    d2 = sum(np.square(x).reshape([-1 if a == b else 1 for b in range(3)]) for a, x in enumerate(near))
                    f2 = sum(np.square(x).reshape([-1 if a == b else 1 for b in range(3)]) for a, x in enumerate(far))
                    meets |= (d2 <= r * r) & ((f2 >= r * r) if marks == "sphere" else True)
                up = meets.repeat(s, 0).repeat(s, 1).repeat(s, 2)
                lev[up & (lev == l)] = l + 1
            while True:                                   # 2:1 across faces
                need = np.zeros_like(lev)
                for a in range(3):
                    v, w = np.moveaxis(need, a, 0), np.moveaxis(lev, a, 0)
                    np.maximum(v[1:], w[:-1] - 1, out=v[1:])
                    np.maximum(v[:-1], w[1:] - 1, out=v[:-1])
                bad = need > lev
                if not bad.any():
                    break
                was = lev.copy()
                for l in range(level):
                    s = 1 << (level - l)
                    m = np.array(root) << l
                    grow = (bad & (was == l)).reshape(m[0], s, m[1], s, m[2], s).any((1, 3, 5))
                    lev[grow.repeat(s, 0).repeat(s, 1).repeat(s, 2)] = l + 1
        ls, ps = [], []
        for l in range(level + 1):
            s = 1 << (level - l)
            at = np.argwhere(lev[::s, ::s, ::s] == l)
            ls.append(np.full(len(at), l))
            ps.append(at)
        lv, ps = np.concatenate(ls), np.concatenate(ps)
        rt = ps >> lv[:, None]
        q = ps - (rt << lv[:, None])                      # position in the root block
        rid = rt[:, 0] + root[0] * (rt[:, 1] + root[1] * rt[:, 2])
        fine = q << (level - lv)[:, None]
        z = np.zeros(len(lv), np.int64)
        for bit in range(level):
            for a in range(3):
                z |= ((fine[:, a] >> bit) & 1) << (3 * bit + a)
        order = np.lexsort((z, rid))
        self.level, self.pos = lv[order], ps[order]
        q, rid = q[order], rid[order]
        self.nb = len(order)
        self.edge = edge
        self.pedigrees = [(int(x) << 48) | (int(y) << 32) | (int(w) << 16) | (int(r) << 4) | int(l)
                          for (x, y, w), r, l in zip(q, rid, self.level)]
        # neighbours on the finest lattice
        own = np.zeros(tuple(n), np.int64)
        f0 = self.pos << (level - self.level)[:, None]
        for l in range(level + 1):
            s = 1 << (level - l)
            sel = np.nonzero(self.level == l)[0]
            g = np.arange(s)
            if len(sel):
                b = f0[sel]
                own[(b[:, 0, None] + g)[:, :, None, None], (b[:, 1, None] + g)[:, None, :, None],
                    (b[:, 2, None] + g)[:, None, None, :]] = sel[:, None, None, None]
        self.same, self.coarse, self.finer, self.outer = {}, {}, {}, {}
        size = 1 << (level - self.level)
        for a in range(3):
            u, v = [b for b in range(3) if b != a]
            for side in (0, 1):
                c = f0.copy()
                c[:, a] += size if side else -1
                out = (c[:, a] < 0) | (c[:, a] >= n[a])
                self.outer[a, side] = np.nonzero(out)[0]
                inn = np.nonzero(~out)[0]
                nbr = own[c[inn, 0], c[inn, 1], c[inn, 2]]
                d = self.level[nbr] - self.level[inn]
                self.same[a, side] = inn[d == 0], nbr[d == 0]
                k = inn[d == -1]                          # on a coarser block: which quarter of it
                self.coarse[a, side] = k, nbr[d == -1], self.pos[k, u] & 1, self.pos[k, v] & 1
                k, four = inn[d == 1], []
                for qv in (0, 1):
                    for qu in (0, 1):
                        e = c[k].copy()
                        e[:, u] += qu * (size[k] // 2)
                        e[:, v] += qv * (size[k] // 2)
                        four.append((qu, qv, own[e[:, 0], e[:, 1], e[:, 2]]))
                self.finer[a, side] = k, four

    def cell_sizes(self, n):
        return (self.edge / np.exp2(self.level))[:, None] / np.array(n)[None, :]


def mesh_of(case):
    return Mesh((case["rx"], case["ry"], case["rz"]), case["level"], case["marks"],
                case.get("mesh_seed", 0), case.get("radius", 0.0))


def edges(case):
    return case["nx"], case["ny"], case["nz"]


# ------------------------------------------------------------- 64-bit results


def _cut(t, a, lo, hi):
    return t.narrow(3 - a, lo, hi - lo)


class Exact:
    """Ghost update, boundary ghosts and 7-point arithmetic on padded bricks
    [block, z, y, x] in double precision."""

    def __init__(self, mesh, n, vc, bc, form):
        self.m, self.n, self.vc, self.bc, self.form = mesh, n, vc, bc, form
        dev = "cuda"
        ix = lambda v: torch.as_tensor(v, device=dev)  # noqa: E731
        self.same = {k: (ix(d), ix(s)) for k, (d, s) in mesh.same.items()}
        self.finer = {k: (ix(d), [(p, q, ix(s)) for p, q, s in f]) for k, (d, f) in mesh.finer.items()}
        self.coarse = {k: tuple(ix(v) for v in c) for k, c in mesh.coarse.items()}
        self.outer = {k: ix(v) for k, v in mesh.outer.items()}

    def inside(self, F):
        v, (nx, ny, nz) = self.vc, self.n
        return F[:, v:v + nz, v:v + ny, v:v + nx]

    def shifted(self, F, a, by):
        v, n = self.vc, self.n
        for b in range(3):
            F = _cut(F, b, v + (by if b == a else 0), v + n[b] + (by if b == a else 0))
        return F

    @staticmethod
    def _lerp(t, a, idx, n):
        i = torch.as_tensor(idx, device=t.device)
        at = torch.clamp(i // 2 - 1 + i % 2, 0, n - 2)
        r = (-0.25 + 0.5 * i - at).double()
        r = r.reshape([-1 if d == 3 - a else 1 for d in range(4)])
        return (1 - r) * t.index_select(3 - a, at) + r * t.index_select(3 - a, at + 1)

    def ghosts(self, F):
        """The ghost update: same level, from finer, from coarser."""
        vc, n = self.vc, self.n
        inner = self.inside(F)
        new = []
        for (a, side), (d, s) in self.same.items():
            lo = 0 if side else n[a] - vc
            if len(d):
                new.append((a, side, d, None, _cut(inner, a, lo, lo + vc)[s]))
        for (a, side), (d, four) in self.finer.items():
            lo = 0 if side else n[a] // 2 - vc
            for qu, qv, s in four:
                if len(d):
                    t = _cut(inner, a, 2 * lo, 2 * lo + 2 * vc)[s]
                    k, z, y, x = t.shape
                    new.append((a, side, d, (qu, qv), t.reshape(k, z // 2, 2, y // 2, 2, x // 2, 2).mean((2, 4, 6))))
        for (a, side), (d, s, pu, pv) in self.coarse.items():
            u, v = [b for b in range(3) if b != a]
            for qu in (0, 1):
                for qv in (0, 1):
                    sel = torch.nonzero((pu == qu) & (pv == qv)).flatten()
                    if not len(sel):
                        continue
                    t = inner[s[sel]]
                    t = self._lerp(t, a, list(range(vc)) if side else list(range(2 * n[a] - vc, 2 * n[a])), n[a])
                    t = self._lerp(t, u, list(range(n[u] * qu, n[u] * (qu + 1))), n[u])
                    t = self._lerp(t, v, list(range(n[v] * qv, n[v] * (qv + 1))), n[v])
                    new.append((a, side, d[sel], None, t))
        for a, side, d, q, t in new:
            at = [None] * 3
            at[a] = slice(vc + n[a], 2 * vc + n[a]) if side else slice(0, vc)
            for j, b in enumerate([b for b in range(3) if b != a]):
                at[b] = slice(vc, vc + n[b]) if q is None else slice(vc + q[j] * n[b] // 2, vc + (q[j] + 1) * n[b] // 2)
            F[d, at[2], at[1], at[0]] = t

    def boundary(self, F, zero=False):
        vc, n = self.vc, self.n
        for (a, side), d in self.outer.items():
            if not len(d):
                continue
            kind, val = self.bc[a, side]
            val = 0.0 if zero else val
            T = F[d]
            for b in range(3):
                if b != a:
                    T = _cut(T, b, vc, vc + n[b])
            near = _cut(T, a, vc + n[a] - 1, vc + n[a]) if side else _cut(T, a, vc, vc + 1)
            g1 = 2 * val - near if kind == "dirichlet" else (near + val if side else near - val)
            at = [slice(vc, vc + n[b]) for b in range(3)]
            at[a] = slice(vc + n[a], vc + n[a] + 1) if side else slice(vc - 1, vc)
            F[d, at[2], at[1], at[0]] = g1
            if vc >= 2 and (kind == "neumann" or self.form == "two_layers"):
                g2 = torch.full_like(near, val) if kind == "dirichlet" else (near + 2 * val if side else near - 2 * val)
                at[a] = slice(vc + n[a] + 1, vc + n[a] + 2) if side else slice(vc - 2, vc - 1)
                F[d, at[2], at[1], at[0]] = g2

    def impose(self, F, zero=False):
        self.ghosts(F)
        self.boundary(F, zero)

    def off_diagonal(self, A, F):
        return sum(A[1 + 2 * a + k] * self.shifted(F, a, by) for a in range(3) for k, by in ((0, -1), (1, 1)))

    def ax(self, A, F):
        return self.off_diagonal(A, F) + A[0] * self.inside(F)

    def jacobi(self, A, x, b, omega, zero=False):
        new = (b - self.off_diagonal(A, x)) / A[0]
        c = self.inside(x)
        c.copy_(c - omega * (c - new))
        self.impose(x, zero)

    def bicgstab(self, A, b, omega, n_pre, max_iter, eps):
        """Right-preconditioned BiCGSTAB from x = 0 (Jacobi passes)."""
        nb, (nx, ny, nz), v = b.shape[0], self.n, self.vc
        pad = lambda: torch.zeros(nb, nz + 2 * v, ny + 2 * v, nx + 2 * v, dtype=torch.float64, device=b.device)  # noqa: E731
        F = pad()
        self.impose(F)
        r = b - self.ax(A, F)
        x = torch.zeros_like(b)
        r0, p = r.clone(), r.clone()
        bb, rho = (b * b).sum(), (r * r).sum()

        def pre(w):
            z = pad()
            for _ in range(n_pre):
                self.jacobi(A, z, w, omega, zero=True)
            return z

        for _ in range(max_iter):
            ph = pre(p)
            q = self.ax(A, ph)
            alpha = rho / (q * r0).sum()
            s = r - alpha * q
            sh = pre(s)
            t = self.ax(A, sh)
            gamma = (t * s).sum() / (t * t).sum()
            x = x + alpha * self.inside(ph) + gamma * self.inside(sh)
            r = s - gamma * t
            if float((r * r).sum() / bb) <= eps * eps:
                break
            rho, old = (r * r0).sum(), rho
            p = r + rho / old * alpha / gamma * (p - gamma * q)
        self.inside(F).copy_(x)
        self.impose(F)
        return F


# ------------------------------------------------------------------ the cases

# Flat: 27 to 32768 blocks of one level.  Levels: octrees refined around a
# sphere or seeded points.
_SPHERE = dict(rx=4, ry=4, rz=4, level=3, marks="sphere", radius=0.3)


def listed():
    cube = lambda n: dict(nx=n, ny=n, nz=n)  # noqa: E731
    return [
        # the reference's own example: a few hundred tiny blocks, double
        # precision, red-black SOR without a source; launches count
        dict(name="sor_example_f64", op="sor", dtype="f64", vc=1, form=1, iters=50, **cube(2),
             rx=4, ry=4, rz=4, level=1, marks="sphere", radius=0.4),
        # plain Poisson on a uniform cube, 512 blocks, a captured run of sweeps
        dict(name="jacobi_plain_f32", op="jacobi", dtype="f32", vc=1, iters=200, graph=True, **cube(16),
             rx=1, ry=1, rz=1, level=3, marks="flat"),
        # the ghost update alone, all three level differences, as an
        # application with sweeps of its own calls it (begin / end)
        dict(name="ghosts_sphere_f32", op="ghosts", dtype="f32", vc=2, **cube(16), **_SPHERE),
        # red-black SOR with a source on the two-level sphere mesh
        dict(name="sor_sphere_f32", op="sor", dtype="f32", vc=2, form=2, iters=100, **cube(16), **_SPHERE),
        dict(name="sor_sphere_f64", op="sor", dtype="f64", vc=2, form=2, iters=20, **cube(16), **_SPHERE),
        # the largest: 134 M cells, Jacobi sweeps streamed from memory
        dict(name="jacobi_large_f32", op="jacobi", dtype="f32", vc=1, iters=20, graph=False, **cube(16),
             rx=1, ry=1, rz=1, level=5, marks="flat"),
        # Jacobi on 32^3 blocks of five levels
        dict(name="jacobi_points_f32", op="jacobi", dtype="f32", vc=1, iters=10, graph=False, **cube(32),
             rx=1, ry=1, rz=1, level=5, marks="balls16", mesh_seed=3, radius=0.05),
        # sweeps with an operator given as seven coefficient fields (variable
        # coefficients, boundary folded in), double precision
        dict(name="jacobi_fields_f64", op="jacobi_fields", dtype="f64", vc=1, iters=10, **cube(16), **_SPHERE),
        # BiCGSTAB on coefficient fields, blocks of an untypical shape
        dict(name="bicgstab_fields_f64", op="bicgstab_fields", dtype="f64", vc=1, iters=16, nx=24, ny=20, nz=12,
             rx=5, ry=5, rz=5, level=1, marks="balls3", mesh_seed=5, radius=0.2),
        # BiCGSTAB with a constant operator, double precision: one solve at a time
        dict(name="bicgstab_f64", op="bicgstab", dtype="f64", vc=1, iters=16, **cube(32),
             rx=3, ry=3, rz=3, level=2, marks="balls2", mesh_seed=7, radius=0.15),
        # several requests solved together to 1e-8 in mixed precision
        dict(name="served_mixed", op="mixed", dtype="f64", vc=1, requests=6, small=27, large=700, eps=1e-8, **cube(16),
             rx=1, ry=1, rz=1, level=0, marks="flat"),
        # the pieces of a hand-written Krylov loop: residual, products, updates
        dict(name="vector_ops_f32", op="vectors", dtype="f32", vc=1, **cube(20),
             rx=9, ry=8, rz=7, level=1, marks="balls2", mesh_seed=2, radius=0.1),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["ghosts", "ghosts", "sor", "sor", "sor", "jacobi", "jacobi", "jacobi", "jacobi_fields",
                     "jacobi_fields", "bicgstab_fields", "bicgstab", "bicgstab", "mixed", "vectors", "vectors"])
    dtype = rng.choice(["f32", "f64"])
    vc = rng.choice([1, 1, 2])
    if rng.random() < 0.7:
        n = (rng.choice([8, 16, 16, 32]),) * 3
    elif rng.random() < 0.6:
        n = (rng.choice([4, 6, 10, 12, 14, 18, 20, 24, 28]),) * 3
    else:
        n = tuple(rng.choice([6, 8, 10, 12, 16, 20, 24, 32]) for _ in range(3))
    case = dict(op=op, dtype=dtype, vc=vc, nx=n[0], ny=n[1], nz=n[2])
    cell = n[0] * n[1] * n[2]
    # cells in all: two hundred thousand to 40 million (6 to 16 with
    # coefficient fields or for solves)
    top = {"jacobi_fields": 16e6, "bicgstab": 8e6, "bicgstab_fields": 6e6}.get(op, 40e6)
    blocks = max(27, min(20000, _log(rng, 2e5, top) // cell))
    if op == "mixed":
        case.update(dtype="f64", vc=1, requests=rng.randint(2, 6), small=27,
                    large=max(40, min(700, _log(rng, 1e5, 2.2e6) // cell)), eps=1e-8,
                    rx=1, ry=1, rz=1, level=0, marks="flat")
        if case["large"] * cell > 2.4e6:
            case.update(nx=16, ny=16, nz=16)
        return case
    if rng.random() < 0.35:
        level = 0
        while blocks >> (3 * level) > 3000:               # a mesh has 4096 root blocks at most
            level += 1
        blocks >>= 3 * level
        a = max(3, int(round(blocks ** (1 / 3) * rng.uniform(0.8, 1.2))))
        b = max(3, int(round((blocks / a) ** 0.5 * rng.uniform(0.8, 1.2))))
        case.update(rx=a, ry=b, rz=max(3, blocks // (a * b)), level=level, marks="flat")
    else:
        level = rng.choice([1, 1, 2])
        a = min(15, max(2, int((blocks / 8 ** level * 3) ** (1 / 3))))
        case.update(rx=a, ry=max(2, a - rng.randint(0, 1)), rz=max(2, a + rng.randint(-1, 1)), level=level,
                    marks="balls%d" % rng.randint(1, 4), mesh_seed=rng.randint(0, 999), radius=rng.uniform(0.05, 0.2))
    if op == "sor":
        case.update(form=rng.choice([1, 2, 2]), iters=_log(rng, 4, 40 if dtype == "f32" else 10))
    elif op == "jacobi":
        case.update(iters=_log(rng, 2, 40), graph=rng.random() < 0.4)
    elif op == "jacobi_fields":
        case.update(iters=_log(rng, 2, 12))
    elif op.startswith("bicgstab"):
        case.update(iters=_log(rng, 6, 16))
    return case


# ----------------------------------------------------------------- the inputs


def _values(case, seed, mesh):
    """Seeded interiors (of the case's type): a smooth right-hand side with
    noise, a start vector, and what the operator is made of."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (seed % 100003) + 17)
    nx, ny, nz = n = edges(case)
    T = torch.float32 if case["dtype"] == "f32" else torch.float64
    h = torch.as_tensor(mesh.cell_sizes(n), device="cuda")
    # cell-centre coordinates per axis, [block, cells]
    at = [(torch.as_tensor(mesh.pos[:, a], device="cuda")[:, None] * n[a] + torch.arange(n[a], device="cuda") + 0.5)
          * h[:, a, None] for a in range(3)]
    spot = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * 0.6 + 0.2
    e = [torch.exp(-(at[a] - spot[a]) ** 2 / 0.02) for a in range(3)]
    rand = lambda lo, hi: torch.rand(mesh.nb, nz, ny, nx, generator=g, device="cuda",  # noqa: E731
                                     dtype=torch.float32) * (hi - lo) + lo
    b = (e[2][:, :, None, None] * e[1][:, None, :, None] * e[0][:, None, None, :]).to(T) + 0.01 * rand(-1, 1).to(T)
    return g, rand, h, b, T


def _boundary(case, seed):
    """Dirichlet on every outer face, a value per side of the domain."""
    r = np.random.default_rng(seed)
    return {(a, s): ("dirichlet", float(np.float32(r.uniform(-0.5, 0.5)))) for a in range(3) for s in (0, 1)}


def _laplace(h):
    c = 1.0 / (h * h)
    return torch.stack([-2 * c.sum(1), c[:, 0], c[:, 0], c[:, 1], c[:, 1], c[:, 2], c[:, 2]], 1)


def _fields(case, rand, h, T, mesh, bc, b):
    """Seven coefficient fields of a variable-coefficient operator (in the
    case's type) before their outer faces are folded in."""
    cc = _laplace(h)
    A = [cc[:, k, None, None, None] * (1 + 0.3 * rand(0, 1).double()) for k in range(1, 7)]
    A = [t.to(T) for t in A]
    return [-(A[0] + A[1] + A[2] + A[3] + A[4] + A[5])] + A


def _requests(case):
    """Meshes of one batch: sizes spread over their logarithm."""
    k, lo, hi = case["requests"], case["small"], case["large"]
    out = []
    for i in range(k):
        want = lo * (hi / lo) ** (i / max(1, k - 1))
        a = max(2, int(round((want / 3) ** (1 / 3))))
        out.append(Mesh((a, a, max(2, a - i % 2)), 1, "balls1", seed=i, radius=0.3))
    return out


class _Joined:
    """Several meshes as one block set, no face joining two."""

    def __init__(self, meshes):
        self.meshes = meshes
        self.first = np.concatenate([[0], np.cumsum([m.nb for m in meshes])])
        self.nb = int(self.first[-1])
        self.pos = np.concatenate([m.pos for m in meshes])
        self.level = np.concatenate([m.level for m in meshes])
        join = lambda name, which: {k: np.concatenate([getattr(m, name)[k][which] + o for m, o in zip(meshes, self.first)])  # noqa: E731
                                    for k in meshes[0].same}
        d, s = join("same", 0), join("same", 1)
        self.same = {k: (d[k], s[k]) for k in d}
        self.outer = {k: np.concatenate([m.outer[k] + o for m, o in zip(meshes, self.first)]) for k in d}
        cat = lambda k, i: np.concatenate([m.coarse[k][i] for m in meshes])  # noqa: E731
        d, s = join("coarse", 0), join("coarse", 1)
        self.coarse = {k: (d[k], s[k], cat(k, 2), cat(k, 3)) for k in d}
        self.finer = {}
        for k in d:
            to = np.concatenate([m.finer[k][0] + o for m, o in zip(meshes, self.first)])
            four = [(qu, qv, np.concatenate([m.finer[k][1][j][2] + o for m, o in zip(meshes, self.first)]))
                    for j, (qu, qv, _) in enumerate(meshes[0].finer[k][1])]
            self.finer[k] = to, four

    def cell_sizes(self, n):
        return np.concatenate([m.cell_sizes(n) for m in self.meshes])


# ----------------------------------------------------------- through the API

_STREAM = []


def _stream():
    """One stream for every call, as a program with one queue of work has it."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return ctypes.c_void_p(_STREAM[0].cuda_stream)


class _Memory:
    """A field's device memory for torch (whole bricks, no copy); holds the
    field's manager."""

    def __init__(self, field):
        p, stride, _ = field.layout()
        s, item = field.shape, np.dtype(field.dtype).itemsize
        self.owner = field.bm
        self.__cuda_array_interface__ = dict(
            shape=s, typestr="<f%d" % item, data=(p, False), version=2,
            strides=(stride * item, s[2] * s[3] * item, s[3] * item, item))


def bricks(field):
    return torch.as_tensor(_Memory(field), device="cuda")


def _set(field, interior):
    v = field.vc
    torch.cuda.synchronize()
    bricks(field)[:, v:-v, v:-v, v:-v] = interior
    torch.cuda.synchronize()


class State:
    pass


def _manager(case, mesh, bc, form):
    root = bg.RootGrid(*mesh.root, root_length=mesh.edge)
    tree = bg.Octree.from_pedigrees(root, mesh.pedigrees)
    bm = bg.BlockManager(0)
    outer = bm.register_octree(tree, edges(case))
    kind = np.where(outer != 0, bg.BC_DIRICHLET, 0)
    value = np.zeros((mesh.nb, 6))
    for (a, side), (_, v) in bc.items():
        value[outer[:, 2 * a + side] != 0, 2 * a + side] = v
    bm.set_boundary(kind, value, form)
    return bm


def prepare(case, seed):
    st = State()
    st.case = case
    op, n, vc, dt = case["op"], edges(case), case["vc"], case["dtype"]
    if op == "mixed":
        meshes = _requests(case)
        joined = _Joined(meshes)
        loads = [Workload("request", bg.Octree.from_pedigrees(bg.RootGrid(*m.root, root_length=m.edge),
                                                                          m.pedigrees), n[0], vc) for m in meshes]
        st.batch = Batch(loads)
        st.batch.set_dirichlet(0.0)
        st.batch.set_segments()
        st.bm = bm = st.batch.bm
        st.op = st.batch.laplace_op()
        st.x, st.b = bm.setDataClass(dt, vc), bm.setDataClass(dt, vc)
        _set(st.b, _values(case, seed, joined)[3])
        return st
    mesh = mesh_of(case)
    bc = _boundary(case, seed)
    form = bg.DIRICHLET_SOR if op in ("sor", "ghosts") else bg.DIRICHLET_BCX
    st.bm = bm = _manager(case, mesh, bc, form)
    _, rand, h, b, T = _values(case, seed, mesh)
    st.x = bm.setDataClass(dt, vc)
    start = rand(-1, 1).to(T)
    bm.prepareForVCUpdate(st.x)
    _set(st.x, start)
    if op != "ghosts":
        bm.imposeBoundaryCondition(st.x)
    hs = mesh.cell_sizes(n)
    if op == "sor":
        st.s = None
        if case["form"] == 2:
            st.s = bm.setDataClass(dt, vc)
            _set(st.s, b)
            st.coef, st.omega = bg.sor2_coef(hs), 1.8
        else:
            st.coef, st.omega = bg.sor1_coef(hs, 1.2), 1.2
    elif op != "ghosts":
        st.b = bm.setDataClass(dt, vc)
        _set(st.b, b)
        if op.endswith("fields"):
            st.fields = [bm.setDataClass(dt, vc) for _ in range(7)]
            for f, t in zip(st.fields, _fields(case, rand, h, T, mesh, bc, b)):
                _set(f, t)
            st.op = bm.op_fields(st.fields)
            bm.fold_boundary(st.op, st.b)
        else:
            st.op = bm.op_const(bg.laplace_coef(hs))
        if op == "vectors":
            st.r, st.p, st.y = (bm.setDataClass(dt, vc) for _ in range(3))
            _set(st.p, rand(-1, 1).to(T))
    bm.sync()
    torch.cuda.synchronize()
    return st


def run(st):
    case, bm, q = st.case, st.bm, _stream()
    op = case["op"]
    if op == "ghosts":
        bm.beginUpdateVC(st.x, stream=q)
        bm.endUpdateVC(st.x)
        bm.setBoundaryCondition(st.x, stream=q)
    elif op == "sor":
        bm.sor_run(st.x, st.coef, st.omega, form=case["form"], n_inner=1, n_outer=case["iters"], s=st.s, stream=q)
    elif op == "jacobi":
        bm.jacobi_run(st.op, st.x, st.b, 0.8, case["iters"], use_graph=case["graph"], stream=q)
    elif op == "jacobi_fields":
        bm.jacobi_run(st.op, st.x, st.b, 0.8, case["iters"], stream=q)
    elif op == "vectors":
        # one round of r = b - A x; y = A p; x += a p; r' = r - a y with the
        # step a = (r, p) / (p, A p); then p = r' + beta p
        bm.imposeBoundaryCondition(st.p, stream=q)
        bm.calc_r(st.op, st.r, st.x, st.b, stream=q)
        bm.calc_ax(st.op, st.y, st.p, stream=q)
        rp, pap = bm.dot(st.r, st.p, stream=q), bm.dot(st.p, st.y, stream=q)
        bm.axpy(st.x, st.p, 1e-3 * rp / pap, stream=q)
        bm.axpyz(st.r, st.y, st.r, -1e-3 * rp / pap, stream=q)
        bm.xpay(st.p, st.r, 1e-3, stream=q)
        bm.imposeBoundaryCondition(st.x, stream=q)
        rr = bm.calc_r2(st.op, st.x, st.b, stream=q)
        return dict(rp=rp, pap=pap, rr=rr, x=bricks(st.x), r=bricks(st.r), p=bricks(st.p), y=bricks(st.y))
    else:
        st.x.fill(0.0, stream=q)
        bm.imposeBoundaryCondition(st.x, stream=q)
        if op == "mixed":
            bm.bicgstab_mixed(st.op, st.x, st.b, omega=0.8, n_pre=2, max_inner=200, eps_inner=1e-2, max_outer=40,
                              eps=case["eps"], stream=q)
        else:
            bm.bicgstab(st.op, st.x, st.b, omega=0.8, n_pre=2, max_iter=case["iters"], eps=1e-12, stream=q)
    return bricks(st.x)


def exact(case, seed):
    op, n, vc = case["op"], edges(case), case["vc"]
    nx, ny, nz = n
    if op == "mixed":
        joined = _Joined(_requests(case))
        b = _values(case, seed, joined)[3].double()
        out = []
        for m, o in zip(joined.meshes, joined.first):
            e = Exact(m, n, vc, {k: ("dirichlet", 0.0) for k in m.outer}, "one_layer")
            A = [c[:, None, None, None] for c in _laplace(torch.as_tensor(m.cell_sizes(n), device="cuda")).unbind(1)]
            out.append(e.bicgstab(A, b[o:o + m.nb], 0.8, 2, 3000, 1e-12))
        return torch.cat(out)
    mesh = mesh_of(case)
    bc = _boundary(case, seed)
    _, rand, h, b, T = _values(case, seed, mesh)
    e = Exact(mesh, n, vc, bc, "one_layer" if op in ("sor", "ghosts") else "two_layers")
    x = torch.zeros(mesh.nb, nz + 2 * vc, ny + 2 * vc, nx + 2 * vc, dtype=torch.float64, device="cuda")
    e.inside(x).copy_(rand(-1, 1).to(T))
    e.impose(x)
    if op == "ghosts":
        return x
    b = b.double()
    if op == "sor":
        c = (1.0 / (h * h))[:, :, None, None, None].unbind(1)
        w = 1.8 if case["form"] == 2 else 1.2
        odd = sum(torch.arange(k, device="cuda").reshape(s) for k, s in ((nx, (1, 1, 1, -1)), (ny, (1, 1, -1, 1)), (nz, (1, -1, 1, 1)))) % 2
        src = b if case["form"] == 2 else 0.0
        for _ in range(case["iters"]):
            for colour in (0, 1):
                s = sum(c[a] * (e.shifted(x, a, -1) + e.shifted(x, a, 1)) for a in range(3))
                f = e.inside(x)
                f.copy_(torch.where(odd == colour, (1 - w) * f + w * (s - src) / (2 * (c[0] + c[1] + c[2])), f))
            e.impose(x)
        return x
    if op.endswith("fields"):
        A = [t.double() for t in _fields(case, rand, h, T, mesh, bc, b)]
        for (a, side), d in e.outer.items():
            k, val = 1 + 2 * a + side, bc[a, side][1]
            at = n[a] - 1 if side else 0
            for i in (d,):
                face = A[k].select(3 - a, at)
                A[0].select(3 - a, at)[i] -= face[i]
                b.select(3 - a, at)[i] -= 2 * face[i] * val
                face[i] = 0
    else:
        A = [c[:, None, None, None] for c in _laplace(h).unbind(1)]
    if op.startswith("jacobi"):
        for _ in range(case["iters"]):
            e.jacobi(A, x, b, 0.8)
        return x
    if op == "vectors":
        p = torch.zeros_like(x)
        e.inside(p).copy_(rand(-1, 1).to(T))
        e.impose(p)
        pad = lambda t: torch.nn.functional.pad(t, (vc,) * 6)  # noqa: E731
        r, y = b - e.ax(A, x), e.ax(A, p)
        rp, pap = float((r * e.inside(p)).sum()), float((e.inside(p) * y).sum())
        step = 1e-3 * rp / pap
        e.inside(x).add_(e.inside(p), alpha=step)
        r = r - step * y
        e.inside(p).copy_(r + 1e-3 * e.inside(p))
        e.impose(x)
        rr = float(((b - e.ax(A, x)) ** 2).sum())
        return dict(rp=rp, pap=pap, rr=rr, x=x, r=pad(r), p=p, y=pad(y))
    return e.bicgstab(A, b, 0.8, 2, case["iters"], 1e-12)


def work(case):
    """One pass: every sweep, product or update reads its vectors (and
    coefficient fields) once and writes its result once; a ghost layer is
    written once from cells read once."""
    n, op, size = edges(case), case["op"], 4 if case["dtype"] == "f32" else 8
    mesh = _Joined(_requests(case)) if op == "mixed" else mesh_of(case)
    cells = mesh.nb * n[0] * n[1] * n[2]
    ghosts = case["vc"] * sum((len(mesh.same[k][0]) + len(mesh.coarse[k][0]) + len(mesh.finer[k][0]) + len(mesh.outer[k]))
                              * (cells // mesh.nb // n[k[0]]) for k in mesh.same)
    layer = ghosts // case["vc"]
    if op == "ghosts":
        return dict(bytes=2.0 * ghosts * size, flops=1.0 * ghosts)
    if op == "sor":
        k = case["iters"]
        return dict(bytes=k * ((3 if case["form"] == 2 else 2) * cells + layer) * size, flops=13.0 * k * cells)
    if op == "jacobi":
        return dict(bytes=case["iters"] * (3 * cells + layer) * size, flops=16.0 * case["iters"] * cells)
    if op == "jacobi_fields":
        return dict(bytes=case["iters"] * (10 * cells + layer) * size, flops=16.0 * case["iters"] * cells)
    if op == "vectors":
        return dict(bytes=(24.0 * cells + 2 * layer) * size, flops=60.0 * cells)
    # BiCGSTAB: per iteration two preconditioners of two sweeps, two products,
    # three vector updates and their inner products
    k = 150 if op == "mixed" else case["iters"]
    extra = 6 * 7 if op == "bicgstab_fields" else 0
    size = 4 if op == "mixed" else size
    return dict(bytes=k * ((31.0 + extra) * cells + 4 * layer) * size, flops=k * 110.0 * cells)
